"""1D FP64 problems with more cells than particles: the several-step kernel's
timestep comes from every CTA's share of the cells, with one CTA and many,
most cells empty, a matter potential that alone limits it, several launches
between re-sorts.  Against the oracle: 1e-11 normwise after the steps, every
step's dt through the time reached and the next dt."""
import numpy as np
import pytest

from emu_b200 import api
from oracle.oracle import Oracle
from tests.golden.make_golden import _case
from tests.helpers import colwise_rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nf,nz,n,order,rho", [(2, 5000, 300, 2, 0.0), (3, 3001, 700, 1, 2e9), (2, 9000, 4000, 2, 0.0),
                                               (3, 700, 60, 2, 2e9), (2, 4001, 2000, 0, 1e13), (3, 2500, 2400, 2, 0.0)])
@pytest.mark.parametrize("resort", [-1, 2])
def test_steps_match_oracle(nf, nz, n, order, rho, resort):
    _, p, parts = _case("x", nf, (1, 1, 8), order, (1.0, 1.0, 4.0), -(-n // 8), 91, rho=rho, maxError=1e-2, cfl_factor=-1.0)
    api.set_param(p, "ncell", (1, 1, nz))
    p.Lz = 0.5 * nz
    p.resort_interval = resort
    parts = parts[:n].copy()
    parts[:, 2] = parts[:, 6] = np.random.default_rng(nz).uniform(0.0, p.Lz, n)
    o = Oracle(p)
    ref, t, dts, _ = o.evolve(parts, 6)
    with api.Context(p) as c:
        c.load_particles(parts)
        c.evolve_begin(0.0, float("inf"), 6)
        c.evolve_steps(1)
        c.evolve_steps(5)
        info = c.evolve_end()
        assert info.steps_done == 6 and abs(info.time - t) <= 1e-12 * t
        nxt, _ = o.compute_dt(c.get_mesh(), o.vvac_max(parts))
        assert abs(info.dt_next - nxt) <= 1e-12 * nxt
        assert colwise_rel(c.get_particles(), ref) < 1e-11
    if rho == 0.0:   # (elsewhere the matter potential is the larger)
        assert len(set(dts)) > 1
