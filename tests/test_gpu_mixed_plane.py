"""The mixed path in the y-z plane (TSC, fixed 1 x 3 x 3 stencils): one step and
the deposit against the oracle, with the tolerances of test_gpu_mixed (2e-6
per flavor attribute, 1e-6 of the summed magnitude per mesh component), at
extents narrower than a stencil, ragged ones and particle counts around a
tile; and a run split into calls bit for bit against one call."""
import numpy as np
import pytest

from emu_b200 import api
from emu_b200 import workloads as W
from oracle.oracle import Oracle
from tests.helpers import colwise_rel, flavor_cols, magnitude_mesh, mesh_rel_mag

pytestmark = pytest.mark.gpu


def _params(nf, ny, nz, ndirs):
    p = W.c5_3d(n=4, ndirs=ndirs, mixed=True)
    p.nflavors = nf
    api.set_param(p, "ncell", (1, ny, nz))
    p.Lx, p.Ly, p.Lz = 0.5, 0.5 * ny, 0.5 * nz
    return p


@pytest.mark.parametrize("nf,ny,nz,ndirs", [(3, 6, 7, 9), (2, 6, 7, 9), (3, 2, 3, 43), (2, 8, 4, 4), (3, 43, 3, 3)])
def test_step_and_deposit(nf, ny, nz, ndirs):
    p = _params(nf, ny, nz, ndirs)
    parts = api.init_particles(p)
    o = Oracle(p)
    ref = o.deposit(parts)
    dt, _ = o.compute_dt(ref, o.vvac_max(parts))
    with api.Context(p) as c:
        c.load_particles(parts)
        assert mesh_rel_mag(c.get_mesh(), ref, magnitude_mesh(o, parts), 3 + 8 * nf * nf) < 1e-6
        c.step(dt)
        out = c.get_particles()
    q = parts.copy()
    o.rk_step(q, dt)
    fc = flavor_cols(nf)
    assert colwise_rel(out[:, fc], q[:, fc]) < 2e-6
    assert colwise_rel(out[:, :11], q[:, :11]) < 1e-14


@pytest.mark.parametrize("nf", [2, 3])
def test_split_run_gives_the_same_bits(nf):
    p = _params(nf, 9, 8, 10)
    parts = api.init_particles(p)
    outs = []
    for split in ([40], [1, 16, 23]):
        with api.Context(p) as c:
            c.load_particles(parts)
            c.evolve_begin(0.0, float("inf"), 40)
            for n in split:
                c.evolve_steps(n)
            c.evolve_end()
            outs.append((c.get_particles(), c.get_mesh()))
    assert np.array_equal(outs[0][0], outs[1][0]) and np.array_equal(outs[0][1], outs[1][1])
