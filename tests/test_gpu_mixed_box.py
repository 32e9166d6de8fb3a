"""The mixed path on 3D boxes whose CTAs stage, or cannot stage, the mesh
neighbourhood of their particles: extents of one stencil, rows that wrap in
x within a tile, tiles over two rows and over two planes, more cells than the
staged area holds, and a ragged last tile; and a run that ends inside a call.
One step and the deposit against the oracle with the tolerances of
test_gpu_mixed (2e-6 per flavor attribute, 1e-6 of the summed magnitude per
mesh component)."""
import numpy as np
import pytest

from emu_b200 import api
from emu_b200 import workloads as W
from oracle.oracle import Oracle
from tests.helpers import colwise_rel, flavor_cols, magnitude_mesh, mesh_rel_mag

pytestmark = pytest.mark.gpu


def _params(nf, n, ndirs):
    p = W.c5_3d(n=4, ndirs=ndirs, mixed=True)
    p.nflavors = nf
    api.set_param(p, "ncell", n)
    p.Lx, p.Ly, p.Lz = (0.5 * k for k in n)
    return p


@pytest.mark.parametrize("nf,n,ndirs", [(3, (3, 3, 3), 43), (2, (3, 3, 4), 43), (3, (7, 4, 3), 24), (2, (9, 3, 5), 13),
                                        (3, (33, 3, 3), 3), (2, (4, 5, 3), 128), (3, (5, 6, 4), 99)])
def test_step_and_deposit(nf, n, ndirs):
    p = _params(nf, n, ndirs)
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
def test_steps_past_the_end_of_a_run_change_nothing(nf):
    p = _params(nf, (7, 4, 3), 24)
    parts = api.init_particles(p)
    outs = []
    for n in (6, 11):
        with api.Context(p) as c:
            c.load_particles(parts)
            c.evolve_begin(0.0, float("inf"), 6)
            c.evolve_steps(n)
            info = c.evolve_end()
            assert info.steps_done == 6
            q = c.get_particles()
            outs.append(q[np.lexsort(q[:, 3:11].T[::-1])])
    assert np.array_equal(outs[0][:, :], outs[1][:, :])
