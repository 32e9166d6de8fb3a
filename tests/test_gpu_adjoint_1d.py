"""The 1D adjoint with every step stored (recorded k_steps_1d, k_adjoint_1d)
against the one that recomputes its segments with the tile kernels
(EMU_ADJOINT_FULL_STORE=0), which test_gpu_adjoint checks against autograd:
one and several CTAs, windows wider than the staging area, domains narrower
than a stencil, stencil orders 0 to 2, a last segment shorter than the others,
re-sorts between segments.  Tolerance: the adjoint's 1e-9 normwise."""
import numpy as np
import pytest

from emu_b200 import api
from tests.test_gpu_steps1d import _make

pytestmark = pytest.mark.gpu

CASES = [(2, 1, 2, 2, 0), (2, 2, 2, 30, 0), (3, 3, 2, 60, 0), (2, 64, 2, 9, 0), (3, 40, 2, 12, 0), (2, 43, 1, 7, 0),
         (3, 20, 0, 13, 0), (2, 900, 2, 3, 300), (3, 300, 1, 3, 128), (2, 200, 2, 120, 0)]


def _run(p, parts, nsteps, interval):
    with api.Context(p) as c:
        c.load_particles(parts)
        store = c.adjoint_reserve(nsteps, interval)[1]
        dts, info = c.adjoint_forward(nsteps, interval)
        out, mesh = c.get_particles(), c.get_mesh()
        J, lf, lN = c.adjoint_objective()
        gf, gN = c.adjoint_backward(lf, lN)
        # the context goes on from the run's final state
        more = c.evolve(2, info.time)
        assert more.steps_done == 2
        return store, dts, out, mesh, J, gf, gN, c.get_particles()


@pytest.mark.parametrize("case", CASES, ids=lambda c: "nf%d_%dcells_o%d_%d_%d" % c)
@pytest.mark.parametrize("resort", [0, 2])
def test_stored_run_matches_recomputed(case, resort, monkeypatch):
    p, parts = _make(*case)
    p.resort_interval = resort
    p.maxError = 1e-2   # (Renormalize off: its branches are test_gpu_adjoint's)
    got = _run(p, parts, 7, 3)
    monkeypatch.setenv("EMU_ADJOINT_FULL_STORE", "0")
    want = _run(p, parts, 7, 3)
    assert got[0] == 2 and want[0] < 2
    for a, b in zip(got[1:], want[1:]):
        a, b = np.asarray(a), np.asarray(b)
        assert np.abs(a - b).max() <= 1e-9 * np.abs(b).max()
