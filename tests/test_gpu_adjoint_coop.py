"""Cooperative adjoint segments (two flavors), whose CTAs read meshes that
others write in the same launch, over a long segment: every address of the
adjoint meshes is zeroed, summed and read again some ten times.  Against the
same run swept with one launch per stage; the adjoint's 1e-9 normwise, for
runs recorded whole and for segments recomputed."""
import numpy as np
import pytest

from emu_b200 import api
from tests.golden.make_golden import _case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,order,ndirs", [((5, 4, 6), 2, 12), ((1, 9, 8), 2, 16), ((4, 5, 3), 1, 9)])
def test_long_segment_matches_launch_per_stage(cells, order, ndirs, monkeypatch):
    L = tuple(0.5 * c if c > 1 else 1.0 for c in cells)
    # (Renormalize off, as in test_gpu_adjoint_1d: 24 steps of this state end in its checks, the oracle too)
    _, p, parts = _case("x", 2, cells, order, L, ndirs, 41, rho=2e9, maxError=1e-2)
    out = {}
    for mode, env in (("whole", {}), ("segments", {"EMU_ADJOINT_FULL_STORE": "0"}),
                      ("stages", {"EMU_ADJOINT_STORE_MAX_BYTES": "0"})):
        for k, v in env.items():
            monkeypatch.setenv(k, v)
        with api.Context(p) as c:
            c.load_particles(parts)
            store = c.adjoint_reserve(24, 12)[1]
            c.adjoint_forward(24, 12)
            J, lf, lN = c.adjoint_objective()
            out[mode] = (store, J) + c.adjoint_backward(lf, lN)
        for k in env:
            monkeypatch.delenv(k)
    assert [out[m][0] for m in ("whole", "segments", "stages")] == [2, 1, 0]
    for m in ("whole", "segments"):
        for a, b in zip(out[m][1:], out["stages"][1:]):
            assert np.abs(np.asarray(a) - b).max() <= 1e-9 * np.abs(b).max()
