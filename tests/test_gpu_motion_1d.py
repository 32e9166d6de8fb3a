"""The 1D kernels (k_steps_1d, k_adjoint_1d) where the particles cross many
cells within a launch (steps limited by translation, half a cell each): all
directions forward, all backward or mixed, with a last CTA of a few particles
whose other warps have none, up to a first re-sort and past it at the
automatic interval, single windows and windows wider than the staging area.

Tolerances: 1e-11 normwise, as test_gpu_steps1d (rounding of 40 steps at
phases of a hundredth of a radian stays below 1e-13); the adjoint's 1e-9
between the stored and the recomputed sweep."""
import numpy as np
import pytest

from emu_b200 import api
from oracle.oracle import Oracle
from tests.golden.make_golden import _case
from tests.test_gpu_adjoint_1d import _run
from tests.test_gpu_steps1d import _check

pytestmark = pytest.mark.gpu

#   nf, cells, order, directions, sign of v_z (0: as generated), particles kept
CASES = [
    (2, 70, 2, 3, 1, 0), (3, 70, 2, 3, 1, 0), (2, 70, 1, 3, 1, 0), (2, 70, 2, 3, -1, 0), (3, 150, 1, 2, -1, 210),
    (2, 129, 2, 2, 1, 130), (2, 90, 2, 9, 0, 0), (3, 200, 2, 5, 0, 999),
]


def _make(nf, nz, order, ndirs, sign, keep):
    # densities a hundredth of the other tests': dt = 0.5 dz / c
    _, p, parts = _case("x", nf, (1, 1, nz), order, (1.0, 1.0, 0.5 * nz), ndirs, 5 + nz, rho=2e7, st4_ndens=4.89e30,
                        st4_ndensbar=3.1e30)
    parts = parts[:keep].copy() if keep else parts
    if sign:
        rng = np.random.default_rng(nz)
        u, a = rng.uniform(0.6, 1.0, len(parts)), rng.uniform(0.0, 2 * np.pi, len(parts))
        s, E = np.sqrt(1.0 - u * u), parts[:, 10]
        parts[:, 7], parts[:, 8], parts[:, 9] = E * s * np.cos(a), E * s * np.sin(a), sign * E * u
    return p, parts


@pytest.mark.parametrize("case", CASES, ids=lambda c: "nf%d_%dcells_o%d_%d_%+d_%d" % c)
@pytest.mark.parametrize("resort", [0, -1])
def test_steps_match_oracle(case, resort):
    p, parts = _make(*case)
    p.resort_interval = resort
    n = 40
    o = Oracle(p)
    ref = parts.copy()
    mesh_ref = o.deposit(ref)
    vv, t = o.vvac_max(ref), 0.0
    for _ in range(n):
        dt, _ = o.compute_dt(mesh_ref, vv)
        assert dt * api.CLIGHT > 0.49 * p.Lz / p.ncell[2]
        mesh_ref = o.rk_step(ref, dt)[0]
        t += dt
    with api.Context(p) as c:
        c.load_particles(parts)
        info = c.evolve(n)
        assert info.steps_done == n and abs(info.time - t) <= 1e-12 * t
        _check(p, c.get_particles(), ref, c.get_mesh(), mesh_ref, o)


@pytest.mark.parametrize("case", [(2, 70, 2, 3, 0, 0), (2, 70, 2, 3, -1, 0), (3, 70, 1, 3, -1, 0), (2, 70, 2, 3, 1, 0),
                                  (2, 90, 2, 9, 0, 0)], ids=lambda c: "nf%d_%dcells_o%d_%d_%+d_%d" % c)
def test_stored_adjoint_matches_recomputed(case, monkeypatch):
    p, parts = _make(*case)
    p.resort_interval = 0
    p.maxError = 1e-2
    got = _run(p, parts, 24, 24)
    monkeypatch.setenv("EMU_ADJOINT_FULL_STORE", "0")
    want = _run(p, parts, 24, 24)
    assert got[0] == 2 and want[0] < 2
    for a, b in zip(got[1:], want[1:]):
        a, b = np.asarray(a), np.asarray(b)
        assert np.abs(a - b).max() <= 1e-9 * np.abs(b).max()
