"""States that are not finite stay where the equations take them: one particle
with a NaN or an infinite flavor component, or NaN numbers, changes the cells
of its stencil and from there the particles that touch them, stage by stage,
and no other, as in the oracle.  Kernels whose products meet other particles
or cells with weight zero must not carry it further.  One step: the particles
that become NaN are the oracle's, every other agrees to the FP64 parity
tolerance (1e-11 normwise); the mesh likewise, cell by cell."""
import numpy as np
import pytest

from emu_b200 import api
from oracle.oracle import Oracle
from tests.golden.make_golden import _case
from tests.helpers import magnitude_mesh

pytestmark = pytest.mark.gpu

#   nf, cells, order, directions
CASES = [(2, (1, 1, 60), 2, 2), (3, (1, 1, 60), 2, 2), (2, (1, 1, 100), 1, 3), (2, (1, 1, 200), 2, 12),
         (3, (1, 1, 150), 2, 4), (3, (1, 1, 90), 1, 7), (2, (1, 1, 900), 2, 20), (3, (24, 23, 22), 2, 2),
         (2, (16, 15, 14), 1, 6), (2, (1, 30, 31), 2, 5), (3, (1, 30, 31), 1, 9), (2, (60, 1, 1), 2, 6)]


def _spoil(parts, nf, which, k):
    f = 3 + 10
    if which == "nan":
        parts[k, f + 1] = np.nan
    elif which == "inf":
        parts[k, f + 1] = np.inf
    else:
        parts[k, 3 + 8] = np.nan
    return parts


@pytest.mark.parametrize("which", ["nan", "inf", "number"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "nf%d_%s_o%d_%d" % (c[0], "x".join(map(str, c[1])), *c[2:]))
def test_one_bad_particle(case, which):
    nf, cells, order, ndirs = case
    L = tuple(0.5 * c if c > 1 else 1.0 for c in cells)
    _, p, parts = _case("x", nf, cells, order, L, ndirs, 51, rho=2e9, maxError=1e-2)
    o = Oracle(p)
    good = parts.copy()
    dt, _ = o.compute_dt(o.deposit(good), o.vvac_max(good))
    parts = _spoil(parts, nf, which, len(parts) // 2)
    ref = parts.copy()
    mesh_ref = o.rk_step(ref, dt)[0].reshape(3 + 8 * nf * nf, -1)[3:]
    with api.Context(p) as c:
        c.load_particles(parts)
        dep = c.get_mesh().reshape(3 + 8 * nf * nf, -1)[3:]
        want = o.deposit(parts).reshape(3 + 8 * nf * nf, -1)[3:]
        c.step(dt, raise_on_error=False)
        out, mesh = c.get_particles(), c.get_mesh().reshape(3 + 8 * nf * nf, -1)[3:]
    # (a zero weight times the bad value: the oracle has it in the cell, a kernel may leave it out)
    touched = ~np.isfinite(want).all(axis=0)
    assert 0 < touched.sum() < 0.5 * touched.size and np.isfinite(dep[:, ~touched]).all()
    bad = ~np.isfinite(ref).all(axis=1)
    assert 0 < bad.sum() < 0.9 * len(ref)
    assert not (~np.isfinite(out).all(axis=1) & ~bad).any()
    scale = np.abs(ref[~bad]).max(axis=0)
    assert (np.abs(out[~bad] - ref[~bad]) <= 1e-11 * scale).all()
    cells_ok = np.isfinite(mesh_ref).all(axis=0)
    assert np.isfinite(mesh[:, cells_ok]).all()
    mag = np.abs(magnitude_mesh(o, good).reshape(3 + 8 * nf * nf, -1)[3:]).reshape(8, -1).max(axis=1)
    err = np.abs(mesh - mesh_ref)[:, cells_ok].reshape(8, -1).max(axis=1)
    assert (err <= 1e-11 * mag).all()
    # and what touches the bad particle's cells is bad
    sure = bad & ~np.isfinite(o.interpolate_rhs(o.deposit(parts), parts)).all(axis=1)
    assert (~np.isfinite(out).all(axis=1))[sure].mean() > 0.5


@pytest.mark.parametrize("where", ["lam", "lamN", "state"])
@pytest.mark.parametrize("nf,nz,order,ndirs", [(2, 120, 2, 2), (3, 150, 2, 4), (3, 160, 1, 9)])
def test_one_bad_adjoint_row(nf, nz, order, ndirs, where, monkeypatch):
    """the stored 1D sweep against the one with a launch per stage"""
    _, p, parts = _case("x", nf, (1, 1, nz), order, (1.0, 1.0, 0.5 * nz), ndirs, 61, rho=2e9, maxError=1e-2)
    p.resort_interval = 0
    rng = np.random.default_rng(2)
    k = len(parts) // 2
    lam, lamN = rng.standard_normal((len(parts), 2 * nf * nf)), rng.standard_normal((len(parts), 2))
    if where == "lam":
        lam[k, 1] = np.nan
    elif where == "lamN":
        lamN[k, 0] = np.inf
    else:
        parts[k, 3 + 11] = np.nan
    out = []
    for store in (None, "0"):
        if store is not None:
            monkeypatch.setenv("EMU_ADJOINT_STORE_MAX_BYTES", store)
        with api.Context(p) as c:
            c.load_particles(parts)
            assert c.adjoint_reserve(2, 2)[1] == (2 if store is None else 0)
            c.adjoint_forward(2, 2)
            state = c.get_particles()
            out.append((state,) + c.adjoint_backward(lam, lamN))
    for got, want in zip(*out):
        bad = ~np.isfinite(want).all(axis=1)
        assert bad.sum() < 0.9 * len(want) and not (~np.isfinite(got).all(axis=1) & ~bad).any()
        assert np.abs(got[~bad] - want[~bad]).max() <= 1e-9 * np.abs(want[~bad]).max()
