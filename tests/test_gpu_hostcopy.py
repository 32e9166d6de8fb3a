"""Large copies between the device and pageable host memory go through a
pinned ring in chunks of 1 MiB (16 MiB and more).  Downloads and uploads at
record counts just below and above that size and around whole chunks: a
download bit for bit against one into pinned memory, the adjoint's uploads by
the gradient of pinned inputs (its atomics' 1e-9 normwise)."""
import numpy as np
import pytest
import torch

from emu_b200 import api
from tests.golden.make_golden import _case

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _make(n):
    cells = 64
    _, p, parts = _case("x", 2, (1, 1, cells), 2, (1.0, 1.0, 32.0), -(-n // cells), 3, rho=2e9, maxError=1e-2)
    return p, parts[:n].copy()


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64).pin_memory()


def _around(row, base):
    """row counts whose bytes lie just below and above a multiple of a chunk"""
    k = base // row
    return [k, k + 1]


@pytest.mark.parametrize("n", _around(184, 16 * MIB) + _around(184, 17 * MIB) + _around(184, 29 * MIB))
def test_download_matches_pinned(n):
    p, parts = _make(n)
    with api.Context(p) as c:
        c.load_particles(parts)
        got = c.get_particles()
        buf = _pinned((n, api.nreal(2)))
        c.get_particles_ptr(buf.data_ptr(), n)
        assert np.array_equal(got, buf.numpy()) and np.array_equal(got, parts)


@pytest.mark.parametrize("n", [16 * MIB // 64 - 1, 16 * MIB // 64, 16 * MIB // 64 + 1, 27 * MIB // 64 + 1])
def test_upload_matches_pinned(n):
    p, parts = _make(n)
    rng = np.random.default_rng(n)
    lam, lamN = rng.standard_normal((n, 8)), rng.standard_normal((n, 2))
    with api.Context(p) as c:
        c.load_particles(parts)
        c.adjoint_forward(1, 1)
        got = c.adjoint_backward(lam, lamN)
        pl, pn = _pinned((n, 8)), _pinned((n, 2))
        pl.numpy()[:], pn.numpy()[:] = lam, lamN
        want = c.adjoint_backward(pl.numpy(), pn.numpy())
        for a, b in zip(got, want):
            assert np.abs(a - b).max() <= 1e-9 * np.abs(b).max()
