"""Gradients of runs whose particles change cells and are re-sorted inside
every checkpoint segment, the last one among them, against torch autograd: the
adjoint state and the static fields have to be taken through each segment's
composed map in every storage mode.  Positions off the cell centres, half a
cell of motion per step (steps limited by translation), TSC and CIC in one,
two and three dimensions, a run recorded after an evolve.  Tolerance: the
adjoint's 1e-9 normwise."""
import numpy as np
import pytest
import torch

from emu_b200 import api
from emu_b200.adjoint import flavor_columns, number_columns
from tests.golden.make_golden import _case
from tests.torch_ref import TorchEmu

pytestmark = pytest.mark.gpu

#   nf, cells, order, directions
CASES = [(3, (3, 4, 3), 2, 4), (2, (4, 3, 3), 2, 5), (3, (1, 5, 4), 2, 5), (2, (1, 4, 6), 2, 6), (3, (3, 3, 3), 1, 4),
         (2, (3, 3, 4), 1, 5), (3, (1, 4, 5), 1, 5), (2, (1, 1, 30), 2, 5), (3, (1, 1, 140), 1, 2)]
STORES = ["default", "segment", "per_step", "per_step_sub2"]


def _rel(a, b):
    return np.linalg.norm(np.asarray(a) - np.asarray(b)) / np.linalg.norm(np.asarray(b))


def _make(nf, cells, order, ndirs):
    L = tuple(0.5 * c if c > 1 else 1.0 for c in cells)
    _, p, parts = _case("x", nf, cells, order, L, ndirs, 21 + cells[2], rho=2e7, st4_ndens=4.89e30, st4_ndensbar=3.1e30)
    return p, parts


@pytest.mark.parametrize("store", STORES)
@pytest.mark.parametrize("case", CASES, ids=lambda c: "nf%d_%s_o%d" % (c[0], "x".join(map(str, c[1])), c[2]))
@pytest.mark.parametrize("resort,before", [(1, 0), (2, 3)])
def test_gradient_matches_autograd(case, store, resort, before, monkeypatch):
    if store == "segment":
        monkeypatch.setenv("EMU_ADJOINT_FULL_STORE", "0")
    elif store != "default":
        monkeypatch.setenv("EMU_ADJOINT_STORE_MAX_BYTES", "0")
    if store == "per_step_sub2":
        monkeypatch.setenv("EMU_ADJOINT_SUBCHECKPOINT", "2")
        monkeypatch.setenv("EMU_ADJOINT_SEG_SLOTS", "3")
    p, parts = _make(*case)
    p.resort_interval = resort
    nf = p.nflavors
    with api.Context(p) as c:
        c.load_particles(parts)
        if before:
            c.evolve(before)
            parts = c.get_particles()
        dts, _ = c.adjoint_forward(7, 4)
        end = c.get_particles()
        J, lf, lN = c.adjoint_objective()
        g, gN = c.adjoint_backward(lf, lN)
        assert np.array_equal(c.get_particles(), end)
    assert dts.sum() * api.CLIGHT > 3 * 0.5   # (cells are half a centimetre wide)
    te = TorchEmu(p, parts)
    f0 = torch.tensor(parts[:, flavor_columns(nf)], requires_grad=True)
    N = torch.tensor(parts[:, number_columns(nf)], requires_grad=True)
    Jr = te.loss(f0, N, dts)
    Jr.backward()
    assert abs(J - Jr.item()) <= 1e-10 * abs(Jr.item())
    assert _rel(g, f0.grad.numpy()) < 1e-9
    assert _rel(gN, N.grad.numpy()) < 1e-9
