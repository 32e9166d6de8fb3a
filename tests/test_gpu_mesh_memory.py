"""The FP64 paths on combined meshes hold no more device memory than those on
four full meshes (fused = 2): the combined meshes live in three of them.  And
the mesh that a caller reads is right where the two share memory: after a
load, runs, single steps, a deposit, a recorded run, an objective and a sweep
in any order, against the oracle (1e-11 of the summed magnitudes per field)."""
import numpy as np
import pytest
import torch

from emu_b200 import api
from oracle.oracle import Oracle
from tests.golden.make_golden import _case
from tests.helpers import colwise_rel, magnitude_mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nf,cells", [(2, (64, 64, 64)), (3, (64, 64, 64)), (3, (1, 1, 30000))])
def test_memory_is_that_of_four_full_meshes(nf, cells):
    L = tuple(0.5 * c if c > 1 else 1.0 for c in cells)
    _, p, parts = _case("x", nf, (1, 1, 4), 2, L, 30, 5, rho=2e9)
    api.set_param(p, "ncell", cells)
    used = {}
    for fused in (2, 1, 2, 1):
        p.fused = fused
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        with api.Context(p) as c:
            c.load_particles(parts)
            c.evolve(1)
            used[fused] = free - torch.cuda.mem_get_info()[0]
    # (a step graph and the like: a few MB whatever the mesh)
    assert used[1] <= used[2] + (16 << 20)


@pytest.mark.parametrize("store", ["default", "per_step"])
@pytest.mark.parametrize("nf,cells,ndirs", [(2, (1, 1, 50), 6), (3, (1, 1, 140), 2), (2, (3, 4, 3), 14), (3, (3, 3, 4), 9),
                                            (2, (1, 5, 6), 8), (2, (1, 1, 2), 3)])
def test_meshes_in_any_order(nf, cells, ndirs, store, monkeypatch):
    if store != "default":
        monkeypatch.setenv("EMU_ADJOINT_STORE_MAX_BYTES", "0")
    L = tuple(0.5 * c if c > 1 else 1.0 for c in cells)
    _, p, ref = _case("x", nf, cells, 2, L, ndirs, 81, rho=2e9, maxError=1e-2)
    o = Oracle(p)
    mag = np.abs(magnitude_mesh(o, ref).reshape(3 + 8 * nf * nf, -1)[3:]).reshape(8, -1).max(axis=1)

    def check(c, mesh):
        got = c.get_mesh().reshape(3 + 8 * nf * nf, -1)[3:]
        err = np.abs(got - mesh.reshape(3 + 8 * nf * nf, -1)[3:]).reshape(8, -1).max(axis=1)
        assert (err <= 1e-11 * mag).all()
        assert colwise_rel(c.get_particles(), ref) < 1e-11

    dt, _ = o.compute_dt(o.deposit(ref), o.vvac_max(ref))
    rng = np.random.default_rng(7)
    with api.Context(p) as c:
        c.load_particles(ref)
        lam = None
        for what in ["load"] + list(rng.permutation(["evolve", "step", "deposit", "record", "sweep", "dt"] * 4)):
            if what == "load":
                mesh = o.deposit(ref)
            elif what == "evolve":
                ref = ref.copy()
                vv = o.vvac_max(ref)
                d, _ = o.compute_dt(o.deposit(ref), vv)
                for _ in range(2):
                    mesh = o.rk_step(ref, d)[0]
                    d, _ = o.compute_dt(mesh, vv)
                c.evolve(2)
                lam = None
            elif what == "step":
                mesh = o.rk_step(ref, dt)[0]
                c.step(dt)
                lam = None
            elif what == "deposit":
                mesh = o.deposit(ref)
                c.deposit()
            elif what == "record":
                dts, _ = c.adjoint_forward(3, 2)
                for d in dts:
                    mesh = o.rk_step(ref, d)[0]
                lam = c.adjoint_objective()[1:]
            elif what == "sweep" and lam is not None:
                c.adjoint_backward(*lam)
                mesh = o.deposit(ref)
            elif what == "dt":
                d, _ = c.compute_dt()
                want, _ = o.compute_dt(mesh, o.vvac_max(ref))
                assert abs(d - want) <= 1e-11 * want
            check(c, mesh)
