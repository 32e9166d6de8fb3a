"""Several FP64 steps per cooperative launch (k_steps_1d: 1D problems whose
grid fits on the GPU at once) vs the oracle, at the sizes where its parts
change: one CTA with its meshes in shared memory (to 128 particles and 128
cells), windows of a few cells, windows wider than the staging area (160
cells), domains narrower than a stencil, stencil orders 0 to 2, a final step
clipped to the end time, single steps.

Tolerance: the FP64 parity tolerance of a run of a few steps (1e-11 normwise
per attribute, as the other device-resident loop tests).  A mesh component
is measured against the largest summed magnitude of its field (number or a
flux, of one species): the last stage's mesh is of a state that the step has
not renormalised yet, whose components round relative to the whole matrix."""
import numpy as np
import pytest

from emu_b200 import api
from oracle.oracle import Oracle
from tests.golden.make_golden import _case
from tests.helpers import colwise_rel, flavor_cols, magnitude_mesh

pytestmark = pytest.mark.gpu

#   nf, cells, order, directions, random positions
CASES = [
    (2, 1, 2, 2, 0), (3, 1, 2, 5, 0), (2, 2, 2, 3, 0), (3, 2, 1, 4, 0), (2, 50, 2, 2, 0), (3, 64, 2, 2, 0),
    (2, 128, 2, 3, 128), (3, 128, 1, 3, 128), (2, 129, 2, 3, 128), (3, 43, 2, 3, 0), (2, 43, 0, 3, 0),
    (2, 16, 2, 33, 0), (3, 16, 1, 33, 0), (3, 11, 0, 30, 0), (2, 3, 2, 200, 0), (3, 2, 2, 150, 0),
    (2, 900, 2, 3, 300), (3, 900, 1, 3, 300), (3, 300, 2, 3, 128), (2, 160, 2, 9, 700),
]


def _make(nf, nz, order, ndirs, nrandom):
    L = (1.0, 1.0, 0.5 * nz)
    _, p, parts = _case("x", nf, (1, 1, nz), order, L, ndirs, 7 + nz, rho=2e9)
    if nrandom:
        parts = parts[:nrandom].copy()
        parts[:, 2] = np.random.default_rng(5).uniform(0.0, L[2], len(parts))
        parts[:, 6] = parts[:, 2]
    return p, parts


def _check(p, out, ref, mesh, mesh_ref, o):
    assert colwise_rel(out, ref) < 1e-11
    assert colwise_rel(out[:, flavor_cols(p.nflavors)], ref[:, flavor_cols(p.nflavors)]) < 1e-11
    nh = p.nflavors ** 2
    mag = np.abs(magnitude_mesh(o, ref).reshape(3 + 8 * nh, -1)[3:]).reshape(8, -1).max(axis=1)
    err = np.abs(mesh - mesh_ref).reshape(3 + 8 * nh, -1)[3:].reshape(8, -1).max(axis=1)
    assert (err <= 1e-11 * mag).all()


@pytest.mark.parametrize("case", CASES, ids=lambda c: "nf%d_%dcells_o%d_%d_%d" % c)
@pytest.mark.parametrize("resort", [0, 3])
def test_steps_match_oracle(case, resort):
    p, parts = _make(*case)
    p.resort_interval = resort
    o = Oracle(p)
    ref = parts.copy()
    mesh_ref = o.deposit(ref)
    vv, t = o.vvac_max(ref), 0.0
    n = 5
    for _ in range(n):
        dt, _ = o.compute_dt(mesh_ref, vv)
        mesh_ref = o.rk_step(ref, dt)[0]
        t += dt
    with api.Context(p) as c:
        c.load_particles(parts)
        info = c.evolve(n)
        assert info.status & ~(api.EMU_ERR_TRACE | api.EMU_ERR_LENGTH | api.EMU_ERR_NEGDIAG) == 0
        assert info.steps_done == n and abs(info.time - t) <= 1e-12 * t
        nxt, _ = o.compute_dt(mesh_ref, vv)
        assert abs(info.dt_next - nxt) <= 1e-11 * nxt
        _check(p, c.get_particles(), ref, c.get_mesh(), mesh_ref, o)
        # on from there: the run's start takes dt from the current state
        dt, _ = o.compute_dt(o.deposit(ref), vv)
        mesh_ref = o.rk_step(ref, dt)[0]
        info = c.evolve(1, info.time)
        assert info.steps_done == 1 and abs(info.time - (t + dt)) <= 1e-11 * t
        _check(p, c.get_particles(), ref, c.get_mesh(), mesh_ref, o)


@pytest.mark.parametrize("nf,nz,ndirs", [(2, 20, 4), (3, 40, 12)])
def test_end_time_and_single_steps(nf, nz, ndirs):
    p, parts = _make(nf, nz, 2, ndirs, 0)
    o = Oracle(p)
    vv = o.vvac_max(parts)
    dt, _ = o.compute_dt(o.deposit(parts), vv)
    end = 2.5 * dt
    ref, t_ref, dts, _ = o.evolve(parts, 10, end_time=end)
    with api.Context(p) as c:
        c.load_particles(parts)
        info = c.evolve(10, 0.0, end)
        assert info.steps_done == len(dts) and abs(info.time - end) <= 1e-12 * end
        assert colwise_rel(c.get_particles(), ref) < 1e-11
        c.load_particles(parts)
        ref2 = parts.copy()
        for _ in range(3):
            mesh_ref = o.rk_step(ref2, dt)[0]
            c.step(dt, raise_on_error=False)
        _check(p, c.get_particles(), ref2, c.get_mesh(), mesh_ref, o)
        d, _ = c.compute_dt()
        want, _ = o.compute_dt(mesh_ref, vv)
        assert abs(d - want) <= 1e-11 * want
