"""FP64 RK4 stages on combined meshes (k_stage64 and its deposits) vs the
oracle, over the stencil classes (3D TSC, TSC in the y-z plane and along z,
any other stencil of at most 4 or 12 cells) and where their parts change:
domains narrower than a stencil (cells counted twice), tiles with one run of
equal stencils and with 128, particle counts around a tile, re-sorts after
every step (stage 4 scatters), now and then (stage 4 deposits at the moved
positions) and never, single steps, 1D problems beyond one CTA per SM.

Tolerance: the FP64 parity tolerance of a run of a few steps (1e-11 normwise
per attribute); a mesh component against the largest summed magnitude of its
field, as in test_gpu_steps1d."""
import numpy as np
import pytest

from emu_b200 import api
from oracle.oracle import Oracle
from tests.golden.make_golden import _case
from tests.helpers import colwise_rel, flavor_cols, magnitude_mesh

pytestmark = pytest.mark.gpu

#   nf, cells, order, directions, particles kept (0: all)
CASES = [
    (3, (4, 5, 3), 2, 9, 0), (2, (4, 5, 3), 2, 9, 0), (3, (2, 2, 2), 2, 40, 0), (2, (3, 2, 7), 2, 11, 0),
    (3, (6, 6, 6), 2, 3, 127), (3, (6, 6, 6), 2, 3, 129), (2, (9, 8, 7), 2, 4, 0), (3, (1, 1, 1), 2, 300, 0),
    (3, (1, 6, 7), 2, 13, 0), (2, (1, 6, 7), 2, 13, 0), (3, (6, 1, 5), 2, 10, 0), (2, (5, 6, 1), 2, 10, 0),
    (3, (7, 1, 1), 2, 21, 0), (2, (40, 1, 1), 2, 8, 0), (3, (4, 3, 5), 1, 12, 0), (2, (4, 3, 5), 1, 12, 0),
    (3, (1, 5, 4), 1, 12, 0), (2, (6, 1, 1), 1, 31, 0), (3, (3, 4, 2), 0, 16, 0), (2, (1, 4, 3), 0, 16, 0),
    (3, (1, 2, 2), 2, 70, 0), (2, (1, 30, 31), 2, 3, 0),
]


def _make(nf, cells, order, ndirs, keep):
    L = tuple(0.5 * c if c > 1 else 1.0 for c in cells)
    _, p, parts = _case("x", nf, cells, order, L, ndirs, 3 + cells[2], rho=2e9)
    return p, parts[:keep].copy() if keep else parts


def _check(p, out, ref, mesh, mesh_ref, o, tol=1e-11):
    nh = p.nflavors ** 2
    assert colwise_rel(out, ref) < tol
    assert colwise_rel(out[:, flavor_cols(p.nflavors)], ref[:, flavor_cols(p.nflavors)]) < tol
    mag = np.abs(magnitude_mesh(o, ref).reshape(3 + 8 * nh, -1)[3:]).reshape(8, -1).max(axis=1)
    err = np.abs(mesh - mesh_ref).reshape(3 + 8 * nh, -1)[3:].reshape(8, -1).max(axis=1)
    assert (err <= tol * mag).all()


def _run_oracle(p, parts, n):
    o = Oracle(p)
    ref = parts.copy()
    mesh = o.deposit(ref)
    vv, t = o.vvac_max(ref), 0.0
    for _ in range(n):
        dt, _ = o.compute_dt(mesh, vv)
        mesh = o.rk_step(ref, dt, nthreads=4)[0]
        t += dt
    return o, ref, mesh, t, o.compute_dt(mesh, vv)[0]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "nf%d_%s_o%d_%d_%d" % (c[0], "x".join(map(str, c[1])), *c[2:]))
@pytest.mark.parametrize("resort", [0, 1, 3])
def test_steps_match_oracle(case, resort):
    p, parts = _make(*case)
    p.resort_interval = resort
    n = 4
    o, ref, mesh_ref, t, dt_next = _run_oracle(p, parts, n)
    ok = api.EMU_ERR_TRACE | api.EMU_ERR_LENGTH | api.EMU_ERR_NEGDIAG
    with api.Context(p) as c:
        c.load_particles(parts)
        assert colwise_rel(c.get_particles(), parts) == 0.0
        info = c.evolve(n)
        assert info.status & ~ok == 0 and info.steps_done == n
        assert abs(info.time - t) <= 1e-12 * t and abs(info.dt_next - dt_next) <= 1e-11 * dt_next
        _check(p, c.get_particles(), ref, c.get_mesh(), mesh_ref, o)
        # on from there (the run's start takes dt from the current state), the
        # last steps of the call without work
        vv = o.vvac_max(parts)
        dt, _ = o.compute_dt(o.deposit(ref), vv)
        mesh_ref = o.rk_step(ref, dt)[0]
        c.evolve_begin(info.time, float("inf"), 1)
        c.evolve_steps(3)
        info = c.evolve_end()
        assert info.steps_done == 1 and abs(info.time - (t + dt)) <= 1e-11 * t
        _check(p, c.get_particles(), ref, c.get_mesh(), mesh_ref, o)
        # and single steps of a host
        for _ in range(2):
            mesh_ref = o.rk_step(ref, dt)[0]
            c.step(dt, raise_on_error=False)
        _check(p, c.get_particles(), ref, c.get_mesh(), mesh_ref, o)


@pytest.mark.parametrize("nf,nz,ndirs", [(2, 700, 55), (3, 801, 49)])
def test_wide_1d_matches_oracle(nf, nz, ndirs):
    """1D beyond one CTA per SM: the stage kernels along z"""
    p, parts = _make(nf, (1, 1, nz), 2, ndirs, 0)
    assert len(parts) > 148 * 256
    o, ref, mesh_ref, t, _ = _run_oracle(p, parts, 3)
    with api.Context(p) as c:
        c.load_particles(parts)
        info = c.evolve(3)
        assert info.steps_done == 3 and abs(info.time - t) <= 1e-12 * t
        _check(p, c.get_particles(), ref, c.get_mesh(), mesh_ref, o)


def test_end_time_clips_the_last_step():
    p, parts = _make(3, (4, 4, 4), 2, 10, 0)
    o = Oracle(p)
    dt, _ = o.compute_dt(o.deposit(parts), o.vvac_max(parts))
    end = 2.5 * dt
    ref, _, dts, _ = o.evolve(parts, 10, end_time=end)
    with api.Context(p) as c:
        c.load_particles(parts)
        info = c.evolve(10, 0.0, end)
        assert info.steps_done == len(dts) and abs(info.time - end) <= 1e-12 * end
        assert colwise_rel(c.get_particles(), ref) < 1e-11


def test_mesh_can_be_read_after_a_profiled_step():
    p, parts = _make(3, (4, 5, 3), 2, 9, 0)
    meshes = []
    for profiled in (False, True):
        with api.Context(p) as c:
            c.load_particles(parts)
            c.evolve_begin(0.0, float("inf"), 3)
            c.evolve_steps(2 if profiled else 3)
            if profiled:
                c.profile_step()
            meshes.append(c.get_mesh())
    scale = np.abs(meshes[0]).reshape(3 + 72, -1)[3:].reshape(8, -1).max(axis=1)
    err = np.abs(meshes[1] - meshes[0]).reshape(3 + 72, -1)[3:].reshape(8, -1).max(axis=1)
    assert (err <= 1e-11 * scale).all()
