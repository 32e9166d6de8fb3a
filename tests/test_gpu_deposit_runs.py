"""The FP64 full deposit chooses by particles per cell between matrix products
and lanes that sum run by run: the deposit of a load, of emu_deposit and the
stage-4 mesh of single steps on both sides of each line, against the oracle
(1e-13 of the summed magnitudes per field for a deposit, the FP64 parity
tolerance of 1e-11 after steps).  Single steps of a host at the automatic
interval, whose re-sort may wait for the particles to move, among them."""
import numpy as np
import pytest

from emu_b200 import api
from oracle.oracle import Oracle
from tests.golden.make_golden import _case
from tests.helpers import colwise_rel, magnitude_mesh

pytestmark = pytest.mark.gpu

#   nf, cells, order, particles per cell around the line
CASES = [(2, (4, 5, 3), 2, (2, 11, 12, 13)), (3, (3, 4, 4), 2, (2, 12, 30)), (2, (1, 6, 7), 2, (2, 5, 6, 7)),
         (3, (1, 7, 5), 2, (2, 6, 9)), (2, (4, 3, 5), 1, (2, 6, 20)), (3, (4, 3, 3), 1, (5, 6)),
         (2, (1, 1, 40), 2, (2, 63, 64, 70)), (3, (1, 1, 40), 2, (2, 130)), (2, (40, 1, 1), 2, (2, 6, 40)),
         (3, (1, 5, 4), 0, (3, 8))]


def _close(mesh, ref, mag, nh, tol):
    err = np.abs(mesh - ref).reshape(3 + 8 * nh, -1)[3:].reshape(8, -1).max(axis=1)
    scale = np.abs(mag.reshape(3 + 8 * nh, -1)[3:]).reshape(8, -1).max(axis=1)
    return (err <= tol * scale).all()


@pytest.mark.parametrize("case", CASES, ids=lambda c: "nf%d_%s_o%d" % (c[0], "x".join(map(str, c[1])), c[2]))
def test_deposits_on_both_sides(case):
    nf, cells, order, counts = case
    L = tuple(0.5 * c if c > 1 else 1.0 for c in cells)
    for q in counts:
        _, p, parts = _case("x", nf, cells, order, L, q, 17 + q, rho=2e9, maxError=1e-2)
        o = Oracle(p)
        ref, mag = o.deposit(parts), magnitude_mesh(o, parts)
        dt, _ = o.compute_dt(ref, o.vvac_max(parts))
        with api.Context(p) as c:
            c.load_particles(parts)
            assert _close(c.get_mesh(), ref, mag, nf * nf, 1e-13)
            q1 = parts.copy()
            for k in range(4):
                mesh = o.rk_step(q1, dt)[0]
                c.step(dt)
                assert _close(c.get_mesh(), mesh, mag, nf * nf, 1e-11)
            assert colwise_rel(c.get_particles(), q1) < 1e-11
            c.deposit()
            assert _close(c.get_mesh(), o.deposit(q1), mag, nf * nf, 1e-11)
            # a run goes on from a deposit, and single steps from a run
            info = c.evolve(3)
            assert info.steps_done == 3
            run, _, dts, _ = o.evolve(q1, 3)
            assert colwise_rel(c.get_particles(), run) < 1e-11
            mesh = o.rk_step(run, dt)[0]
            c.step(dt)
            assert _close(c.get_mesh(), mesh, mag, nf * nf, 1e-11)
            assert colwise_rel(c.get_particles(), run) < 1e-11


@pytest.mark.parametrize("nf,cells", [(2, (1, 1, 40)), (3, (1, 1, 12)), (2, (1, 5, 6)), (3, (3, 3, 4))])
def test_a_run_goes_on_over_a_load_and_a_deposit(nf, cells):
    L = tuple(0.5 * c if c > 1 else 1.0 for c in cells)
    _, p, a = _case("x", nf, cells, 2, L, 9, 3, rho=2e9, maxError=1e-2)
    b = a[::-1].copy()
    b[:, 0:3] = a[:, 0:3]
    b[:, 4:7] = a[:, 0:3]
    o = Oracle(p)
    with api.Context(p) as c:
        c.load_particles(a)
        c.evolve_begin(0.0, float("inf"), 9)
        c.evolve_steps(3)
        dt = c.evolve_end().dt_next
        c.load_particles(b)
        c.evolve_steps(1)
        mesh = o.rk_step(b, dt)[0]
        assert colwise_rel(c.get_particles(), b) < 1e-11
        c.deposit()
        c.evolve_steps(1)
        # (the step's dt: of the mesh that the step before it left, the load's limit)
        dt, _ = o.compute_dt(mesh, o.vvac_max(b))
        o.rk_step(b, dt)
        info = c.evolve_end()
        assert info.steps_done == 5 and colwise_rel(c.get_particles(), b) < 1e-11
