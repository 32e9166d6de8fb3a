"""Two flavors along z beyond one CTA per SM with fewer and with more than two
particles a cell: the stage kernels on full and on combined meshes.  Evolve,
single steps, a recorded run, and one context that loads both in turn, against
the oracle (1e-11 normwise; the mesh per field)."""
import numpy as np
import pytest

from emu_b200 import api
from oracle.oracle import Oracle
from tests.golden.make_golden import _case
from tests.helpers import colwise_rel, magnitude_mesh

pytestmark = pytest.mark.gpu


def test_loads_on_both_sides_of_the_line():
    nz = 20000
    _, p, parts = _case("x", 2, (1, 1, nz), 2, (1.0, 1.0, 0.5 * nz), 3, 95, rho=2e9, maxError=1e-2)
    o = Oracle(p)
    with api.Context(p) as c:
        for n in (39990, 60000, 39999, 40000, 39000):
            ref = parts[:n].copy()
            mag = np.abs(magnitude_mesh(o, ref).reshape(3 + 32, -1)[3:]).reshape(8, -1).max(axis=1)

            def check(mesh):
                got = c.get_mesh().reshape(3 + 32, -1)[3:]
                err = np.abs(got - mesh.reshape(3 + 32, -1)[3:]).reshape(8, -1).max(axis=1)
                assert (err <= 1e-11 * mag).all() and colwise_rel(c.get_particles(), ref) < 1e-11

            c.load_particles(ref)
            mesh = o.deposit(ref)
            check(mesh)
            vv = o.vvac_max(ref)
            dt, _ = o.compute_dt(mesh, vv)
            for _ in range(2):
                mesh = o.rk_step(ref, dt, nthreads=4)[0]
                dt, _ = o.compute_dt(mesh, vv)
            assert c.evolve(2).steps_done == 2
            check(mesh)
            mesh = o.rk_step(ref, dt, nthreads=4)[0]
            c.step(dt)
            check(mesh)
            dts, _ = c.adjoint_forward(2, 1)
            for d in dts:
                mesh = o.rk_step(ref, d, nthreads=4)[0]
            check(mesh)
