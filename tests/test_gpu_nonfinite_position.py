"""A particle whose position is no number: its deposit is in the cells of one
stencil, whichever, and every other particle's deposit is its own (the deposit
by matrix products takes four particles at a time, of neighbouring runs too).
Tolerance: 1e-13 of the summed magnitudes per field, as the FP64 deposit."""
import numpy as np
import pytest

from emu_b200 import api
from oracle.oracle import Oracle
from tests.golden.make_golden import _case
from tests.helpers import magnitude_mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nf,cells,ndirs", [(2, (6, 5, 7), 20), (3, (5, 6, 5), 30), (3, (1, 9, 8), 12), (2, (1, 1, 50), 70)])
def test_a_bad_position_stays_in_one_stencil(nf, cells, ndirs):
    L = tuple(0.5 * c if c > 1 else 1.0 for c in cells)
    _, p, parts = _case("x", nf, cells, 2, L, ndirs, 71, rho=2e9, maxError=1e-2)
    o = Oracle(p)
    k = len(parts) // 3
    rest = np.delete(parts, k, axis=0)
    want = o.deposit(rest).reshape(3 + 8 * nf * nf, -1)[3:]
    mag = np.abs(magnitude_mesh(o, rest).reshape(3 + 8 * nf * nf, -1)[3:]).reshape(8, -1).max(axis=1)
    parts[k, 0:3] = np.nan
    with api.Context(p) as c:
        c.load_particles(parts)
        mesh = c.get_mesh().reshape(3 + 8 * nf * nf, -1)[3:]
    ok = np.isfinite(mesh).all(axis=0)
    assert 0 < (~ok).sum() <= 3 ** sum(n > 1 for n in cells)
    err = np.abs(mesh[:, ok] - want[:, ok]).reshape(8, -1).max(axis=1)
    assert (err <= 1e-13 * mag).all()
