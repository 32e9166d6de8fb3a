"""Gradients on one context that loads many, few and many particles again:
whether a run is recorded whole depends on the number loaded, while the
context's capacity stays at the largest.  Each against a context of its own,
to the adjoint's 1e-9 normwise."""
import numpy as np
import pytest

from emu_b200 import api
from tests.golden.make_golden import _case

pytestmark = pytest.mark.gpu


def _gradient(c, parts):
    c.load_particles(parts)
    c.adjoint_forward(3, 2)
    J, lf, lN = c.adjoint_objective()
    return (J,) + c.adjoint_backward(lf, lN)


#   1D beyond 256 particles per SM and within; 3D beyond and within a co-resident grid
@pytest.mark.parametrize("nf,cells,ndirs", [(2, (1, 1, 200), 200), (3, (1, 1, 200), 200), (2, (10, 10, 10), 80)])
@pytest.mark.parametrize("sequence", [(0, 700, 0), (700, 0, 700)])
def test_gradients_after_loads_of_other_counts(nf, cells, ndirs, sequence):
    L = tuple(0.5 * c if c > 1 else 1.0 for c in cells)
    _, p, parts = _case("x", nf, cells, 2, L, ndirs, 33, rho=2e9)
    with api.Context(p) as shared:
        shared.load_particles(parts)   # (the capacity)
        for n in sequence:
            q = parts[:n].copy() if n else parts
            got = _gradient(shared, q)
            with api.Context(p) as own:
                want = _gradient(own, q)
            for a, b in zip(got, want):
                assert np.abs(np.asarray(a) - b).max() <= 1e-9 * np.abs(b).max()
