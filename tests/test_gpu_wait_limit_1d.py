"""The bounded waits of the kernels that take small 1D FP64 problems (several
steps per launch, recorded runs, the stored adjoint's sweep) run out without
faulting the GPU, as test_gpu_wait_limit's of the whole-step kernel.  A limit
of 0 polls makes every CTA but the last to arrive give up: the call reports
EMU_ERR_TIMEOUT although more launches are queued behind the one that timed
out, and with the default limit a fresh load matches the oracle."""
import numpy as np
import pytest

from emu_b200 import api
from emu_b200 import workloads as W
from oracle.oracle import Oracle
from tests.helpers import colwise_rel

pytestmark = pytest.mark.gpu


def _params(resort):
    p = W.c2_fast_flavor_1d(ncell_z=40, ndirs=20)    # 800 particles: 13 CTAs
    p.resort_interval = resort
    return p


def _clean(c, p, parts, n):
    ref, t_ref, _, _ = Oracle(p).evolve(parts, n)
    c.load_particles(parts)
    info = c.evolve(n)
    assert info.status == 0 and info.steps_done == n
    assert abs(info.time - t_ref) <= 1e-12 * t_ref
    assert colwise_rel(c.get_particles(), ref) < 1e-11


@pytest.mark.parametrize("resort", [0, 1, 4])
def test_steps(resort):
    p = _params(resort)
    parts = api.init_particles(p)
    with api.Context(p) as c:
        c.load_particles(parts)
        c.set_wait_limit(0)
        with pytest.raises(api.EmuError) as e:
            c.evolve(9)
        assert e.value.code & api.EMU_ERR_TIMEOUT
        with pytest.raises(api.EmuError) as e:
            c.step(1e-13)
        assert e.value.code & api.EMU_ERR_TIMEOUT
        c.set_wait_limit(-1)
        _clean(c, p, parts, 9)


def test_a_run_that_timed_out_takes_no_further_steps():
    p = _params(2)
    parts = api.init_particles(p)
    with api.Context(p) as c:
        c.load_particles(parts)
        c.evolve_begin(0.0, float("inf"), 20)
        c.evolve_steps(5)
        c.synchronize()
        c.set_wait_limit(0)
        c.evolve_steps(6)
        c.set_wait_limit(-1)
        c.evolve_steps(4)
        info = c.evolve_end()
        assert info.status & api.EMU_ERR_TIMEOUT and info.steps_done == 5
        assert info.time > 0.0
        _clean(c, p, parts, 9)


def test_recorded_run_and_sweep():
    p = _params(2)
    parts = api.init_particles(p)
    with api.Context(p) as c:
        c.load_particles(parts)
        assert c.adjoint_reserve(9, 3)[1] == 2
        c.adjoint_forward(9, 3)
        _, lf, lN = c.adjoint_objective()
        want = c.adjoint_backward(lf, lN)
        c.set_wait_limit(0)
        with pytest.raises(api.EmuError) as e:
            c.adjoint_backward(lf, lN)
        assert e.value.code & api.EMU_ERR_TIMEOUT
        # the recorded run stands: the sweep again
        c.set_wait_limit(-1)
        for a, b in zip(c.adjoint_backward(lf, lN), want):
            assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()
        c.load_particles(parts)
        c.set_wait_limit(0)
        with pytest.raises(api.EmuError) as e:
            c.adjoint_forward(9, 3)
        assert e.value.code & api.EMU_ERR_TIMEOUT
        c.set_wait_limit(-1)
        _clean(c, p, parts, 9)
