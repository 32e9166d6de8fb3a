"""Small 1D FP64 problems on a stream that may use a part of the SMs only (a
green context): the grid of the several-step kernel cannot be co-resident
there and its launch is refused, so the stage kernels take the steps, from the
first one or from the step at which the stream was changed.  Evolve, steps
driven by the host, a profiled step and a recorded run, against the oracle
(1e-11 normwise) and the same gradient without the partition (1e-9)."""
import numpy as np
import pytest
import torch

from emu_b200 import api
from emu_b200 import workloads as W
from oracle.oracle import Oracle
from tests.helpers import colwise_rel

driver = pytest.importorskip("cuda.bindings.driver")
pytestmark = pytest.mark.gpu

SMS = 16


def _ok(r):
    assert int(r[0]) == 0, r
    return r[1:] if len(r) > 2 else r[1] if len(r) == 2 else None


@pytest.fixture(scope="module")
def partition():
    """a stream that may use SMS multiprocessors"""
    torch.zeros(1, device="cuda")
    dev = _ok(driver.cuDeviceGet(torch.cuda.current_device()))
    sms = _ok(driver.cuDeviceGetDevResource(dev, driver.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    group = _ok(driver.cuDevSmResourceSplitByCount(1, sms, 0, SMS))[0][0]
    ctx = _ok(driver.cuGreenCtxCreate(_ok(driver.cuDevResourceGenerateDesc([group], 1)), dev,
                                      driver.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    stream = _ok(driver.cuGreenCtxStreamCreate(ctx, driver.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
    yield int(stream)
    _ok(driver.cuStreamDestroy(stream))
    _ok(driver.cuGreenCtxDestroy(ctx))


def _cases():
    # (the third fits the partition)
    return [("nf2", W.c2_fast_flavor_1d(ncell_z=64, ndirs=80)),
            ("nf3", W.c3_three_flavor_1d(ncell_z=256, nphi_equator=16, mixed=False)),
            ("small", W.c2_fast_flavor_1d(ncell_z=16, ndirs=12))]


@pytest.mark.parametrize("name,p", _cases(), ids=[c[0] for c in _cases()])
@pytest.mark.parametrize("resort", [-1, 3])
def test_steps_on_a_partition(name, p, resort, partition):
    p.resort_interval = resort
    parts = api.init_particles(p)
    ref, t, dts, _ = Oracle(p).evolve(parts, 7)
    with api.Context(p) as c:
        c.load_particles(parts)
        c.evolve_begin(0.0, float("inf"), 7)
        c.evolve_steps(2)
        c.set_stream(partition)
        c.evolve_steps(4)
        c.profile_step()
        info = c.evolve_end()
        assert info.status == 0 and info.steps_done == 7 and abs(info.time - t) <= 1e-12 * t
        assert colwise_rel(c.get_particles(), ref) < 1e-11
        c.load_particles(parts)
        for dt in dts:
            c.step(dt)
        assert colwise_rel(c.get_particles(), ref) < 1e-11
        c.load_particles(parts)
        info = c.evolve(7)
        assert info.steps_done == 7 and colwise_rel(c.get_particles(), ref) < 1e-11
        c.load_particles(parts)
        c.evolve_begin(0.0, float("inf"), 7)
        c.profile_step()
        c.evolve_steps(6)
        assert c.evolve_end().steps_done == 7 and colwise_rel(c.get_particles(), ref) < 1e-11


@pytest.mark.parametrize("store", ["default", "per_step"])
def test_gradient_on_a_partition(store, partition, monkeypatch):
    if store == "per_step":
        monkeypatch.setenv("EMU_ADJOINT_STORE_MAX_BYTES", "0")
    p = W.c3_three_flavor_1d(ncell_z=128, nphi_equator=16, mixed=False)
    p.maxError = 1e-2
    parts = api.init_particles(p)
    out = []
    for stream in (None, partition):
        with api.Context(p) as c:
            if stream:
                c.set_stream(stream)
            c.load_particles(parts)
            c.adjoint_forward(7, 3)
            J, lf, lN = c.adjoint_objective()
            out.append((c.get_particles(), J) + c.adjoint_backward(lf, lN))
    for a, b in zip(*out):
        assert np.abs(np.asarray(a) - b).max() <= 1e-9 * np.abs(b).max()
