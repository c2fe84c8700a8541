"""phaseCorrelate when a device-side wait runs out, on the GPU.

The persistent column pass (more column tiles than SMs) waits, bounded, for
each tile's copy.  Fault injection on the host leaves the first copies
unissued, so the waits run out after 1 ms: every way to call phaseCorrelate
says so instead of giving a shift, and the same context and server give the
right one again afterwards."""
from __future__ import annotations

import math

import numpy as np
import pytest

import glscv_gb300 as g
from tests.gpu_util import stream_handle

pytestmark = pytest.mark.gpu

TIMEOUT = 8  # GLSFFT_ERROR_TIMEOUT
LIMIT_NS = 1_000_000
SHAPES = [(1024, 2048), (2048, 1024), (4096, 512)]  # 256 tiles each


@pytest.fixture()
def tctx(native, torch_cuda):
    c = g.Context(0)
    yield c
    c.close()


def _pair(shape):
    a = np.random.default_rng(21).uniform(0, 1, shape).astype(np.float32)
    return a, np.roll(a, (4, -9), axis=(0, 1))


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("calls", [1, 20])
def test_synchronous_call_reports_timeout(tctx, torch_cuda, shape, calls):
    """Launched directly and, after many calls, replayed as a graph."""
    torch = torch_cuda
    a, b = (torch.from_numpy(x).cuda() for x in _pair(shape))
    call = lambda: tctx.phase_correlate(a.data_ptr(), b.data_ptr(), None, *shape, 5,  # noqa: E731
                                        stream_handle(torch))
    for _ in range(calls):
        good = call()
    tctx.inject_stall(LIMIT_NS)
    for _ in range(calls):
        with pytest.raises(g.GlsError) as e:
            call()
        assert e.value.status == TIMEOUT
    with pytest.raises(g.GlsError):  # no surface of a call that failed
        tctx.copy_surface(a.data_ptr(), a.numel(), stream_handle(torch))
    tctx.inject_stall(0)
    assert call() == good
    assert tctx.device_status(clear=True) == TIMEOUT
    assert call() == good and tctx.device_status() == 0


@pytest.mark.parametrize("shape", SHAPES)
def test_asynchronous_result_says_so(tctx, torch_cuda, shape):
    torch = torch_cuda
    a, b = (torch.from_numpy(x).cuda() for x in _pair(shape))
    res = torch.zeros(5, dtype=torch.float64, device="cuda")

    def call():
        tctx.phase_correlate_async(a.data_ptr(), b.data_ptr(), None, *shape, 5, res.data_ptr(),
                                   stream_handle(torch))
        torch.cuda.synchronize()
        return res.tolist()

    good = call()
    tctx.inject_stall(LIMIT_NS)
    dx, dy, response, index, value = call()
    assert index == -1 and all(math.isnan(v) for v in (dx, dy, response, value))
    tctx.inject_stall(0)
    assert call() == good
    assert tctx.device_status(clear=True) == TIMEOUT


@pytest.mark.parametrize("shape", SHAPES)
def test_server_request_fails(tctx, torch_cuda, shape):
    torch = torch_cuda
    a, b = _pair(shape)
    ref, frame = torch.from_numpy(a).cuda(), torch.from_numpy(b).pin_memory()
    with g.Server(tctx, slots=4, hbm_budget=1 << 28) as srv:
        rid = srv.add_reference(ref.data_ptr(), None, *shape)
        good = srv.wait(srv.submit(rid, frame.data_ptr()))[0]
        tctx.inject_stall(LIMIT_NS)
        for ticket in [srv.submit(rid, frame.data_ptr()) for _ in range(3)]:
            with pytest.raises(g.GlsError) as e:
                srv.wait(ticket)
            assert e.value.status == TIMEOUT
        tctx.inject_stall(0)
        assert srv.wait(srv.submit(rid, frame.data_ptr()))[0] == good
        assert srv.stats()["failed"] == 3
    assert tctx.device_status() == 0  # a server's waits are its requests' own
