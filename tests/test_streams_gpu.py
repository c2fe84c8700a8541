"""Several streams at once on the GPU, a context each.

The FFT display of a 512 x 512 frame leaves much of the device idle (128
blocks of a few KB on 152 SMs, three short launches in a row), so four streams
get well over twice one stream's calls per second, unless a launch keeps the
blocks of the others off its SMs.  Results are each stream's own."""
from __future__ import annotations

import pytest

import glscv_gb300 as g

pytestmark = pytest.mark.gpu

N, CALLS, REPLAYS = 512, 20, 10


def _display(torch, frames):
    """(us per call over a stream per frame replaying a graph of calls, results)."""
    ctxs = [g.Context(0) for _ in frames]
    streams = [torch.cuda.Stream() for _ in frames]
    out = [torch.empty_like(f) for f in frames]
    graphs = []
    for c, s, f, d in zip(ctxs, streams, frames, out):
        call = lambda: c.fft_display(  # noqa: E731
            f.data_ptr(), None, d.data_ptr(), N, N, 1.0, s.cuda_stream)
        s.wait_stream(torch.cuda.current_stream())
        call()  # the workspace
        torch.cuda.synchronize()
        graphs.append(torch.cuda.CUDAGraph())
        with torch.cuda.graph(graphs[-1], stream=s):
            for _ in range(CALLS):
                call()
    best = float("inf")
    for _ in range(8):
        torch.cuda.synchronize()
        t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        here = torch.cuda.current_stream()
        t0.record(here)
        for s in streams:
            s.wait_stream(here)
        for _ in range(REPLAYS):
            for s, gr in zip(streams, graphs):
                with torch.cuda.stream(s):
                    gr.replay()
        for s in streams:
            here.wait_stream(s)
        t1.record(here)
        torch.cuda.synchronize()
        best = min(best, 1e3 * t0.elapsed_time(t1) / (CALLS * REPLAYS * len(frames)))
    del graphs
    for c in ctxs:
        c.close()
    return best, out


def test_four_streams_share_the_sms(native, torch_cuda):
    torch = torch_cuda
    gen = torch.Generator(device="cuda").manual_seed(4)
    frames = [torch.rand(N, N, device="cuda", generator=gen) for _ in range(4)]
    alone = [_display(torch, [f]) for f in frames]
    four, out = _display(torch, frames)
    for d, (_, (want,)) in zip(out, alone):
        assert torch.equal(d, want)
    one = min(us for us, _ in alone)
    assert four < 0.48 * one, (one, four)
