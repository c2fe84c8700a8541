"""The one-launch 2-D FFT of small images on the GPU: for every size it takes
(16 points a side and more, at most 4096 pixels; the largest and the thinnest
among them), every flag combination, complex and CV_32FC1 input, batches of an
odd number of images and in place, the result is bit-identical to the row pass
followed by the column pass."""
from __future__ import annotations

import numpy as np
import pytest

import glscv_gb300 as g
from glscv_gb300 import workloads as wl
from tests.gpu_util import stream_handle

pytestmark = pytest.mark.gpu

SHAPES = [(16, 16), (16, 256), (256, 16), (32, 32), (32, 64), (64, 32), (64, 64), (32, 128), (128, 32), (64, 16)]


def _two_passes(ctx, torch, d, flags):
    n, r, c = d.shape
    y = torch.empty_like(d)
    s = stream_handle(torch)
    ctx.fft_rows(d.data_ptr(), y.data_ptr(), r, c, flags, s, n)
    ctx.fft_cols(y.data_ptr(), y.data_ptr(), r, c, flags, s, n)
    return y


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("flags", range(8))
def test_one_launch_equals_two_passes(ctx, torch_cuda, shape, flags):
    torch = torch_cuda
    fl = (flags & 1) * g.DFT_INVERSE | (flags >> 1 & 1) * g.DFT_SCALE | (flags >> 2) * g.GLS_FFT_SHIFT
    s, (r, c) = stream_handle(torch), shape
    for count in (1, 5):
        x = np.stack([wl.complex_uniform(r, c, 7 * i + flags) for i in range(count)])
        d = torch.from_numpy(x).cuda()
        want = _two_passes(ctx, torch, d, fl)
        y = torch.empty_like(d)
        ctx.fft2d_batched(d.data_ptr(), y.data_ptr(), count, r, c, fl, s)
        real = torch.from_numpy(np.ascontiguousarray(x[0].real)).cuda()
        got = torch.empty_like(d[0])
        ctx.fft2d(real.data_ptr(), got.data_ptr(), r, c, fl, s, real_input=True)
        promoted = _two_passes(ctx, torch, real.to(torch.complex64)[None], fl)
        ctx.fft2d_batched(d.data_ptr(), d.data_ptr(), count, r, c, fl, s)  # in place
        torch.cuda.synchronize()
        bits = lambda t: torch.view_as_real(t).view(torch.int32)  # noqa: E731
        assert torch.equal(bits(y), bits(want))
        assert torch.equal(bits(d), bits(want))
        assert torch.equal(got, promoted[0])  # (real input: equal values, -0 as +0)
