"""Which path a batch plan takes, on the GPU: batched pass launches or the
persistent kernel, and what depends on it."""
from __future__ import annotations

import numpy as np
import pytest

import glscv_gb300 as g
from glscv_gb300 import workloads as wl
from tests.gpu_util import stream_handle
from tests.test_batch_gpu import DIRECT_PLANS, _run_batch

pytestmark = pytest.mark.gpu

INV, SCALE, SHIFT = 1, 2, 64


@pytest.fixture()
def tctx(native, torch_cuda):
    c = g.Context(0)
    yield c
    c.close()


def _scattered(n, img):
    """Byte offsets of n images, no three evenly spaced: more runs than a plan
    of pass launches has."""
    offs, end = [], 0
    for i in range(n):
        offs.append(end)
        end += img + 16 * (i + 1) * (i + 1)
    return offs, end


def _plans(ctx, torch, n=20, side=64):
    """A plan of evenly spaced images and one of scattered ones, same sizes."""
    img = side * side * 8
    plans = []
    for offs, end in (([i * img for i in range(n)], n * img), _scattered(n, img)):
        src, dst = (torch.zeros(end // 8, dtype=torch.complex64, device="cuda") for _ in range(2))
        b = g.Batch(ctx, [src.data_ptr() + o for o in offs], [dst.data_ptr() + o for o in offs],
                    [(side, side)] * n, (0,))
        plans.append((b, src, dst))
    return plans


@pytest.mark.parametrize("first", [0, 1])
def test_cached_tuning_is_for_the_same_path(tctx, torch_cuda, tmp_path, first):
    """The default schedule of evenly spaced images is other code than that of
    scattered ones, so one's cached tuning is not applied to the other."""
    s, cache = stream_handle(torch_cuda), str(tmp_path / "plans.jsonl")
    plans = _plans(tctx, torch_cuda)
    order = [plans[first][0], plans[1 - first][0]]
    assert not order[0].autotune(cache, reps=1, stream=s)["from_cache"]
    assert not order[1].autotune(cache, reps=1, stream=s)["from_cache"]
    for b, *_ in _plans(tctx, torch_cuda):
        assert b.autotune(cache, reps=1, stream=s)["from_cache"]
        b.close()
    for b, *_ in plans:
        b.close()


PERSISTENT = {"nine sizes", "narrow images, few and many", "very narrow images"}


@pytest.mark.parametrize("name", DIRECT_PLANS)
@pytest.mark.parametrize("flags", [(0, INV | SCALE), (SHIFT,)])
def test_path_of_the_default_schedule(tctx, torch_cuda, name, flags):
    """Which plans take the pass launches, and that a schedule, the stall
    injection and the statistics bring the persistent kernel back."""
    shapes, gap = DIRECT_PLANS[name]
    offs, end = [], 0
    for r, c in shapes:
        offs.append(end)
        end += r * c * 8 + gap
    x = torch_cuda.zeros(end // 8, dtype=torch_cuda.complex64, device="cuda")
    ptrs = [x.data_ptr() + o for o in offs]
    for pin in (None, lambda b: b.set_variant(3), lambda b: b.set_schedule(1, 0, 0),
                lambda b: b.set_stats(True)):
        b = g.Batch(tctx, ptrs, ptrs, shapes, flags)
        if pin:
            pin(b)
        assert b.uses_launches() == (pin is None and name not in PERSISTENT)
        b.close()


@pytest.mark.parametrize("variants", [(3, 3), (3, None), (None, 3)])
def test_plans_of_either_path_side_by_side(tctx, torch_cuda, variants):
    """Two plans on two streams at once: two persistent launches sized for the
    whole GPU (blocks of the second start as the first's retire, and dynamic
    claiming keeps both correct), or one beside pass launches."""
    torch = torch_cuda
    shapes = ([(512, 512)] * 24, wl.batch_sizes(48, seed=5))
    plans, keep, outs, refs = [], [], [], []
    for k, (sh, variant) in enumerate(zip(shapes, variants)):
        if variant is None:  # evenly spaced, 48 MiB: the pass launches
            sh = [(512, 512)] * 24
            buf = torch.from_numpy(wl.complex_uniform(24 * 512, 512, 1900 + k)).cuda()
            out = torch.zeros_like(buf)
            at = lambda t: [t.data_ptr() + i * 512 * 512 * 8 for i in range(24)]  # noqa: E731
            b = g.Batch(tctx, at(buf), at(out), sh, (0, INV | SCALE))
            b.execute(stream_handle(torch))
            keep.append(buf)
            outs.append([out])
        else:
            b, _, d_in, d_out, _ = _run_batch(tctx, torch, sh, (0, INV | SCALE),
                                              seed0=1700 + 100 * k, variant=variant)
            keep.append(d_in)
            outs.append(d_out)
        torch.cuda.synchronize()
        assert b.uses_launches() == (variant is None)
        plans.append(b)
        refs.append([d.cpu().numpy().copy() for d in outs[-1]])
        for d in outs[-1]:
            d.zero_()
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in plans]
    for _ in range(3):
        for b, s in zip(plans, streams):
            b.execute(s.cuda_stream)
    torch.cuda.synchronize()
    for b, s, out, ref in zip(plans, streams, outs, refs):
        assert b.status(s.cuda_stream) == 0
        for d, want in zip(out, ref):
            assert np.array_equal(d.cpu().numpy().view(np.uint32), want.view(np.uint32))
        b.close()
