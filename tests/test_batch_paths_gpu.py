"""Which path a batch plan takes, on the GPU: batched pass launches or the
persistent kernel, and what depends on it."""
from __future__ import annotations

import pytest

import glscv_gb300 as g
from tests.gpu_util import stream_handle

pytestmark = pytest.mark.gpu

INV, SCALE = 1, 2


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
