"""The phase normalisation's quotients where one part of the cross spectrum is
tiny beside the other, on the GPU: correctly rounded, bit for bit.

Both images are small pulses; the second has an odd pair of tiny values next to
its pulse.  Every value of the cross spectrum is then (m, +-t) or (m, 0) with m
about 2^-48, whose square keeps every bit that counts, and t down to the
smallest normal numbers; the odd part of the surface is 8 t / m beside the
centre: sums that cancel exactly and powers of two leave the quotient's own
rounding."""
from __future__ import annotations

import numpy as np
import pytest

from tests.gpu_util import gpu_phase_correlate

pytestmark = pytest.mark.gpu

F32 = np.float32


@pytest.mark.parametrize("exponent", [-102, -100, -96, -60])
def test_quotient_of_a_tiny_component(ctx, torch_cuda, exponent):
    rng = np.random.default_rng(31)
    p = F32(2.0 ** -24)
    for pulse, odd in rng.uniform(1, 2, (24, 2)).astype(F32):
        eps = odd * F32(2.0 ** exponent)
        a, b = np.zeros((4, 4), F32), np.zeros((4, 4), F32)
        a[0, 0], b[0, 0] = pulse * p, p
        b[0, 1], b[0, 3] = eps, -eps
        _, _, surf = gpu_phase_correlate(ctx, torch_cuda, a, b, None, 5, want_surface=True)
        m, t = a[0, 0] * p, a[0, 0] * (F32(2) * eps)
        assert t > np.finfo(F32).tiny and np.sqrt(m * m) == m
        q = t / m  # IEEE division
        assert surf[2, 2] == 16
        assert abs(surf[2, 1]) == F32(8) * q and surf[2, 3] == -surf[2, 1], (pulse, odd, surf[2])
