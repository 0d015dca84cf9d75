"""vgb_weights' rounding to FP32 at its edges, bit for bit.

W = phi J in FP64, rounded to nearest even in integer operations where the result
is a normal number. With phi = 1 and diagonal J the products are J itself:
halfway cases of either parity and their neighbours, exponents at both ends of
FP32, values that round up to infinity or to the smallest normal number,
subnormals, zeros, infinities, NaN, and random bit patterns."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import dev, host, torch_cuda

pytestmark = pytest.mark.gpu


def values():
    rng = np.random.default_rng(3)
    m = np.r_[rng.integers(0, 1 << 23, 200), 0, 1, 2, (1 << 23) - 2, (1 << 23) - 1].astype(np.uint64)[:, None, None]
    e = np.r_[1, 2, 100, 127, 200, 253, 254].astype(np.uint64)[None, :, None] + np.uint64(896)
    low = np.array([0, 1, (1 << 28) - 1, 1 << 28, (1 << 28) + 1, (1 << 29) - 1], np.uint64)[None, None, :]  # half is 2^28
    x = ((e << np.uint64(52)) | (m << np.uint64(29)) | low).reshape(-1).view(np.float64)
    tiny = np.float64(np.finfo(np.float32).tiny)
    edge = [0.0, 1e-42, 1e-60, 5e-324, tiny, np.nextafter(tiny, 0), tiny * (1 - 2.0**-25), tiny * (1 - 2.0**-24),
            float(np.finfo(np.float32).max), 2.0**128 * (1 - 2.0**-25), np.nextafter(2.0**128 * (1 - 2.0**-25), 0), 2.0**128,
            1e300, np.inf, np.nan]
    bits = rng.integers(0, 1 << 63, 4000, dtype=np.uint64).view(np.float64)
    x = np.r_[x, edge, bits]
    return np.r_[x, -x]


def test_rounding_to_nearest_even():
    import vgb

    torch = torch_cuda()
    x = values()
    x = np.r_[x, np.zeros(-x.size % 2)]
    J = np.zeros((x.size // 2, 2, 2), np.complex128)
    J[:, 0, 0].real, J[:, 1, 1].real = x[0::2], x[1::2]
    W = torch.empty((len(J), 8), device="cuda")
    vgb.weights(dev(J), dev(np.ones(len(J), np.complex128)), len(J), W)
    torch.cuda.synchronize()
    got = host(W)[:, [0, 6]].reshape(-1)
    with np.errstate(over="ignore", under="ignore", invalid="ignore"):
        want = x.astype(np.float32)
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    zero = want == 0
    assert np.array_equal(got[zero], want[zero])
    rest = ~nan & ~zero
    assert np.array_equal(got[rest].view(np.uint32), want[rest].view(np.uint32))
