"""vgb_primary_beam with many distinct delay sets (dead dipoles make most tiles of
an array differ): the sets are shared out over blocks.

The same bits as the three-kernel path (taken when tiles past 2048 are appended)
where sets, shares and pairs leave remainders; and about as fast with every tile
different as with three sets. 128 tiles take 8 rounds of 16 lanes' dipoles in
one block but one round in 8 blocks, and a round is a small part of the call, so
a factor of 3 lies well above the shared form and well below the serial one (7);
for 2,048 tiles, of which a block also has to tell which differ, 10 (serial: 45)."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import dev, torch_cuda

pytestmark = pytest.mark.gpu


def case(ntile, nsets, npnt, nfreq):
    rng = np.random.default_rng(ntile + nsets)
    sets = rng.integers(0, 32, (nsets, 16)).astype(np.uint32)
    sets[rng.random(sets.shape) < 0.05] = 32          # dead dipoles
    sets[:, 15] = np.arange(nsets) % 31               # all different with the next
    sets[:, 14] = np.arange(nsets) // 31 % 31
    sets[:, 13] = np.arange(nsets) // 961
    order = np.r_[np.arange(nsets), rng.integers(0, nsets, ntile - nsets)]
    rng.shuffle(order)
    return (dev(rng.uniform(0, 2 * np.pi, npnt)), dev(np.r_[0.0, rng.uniform(0, 1.2, npnt - 1)]),
            dev(rng.uniform(80e6, 300e6, nfreq)), sets[order])


@pytest.mark.parametrize("ntile,nsets,npnt,nfreq", [(128, 128, 8, 1), (128, 100, 7, 3), (300, 17, 1, 2), (193, 193, 2, 1),
                                                    (2047, 2047, 1, 1), (33, 16, 153, 1), (50, 49, 19, 16)])
@pytest.mark.parametrize("pa", [True, False])
def test_shared_sets_equal_three_kernels(ntile, nsets, npnt, nfreq, pa):
    import vgb

    torch = torch_cuda()
    az, za, f, delays = case(ntile, nsets, npnt, nfreq)
    B = []
    for d in (delays, np.concatenate([delays, np.resize(delays, (2049, 16))])):
        out = torch.full((nfreq, npnt, len(d), 8), float("nan"), dtype=torch.float64, device="cuda")
        vgb.primary_beam(az, za, f, dev(d), out, pa_correction=pa)
        B.append(out[:, :, :ntile])
    assert torch.equal(B[0], B[1])


@pytest.mark.parametrize("ntile,npnt,factor", [(128, 8, 3.0), (2048, 1, 10.0)])
def test_time_with_all_tiles_different(ntile, npnt, factor):
    import vgb

    torch = torch_cuda()
    us = []
    for nsets in (3, ntile):
        az, za, f, delays = case(ntile, nsets, npnt, 1)
        d, B = dev(delays), torch.empty((npnt, ntile, 8), dtype=torch.float64, device="cuda")
        times = []
        for _ in range(10):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            torch.cuda.synchronize()
            a.record()
            for _ in range(20):
                vgb.primary_beam(az, za, f, d, B)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b) * 50)
        us.append(min(times))
    assert us[1] < factor * us[0], us
