"""vgb_primary_beam's one-launch kernel against the three-kernel path.

Up to 2048 tiles and 304 (frequency, pointing) pairs one launch finds the
distinct delay sets, evaluates them and writes every tile; more take three
launches. The operations on a value
are the same, so appending tiles past 2048 must leave the first tiles' matrices
unchanged bit for bit: one tile, all tiles alike, all different, a dead tile,
one and several (frequency, pointing) pairs per block with a ragged last one.
"""
from __future__ import annotations

import numpy as np
import pytest

from helpers import dev, torch_cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ntile,nsets,npnt,nfreq,pa", [
    (1, 1, 1, 1, True), (1, 1, 153, 1, False), (17, 17, 5, 3, True), (128, 3, 8, 1, True), (128, 1, 152, 2, True), (128, 2, 305, 1, True),
    (257, 200, 9, 1, False), (2048, 40, 3, 1, True),
])
def test_one_launch_equals_three(ntile, nsets, npnt, nfreq, pa):
    import vgb

    torch = torch_cuda()
    rng = np.random.default_rng(ntile + npnt)
    sets = rng.integers(0, 32, (nsets, 16)).astype(np.uint32)
    sets[0, 5] = 32                                   # a dead dipole
    if nsets > 2:
        sets[1] = 32                                  # a dead tile
    delays = sets[rng.integers(0, nsets, ntile)]
    more = np.concatenate([delays, sets[rng.integers(0, nsets, 2049)]])
    az = dev(rng.uniform(0, 2 * np.pi, npnt))
    za = dev(np.r_[0.0, rng.uniform(0, 1.2, npnt - 1)])
    f = dev(rng.uniform(80e6, 300e6, nfreq))
    B = []
    for d in (delays, more):
        out = torch.full((nfreq, npnt, len(d), 8), float("nan"), dtype=torch.float64, device="cuda")
        vgb.primary_beam(az, za, f, dev(d), out, pa_correction=pa)
        B.append(out[:, :, :ntile])
    assert torch.equal(B[0], B[1])
    assert not torch.isnan(B[0]).any()
