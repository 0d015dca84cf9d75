"""vgb_renormalise at the edges of its tiles, and vgb_ipfb's 33-frame CTAs.

The 8-bit stage keeps a cluster's samples in shared memory with 32, 16 or 8
channels per block (up to 2,816, 5,632 and 11,264 samples) and otherwise reads
them twice; channels not in 32s and unaligned bytes take the latter too. All
equal the oracle's sequential scan bit for bit: fewer samples than blocks, the
edges of each range, NaN first, NaN elsewhere, infinities, a constant channel,
values at the type's ends. Inverse-PFB outputs around multiples of 33 frames
match a 64-bit restatement within 1e-5 of the rms (FP32 transforms and sums).
"""
from __future__ import annotations

import numpy as np
import pytest

import synthetic as SY
from helpers import dev, host, torch_cuda

pytestmark = pytest.mark.gpu
K = 128


@pytest.mark.parametrize("nstep,nchan,shift", [(1, 32, 0), (5, 128, 0), (8, 128, 4), (63, 64, 0), (2816, 32, 0),
                                               (2817, 32, 0), (5632, 64, 0), (5640, 32, 0), (11264, 32, 0),
                                               (11272, 32, 0), (100, 24, 0), (100, 128, 1), (100, 128, 2)])
def test_renormalise_tiles(nstep, nchan, shift, oracle_mod):
    import vgb

    torch = torch_cuda()
    rng = np.random.default_rng(nstep)
    ncc, npnt, nst = 2, 2, 2
    S = (rng.standard_normal((ncc, npnt, nstep, nst, nchan)) * 100).astype(np.float32)
    S[0, 0, 0, 0, 1] = np.nan                                       # the whole channel becomes NaN
    S[0, 0, nstep // 2, 1, 2] = np.nan if nstep > 1 else 1.0        # skipped
    S[0, 1, nstep - 1, 0, 3] = np.inf
    S[1, 0, :, 0, 4] = 7.5                                          # no range
    S[1, 1, nstep // 3, 1, 5] = np.finfo(np.float32).min
    S[1, 1, nstep - 1, 1, 6] = np.finfo(np.float32).max
    S[1, 1, :, 0, 7] = np.float32(1e-42) * np.arange(nstep)         # subnormal
    out = torch.full((S.size + 64,), 0x5A, dtype=torch.uint8, device="cuda")
    off = torch.empty(ncc * npnt * nst * nchan, dtype=torch.float32, device="cuda")
    scl = torch.empty_like(off)
    per = nstep * nst * nchan
    vgb.renormalise(dev(S), ncc, npnt, nstep, nst, nchan, out[shift:], npnt * per, per, nst * nchan, nchan, off, scl)
    torch.cuda.synchronize()
    got = host(out[shift:shift + S.size]).reshape(S.shape)
    for cc in range(ncc):
        o, s, u = oracle_mod.renormalise(S[cc])
        assert np.array_equal(host(off).reshape(ncc, npnt, nst, nchan)[cc], o, equal_nan=True)
        assert np.array_equal(host(scl).reshape(ncc, npnt, nst, nchan)[cc], s, equal_nan=True)
        assert np.array_equal(got[cc], u)
    assert (host(out[:shift]) == 0x5A).all() and (host(out[shift + S.size:]) == 0x5A).all()


@pytest.mark.parametrize("ns", [1, 16, 17, 33, 34, 50, 66, 99])
def test_ipfb_frames(ns):
    import vgb

    torch = torch_cuda()
    rng = np.random.default_rng(ns)
    f = SY.synthesis_filter().astype(np.float32)
    e = (rng.standard_normal((2, 12 + ns, K, 2)) + 1j * rng.standard_normal((2, 12 + ns, K, 2))).astype(np.complex64)
    d, hist = dev(e[:, 12:]), dev(e[:, :12])
    out = torch.empty((2, ns * K, 2, 2), device="cuda")
    vd = torch.full((2 * ns + 1, 544), 0x5A, dtype=torch.uint8, device="cuda")
    vgb.ipfb(d, ns * K * 16, hist, 12 * K * 16, dev(f), ns, 2, out_f=out, vdif=vd)
    torch.cuda.synchronize()
    y = np.fft.ifft(e.astype(np.complex128), axis=2, norm="forward") * np.where(np.arange(K) % 2, -1.0, 1.0)[None, None, :, None]
    want = sum(f.reshape(12, K)[p].astype(np.float64)[None, None, :, None] * y[:, 12 - p:12 - p + ns] for p in range(12)) / K
    got = host(out).astype(np.float64)
    got = (got[..., 0] + 1j * got[..., 1]).reshape(2, ns, K, 2)
    assert np.abs(got - want).max() < 1e-5 * np.sqrt(np.mean(np.abs(want) ** 2))
    q = np.stack([got.real, got.imag], -1).reshape(2, ns, 512)
    byte = (np.rint(np.clip(q.astype(np.float32), -126, 127)).astype(np.int32) & 0xFF) ^ 0x80
    assert np.array_equal(host(vd)[:2 * ns].reshape(2, ns, 544)[..., 32:], byte.astype(np.uint8))
    assert (host(vd)[2 * ns:] == 0x5A).all()
