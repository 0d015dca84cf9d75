"""The fused front end's leftover tiles of 2 and 4 spectra.

Variants 4 and 8 take whole waves of 8-spectrum tiles and the spectra left over
in smaller ones; variant 5 takes 8-spectrum tiles throughout. Every value is
summed over the tiles in the same order, so the outputs are equal bit for bit:
no whole wave, exact waves (2,432 and 1,216 spectra on 152 SMs), one spectrum
more, leftovers for tiles of 2, of 4 and too many for either, several channels
whose share of a wave is not whole, odd tile counts and each overlap-add.
"""
from __future__ import annotations

import numpy as np
import pytest

import synthetic as SY
from helpers import dev, host, tables, torch_cuda, weights_on_device

pytestmark = pytest.mark.gpu
K = 128


@pytest.mark.parametrize("ncc,ns", [(1, 1), (1, 3), (3, 200), (1, 609), (1, 1216), (1, 1217), (1, 1500), (1, 2432), (1, 2433),
                                    (1, 3100), (1, 4000), (3, 1000), (2, 2465)])
@pytest.mark.parametrize("mode", ["full fp32", "full split", "smart fp32", "smart int32", "full int32"])
def test_leftover_tiles_equal_whole_ones(ncc, ns, mode):
    import vgb

    torch = torch_cuda()
    nant = 3
    rng = np.random.default_rng(ns)
    nblk = -(-ns // 500)
    volt = np.clip(np.round(rng.standard_normal((ncc, nblk + 1, 2 * nant, 64000, 2), dtype=np.float32) * 30), -128, 127).astype(np.int8)
    d = dev(volt.reshape(-1).view(np.uint8))
    v = vgb.reference_buffer_voltages(d, 2 * nant, nblk, ncc, volt[0].nbytes)
    h = SY.analysis_filter_int16()
    if "split" in mode or "int32" in mode:
        h = np.round(h * 3.6).astype(np.int32)
    flags = vgb.PFB_SMART if "smart" in mode else vgb.PFB_FULL_PRECISION
    flags |= {"fp32": vgb.WOLA_FP32, "split": vgb.WOLA_FP32_SPLIT, "int32": vgb.WOLA_INT32}[mode.split()[1]]
    W = torch.cat([weights_on_device(*tables(nant, cc=c)) for c in range(ncc)])
    out = {}
    for g in (5, 4, 8):
        S = torch.full((ncc, ns, 4, K), float("nan"), device="cuda")
        e = torch.full((ncc, ns, K, 2, 2), float("nan"), device="cuda")
        inc = torch.full((ncc, ns, K), float("nan"), device="cuda")
        prev = vgb.pfb_variant(g)
        try:
            vgb.beamform_mwax(v, ncc, ns, dev(h), flags, W, nant, 1 / 6, 4, S, e, inc)
        finally:
            vgb.pfb_variant(prev)
        torch.cuda.synchronize()
        assert vgb.check_device_status() == 0 and vgb.pfb_variant_last() == g
        out[g] = [host(x) for x in (S, e, inc)]
    for g in (4, 8):
        for x, y in zip(out[g], out[5]):
            assert not np.isnan(x).any()
            assert np.array_equal(x, y), g
