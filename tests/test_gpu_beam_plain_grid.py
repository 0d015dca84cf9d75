"""The fused front end's leftover tiles against the plain grid of whole ones.

Variants 4, 5 and 8 take whole waves of 8-spectrum tiles and the spectra left
over in smaller ones: of 2 (variant 4), of 4 (8) and of 4 or 6 (5). Variant 3
takes 8-spectrum tiles only, one block each, and sums every value over the tiles
in the same order, so all four give the same bits. Sizes on 152 SMs: no whole
wave, exact ones (1,216, 2,432 and 3,648 spectra), one spectrum more, leftovers
for each small tile and too many for it, channels whose share of a wave is not
whole; an odd tile count."""
from __future__ import annotations

import numpy as np
import pytest

import synthetic as SY
from helpers import dev, tables, torch_cuda, weights_on_device

pytestmark = pytest.mark.gpu
K = 128


@pytest.mark.parametrize("ncc,ns", [(1, 1), (1, 3), (3, 200), (1, 609), (1, 1216), (1, 1217), (1, 1500), (1, 1825), (1, 2000), (1, 2432),
                                    (1, 2433), (1, 3100), (1, 3648), (1, 3649), (1, 4000), (1, 5700), (3, 1000), (2, 2465)])
@pytest.mark.parametrize("mode", ["full fp32", "full split", "smart fp32", "smart int32", "full int32"])
def test_variants_equal_plain_grid(ncc, ns, mode):
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
    want = None
    for g in (3, 4, 5, 8):
        out = [torch.full(shape, float("nan"), device="cuda") for shape in ((ncc, ns, 4, K), (ncc, ns, K, 2, 2), (ncc, ns, K))]
        prev = vgb.pfb_variant(g)
        try:
            vgb.beamform_mwax(v, ncc, ns, dev(h), flags, W, nant, 1 / 6, 4, *out)
        finally:
            vgb.pfb_variant(prev)
        torch.cuda.synchronize()
        assert vgb.check_device_status() == 0 and vgb.pfb_variant_last() == g
        assert not any(torch.isnan(x).any() for x in out)
        want = want or out
        assert all(torch.equal(x, y) for x, y in zip(out, want)), g
