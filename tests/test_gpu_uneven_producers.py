"""Steps in which some warps copy and others do not, ahead of tensor memory.

Variant 5 of the fused front end and the PFB-only kernel copy a step's frames
with one lane of some warps, just before whole warps read their taps and
twiddles from tensor memory. Input counts that leave the last step's warps idle,
tiles that cross from the carried frames into the second and from one block of
voltages into the next (one, two or three copies an input), and tiles of 4, 6
and 8 spectra: the same bits as variant 3, which keeps its tables in shared
memory and takes whole tiles, and as the staged PFB chain."""
from __future__ import annotations

import numpy as np
import pytest

import synthetic as SY
from helpers import dev, host, tables, torch_cuda, weights_on_device

pytestmark = pytest.mark.gpu
K = 128
MODES = {"fp32": 0, "split": 1, "int32": 2}


def voltages(vgb, ninputs, nblk, seed):
    rng = np.random.default_rng(seed)
    volt = np.clip(np.round(rng.standard_normal((nblk + 1, ninputs, 64000, 2), dtype=np.float32) * 30), -128, 127).astype(np.int8)
    d = dev(volt.reshape(-1).view(np.uint8))
    return d, vgb.reference_buffer_voltages(d, ninputs, nblk)


@pytest.mark.parametrize("nant", [1, 2, 3, 5])
@pytest.mark.parametrize("ns", [4, 6, 8, 13, 508, 1000])
@pytest.mark.parametrize("mode", list(MODES))
@pytest.mark.parametrize("smart", [False, True])
def test_front_end_variant_5(nant, ns, mode, smart):
    import vgb

    torch = torch_cuda()
    d, v = voltages(vgb, 2 * nant, -(-ns // 500), ns + nant)
    h = SY.analysis_filter_int16()
    if mode != "fp32":
        h = np.round(h * 3.6).astype(np.int32)
    flags = (vgb.PFB_SMART if smart else vgb.PFB_FULL_PRECISION) | [vgb.WOLA_FP32, vgb.WOLA_FP32_SPLIT, vgb.WOLA_INT32][MODES[mode]]
    W = weights_on_device(*tables(nant))
    out = []
    for g in (3, 5):
        S = torch.full((ns, 4, K), float("nan"), device="cuda")
        e = torch.full((ns, K, 2, 2), float("nan"), device="cuda")
        prev = vgb.pfb_variant(g)
        try:
            vgb.beamform_mwax(v, 1, ns, dev(h), flags, W, nant, 1 / 6, 4, S, e)
        finally:
            vgb.pfb_variant(prev)
        torch.cuda.synchronize()
        assert vgb.check_device_status() == 0 and vgb.pfb_variant_last() == g
        out.append((host(S), host(e)))
    for x, y in zip(*out):
        assert not np.isnan(x).any() and np.array_equal(x, y)


@pytest.mark.parametrize("ninputs", [1, 2, 3, 5, 9, 18])
@pytest.mark.parametrize("ns", [4, 13, 508])
@pytest.mark.parametrize("smart", [False, True])
def test_pfb_only(ninputs, ns, smart):
    import vgb

    torch = torch_cuda()
    d, v = voltages(vgb, ninputs, -(-ns // 500), ninputs)
    dh, di = dev(SY.analysis_filter_int16()), dev(np.random.default_rng(1).permutation(ninputs).astype(np.int32))
    flags = vgb.PFB_SMART if smart else vgb.PFB_FULL_PRECISION
    size = ns * K * ninputs * (1 if flags & vgb.PFB_COMPLEX_INT4 else 16)
    b = torch.empty(ns * ninputs * K * 2, dtype=torch.int32, device="cuda")
    want = torch.empty(size, dtype=torch.uint8, device="cuda")
    vgb.wola(v, ns, dh, b)
    vgb.round_(b, b.numel(), bool(flags & vgb.PFB_EMULATE_FPGA))
    vgb.fft128(b, ns * ninputs)
    vgb.pack(b, ns, ninputs, di, flags, want)
    for wola in (0, vgb.WOLA_FP32, vgb.WOLA_FP32_SPLIT):
        got = torch.full((size,), 0x5A, dtype=torch.uint8, device="cuda")
        vgb.fpfb(v, 1, ns, dh, di, flags | wola, got)
        torch.cuda.synchronize()
        same = torch.equal(got, want) if smart else torch.equal(got.view(torch.float64), want.view(torch.float64))
        assert same, wola
    assert vgb.check_device_status() == 0
