"""vgb_fpfb with its columns shared between CTAs, against the staged chain.

A CTA takes a multiple of four steps (16 output columns), at least eight where
there are that many; 4-bit rows are written 16, 4 or 1 bytes at a time as the
input count and the output's alignment allow. The staged chain (vgb_wola ->
vgb_round -> vgb_fft128 -> vgb_pack) does the same operations on each value, so
the outputs are equal bit for bit: one share and several, a ragged last step
and share, a ragged last tile of spectra, a misaligned output and inputs whose
voltages are zero (complex doubles of zeros take the conversion instruction).
"""
from __future__ import annotations

import numpy as np
import pytest

import synthetic as SY
from helpers import dev, torch_cuda

pytestmark = pytest.mark.gpu
K = 128


@pytest.mark.parametrize("ninputs,ns,shift", [(2, 3, 0), (10, 9, 0), (12, 8, 0), (32, 17, 0), (64, 8, 4), (66, 9, 0),
                                              (128, 5, 1), (250, 7, 0), (256, 13, 0), (272, 8, 8), (512, 4, 0)])
@pytest.mark.parametrize("mode", ["smart", "full", "smart imag first", "full fpga"])
def test_shares_equal_staged_chain(ninputs, ns, shift, mode):
    import vgb

    torch = torch_cuda()
    rng = np.random.default_rng(ninputs)
    volt = np.zeros((2, ninputs, 64000, 2), np.int8)
    volt[0, :, -12 * K:] = np.clip(np.round(rng.standard_normal((ninputs, 12 * K, 2)) * 20), -128, 127)
    volt[1, :, : ns * K] = np.clip(np.round(rng.standard_normal((ninputs, ns * K, 2)) * 20), -128, 127)
    volt[:, ninputs // 2] = 0
    h = SY.analysis_filter_int16()
    idx = rng.permutation(ninputs).astype(np.int32)
    flags = {"smart": vgb.PFB_SMART, "full": vgb.PFB_FULL_PRECISION,
             "smart imag first": vgb.PFB_SMART | vgb.PFB_IMAG_PART_FIRST,
             "full fpga": vgb.PFB_FULL_PRECISION | vgb.PFB_EMULATE_FPGA}[mode]
    flags ^= vgb.PFB_IMAG_PART_FIRST if mode == "full" else 0
    size = 1 if flags & vgb.PFB_COMPLEX_INT4 else 16
    shift *= 1 if size == 1 else 16
    d, dh, di = dev(volt.reshape(-1).view(np.uint8)), dev(h), dev(idx)
    v = vgb.reference_buffer_voltages(d, ninputs, 1)
    b = torch.empty(ns * ninputs * K * 2, dtype=torch.int32, device="cuda")
    vgb.wola(v, ns, dh, b)
    vgb.round_(b, b.numel(), bool(flags & vgb.PFB_EMULATE_FPGA))
    vgb.fft128(b, ns * ninputs)
    want = torch.empty(ns * K * ninputs * size, dtype=torch.uint8, device="cuda")
    vgb.pack(b, ns, ninputs, di, flags, want)
    for wola in (0, vgb.WOLA_FP32, vgb.WOLA_FP32_SPLIT):
        out = torch.full((ns * K * ninputs * size + 256,), 0x5A, dtype=torch.uint8, device="cuda")
        vgb.fpfb(v, 1, ns, dh, di, flags | wola, out[shift:])
        torch.cuda.synchronize()
        got = out[shift:shift + want.numel()]
        if size == 16:
            assert torch.equal(got.clone().view(torch.float64), want.view(torch.float64)), wola
        else:
            assert torch.equal(got, want), wola
        assert (out[:shift] == 0x5A).all() and (out[shift + want.numel():] == 0x5A).all()
    assert vgb.check_device_status() == 0
