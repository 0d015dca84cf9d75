"""vgb_fpfb of short runs, whose steps are shared out four at a time.

A run whose shares of eight steps (32 columns) are less than a wave and a half
of the GPU's places takes shares of four. Bytes and doubles equal the staged
chain's bit for bit at step counts that leave each remainder of a share, in
every store width. A short run's 13 steps (50 inputs) as shares of 4 take well
under 13 / 4 of the time of a run of 4 steps (16 inputs), each on a few CTAs;
one after the other in one share they would take about that."""
from __future__ import annotations

import numpy as np
import pytest

import synthetic as SY
from helpers import dev, torch_cuda

pytestmark = pytest.mark.gpu
K = 128


def setup(vgb, torch, ninputs, ncc, seed=0):
    rng = np.random.default_rng(ninputs + seed)
    volt = np.clip(np.round(rng.standard_normal((ncc, 2, ninputs, 64000, 2), dtype=np.float32) * 20), -128, 127).astype(np.int8)
    d = dev(volt.reshape(-1).view(np.uint8))
    return d, vgb.reference_buffer_voltages(d, ninputs, 1, ncc, volt[0].nbytes), dev(rng.permutation(ninputs).astype(np.int32))


@pytest.mark.parametrize("ninputs", [14, 16, 18, 34, 48, 50, 66, 96])
@pytest.mark.parametrize("ns", [9, 150, 500])
@pytest.mark.parametrize("smart", [True, False])
def test_shares_of_four_steps(ninputs, ns, smart):
    import vgb

    torch = torch_cuda()
    d, v, di = setup(vgb, torch, ninputs, 2)
    dh = dev(SY.analysis_filter_int16())
    flags = vgb.PFB_SMART if smart else vgb.PFB_FULL_PRECISION
    size = ns * K * ninputs * (1 if smart else 16)
    want = torch.empty(2 * size, dtype=torch.uint8, device="cuda")
    b = torch.empty(ns * ninputs * K * 2, dtype=torch.int32, device="cuda")
    for cc in range(2):
        one = vgb.reference_buffer_voltages(d[cc * d.numel() // 2:], ninputs, 1)
        vgb.wola(one, ns, dh, b)
        vgb.round_(b, b.numel(), bool(flags & vgb.PFB_EMULATE_FPGA))
        vgb.fft128(b, ns * ninputs)
        vgb.pack(b, ns, ninputs, di, flags, want[cc * size:])
    for wola in (0, vgb.WOLA_FP32, vgb.WOLA_FP32_SPLIT):
        got = torch.full((2 * size,), 0x5A, dtype=torch.uint8, device="cuda")
        vgb.fpfb(v, 2, ns, dh, di, flags | wola, got)
        torch.cuda.synchronize()
        same = torch.equal(got, want) if smart else torch.equal(got.view(torch.float64), want.view(torch.float64))
        assert same, wola
    assert vgb.check_device_status() == 0


@pytest.mark.parametrize("ns", [150, 300])
def test_short_run_is_shared_out(ns):
    import vgb

    torch = torch_cuda()
    dh = dev(SY.analysis_filter_int16())

    def us(ninputs):
        d, v, di = setup(vgb, torch, ninputs, 1)
        out = torch.empty(ns * K * ninputs, dtype=torch.uint8, device="cuda")
        times = []
        for _ in range(10):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            torch.cuda.synchronize()
            a.record()
            for _ in range(20):
                vgb.fpfb(v, 1, ns, dh, di, vgb.PFB_SMART, out)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b) * 50)
        return min(times)

    # 16 inputs are 4 steps, one share either way; 50 inputs 13 steps
    four, thirteen = us(16), us(50)
    assert thirteen < 0.8 * four * 13 / 4, (four, thirteen)
