"""vgb_pipeline_set_filters between seconds of a pipeline that replays graphs.

The filter's size decides how the overlap-add sums (FP32, split FP32 or int32
with FPGA rounding), and a captured second holds that kernel. Seconds with an
int16 filter, then with one of FINEPFB's size on the same buffers and parity,
then the first again: every product equals the same seconds run eagerly, bit
for bit. On full-range voltages a single FP32 sum of the larger filter rounds."""
from __future__ import annotations

import os

import numpy as np
import pytest

import synthetic as SY
from helpers import dev, tables, torch_cuda, weights_on_device

pytestmark = pytest.mark.gpu
K, NANT = 128, 6


@pytest.mark.parametrize("smart", [False, True])
def test_filter_swap(smart):
    import vgb

    torch = torch_cuda()
    rng = np.random.default_rng(6)
    small = SY.analysis_filter_int16()
    large = np.load(os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "ref_filters.npz"))["finepfb"]
    assert vgb.filter_wola_flags(small) != vgb.filter_wola_flags(large)
    syn = SY.synthesis_filter(scale=SY.synthesis_scale(small)).astype(np.float32)
    volts = [dev(rng.integers(-128, 128, 2 * NANT * 64000 * 2, dtype=np.int8).view(np.uint8)) for _ in range(2)]
    W = weights_on_device(*tables(NANT))
    torch.cuda.synchronize()

    def seconds(graphs):
        p = vgb.Pipeline(1, NANT, 1, nstokes=4, do_ipfb=True,
                         pfb_flags=vgb.PFB_SMART if smart else vgb.PFB_FULL_PRECISION)
        p.set_weights(W, on_device=True)
        p.set_vdif_header(np.stack([vgb.vdif_populate_header(58000, 0.99999, threadid=0)]))
        p.enable_graphs(graphs)
        out = []
        for h in (small, large, small):
            p.set_filters(h, syn)
            for s in range(4):
                p.run_device(volts[s % 2])
                ps, vd = np.empty((500, 4, K), np.uint8), np.empty((1, 500, 544), np.uint8)
                off, scl = np.empty((1, 4, K), np.float32), np.empty((1, 4, K), np.float32)
                p.fetch(ps, off, scl, vd)
                out.append((ps, off, scl, vd))
        return out

    for s, (got, want) in enumerate(zip(seconds(True), seconds(False))):
        for k, (x, y) in enumerate(zip(got, want)):
            assert np.array_equal(x, y), (s, k)
    assert vgb.check_device_status() == 0
