"""A second's stages side by side on several streams against one after the other.

With stage timing on the pipeline runs every stage in order on one stream;
otherwise the history, the two renormalises and the inverse PFB run beside one
another, from a captured graph or eagerly. Every product of four different
seconds is the same bit for bit, with and without the inverse PFB, and for a pipeline that loads its state at an
odd or an even second (the extremes for the 8-bit stage are kept by parity).
"""
from __future__ import annotations

import numpy as np
import pytest

import synthetic as SY
from helpers import dev, tables, torch_cuda, weights_on_device

pytestmark = pytest.mark.gpu
K, NANT, NBLK = 128, 6, 1


@pytest.mark.parametrize("ipfb", [True, False])
@pytest.mark.parametrize("nstokes", [1, 4])
def test_side_streams_equal_serial(ipfb, nstokes):
    import vgb

    torch = torch_cuda()
    rng = np.random.default_rng(4)
    ncc, nsec = 2, 4
    h = SY.analysis_filter_int16()
    syn = SY.synthesis_filter(scale=SY.synthesis_scale(h)).astype(np.float32)
    # seconds of different power, so that stale extremes would show
    volts = [dev(np.clip(np.round(rng.standard_normal((ncc, NBLK, 2 * NANT, 64000, 2)) * sg), -127, 127).astype(np.int8)
                 .reshape(-1).view(np.uint8)) for sg in (40, 5, 25, 10)]
    W = torch.cat([weights_on_device(*tables(NANT, cc=c)) for c in range(ncc)])
    ns = NBLK * 500

    def products(p):
        out = dict(ps=np.empty((ns, nstokes, ncc * K), np.uint8), off=np.empty((ncc, nstokes, K), np.float32),
                   scl=np.empty((ncc, nstokes, K), np.float32), inc=np.empty((ns, ncc * K), np.uint8),
                   ioff=np.empty((ncc, K), np.float32), iscl=np.empty((ncc, K), np.float32))
        vd = np.empty((ncc, ns, 544), np.uint8) if ipfb else None
        p.fetch(out["ps"], out["off"], out["scl"], vd)
        p.fetch_incoh(out["inc"], out["ioff"], out["iscl"])
        if ipfb:
            out["vdif"] = vd
        return out

    def make(mode):
        p = vgb.Pipeline(ncc, NANT, NBLK, nstokes=nstokes, do_ipfb=ipfb)
        p.set_filters(h, syn if ipfb else None)
        p.set_weights(W, on_device=True)
        if ipfb:
            p.set_vdif_header(np.stack([vgb.vdif_populate_header(58000, 0.99999, threadid=c) for c in range(ncc)]))
        p.enable_timing(mode == "serial")
        p.enable_graphs(mode == "graph")
        return p

    torch.cuda.synchronize()
    want, states = [], []
    p = make("serial")
    for v in volts:
        states.append(p.save_state())
        p.run_device(v)
        want.append(products(p))
    for mode in ("graph", "eager"):
        p = make(mode)
        for s, v in enumerate(volts):
            p.run_device(v)
            for k, x in products(p).items():
                assert np.array_equal(x, want[s][k]), (mode, s, k)
        for start in (1, 2):
            q = make(mode)
            q.run_device(volts[0])                      # its own extremes and history, then another second's state
            q.load_state(states[start])
            for s in range(start, nsec):
                q.run_device(volts[s])
                for k, x in products(q).items():
                    assert np.array_equal(x, want[s][k]), (mode, start, s, k)
    assert vgb.check_device_status() == 0
