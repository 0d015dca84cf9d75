"""Timed cases of the voltage hot path, through the library's public calls.

Each kind below is one call (or the short run of calls) that a VCSBeam-style
program makes per second of data: the streaming pipeline's second, the fused
PFB + beamformer of MWAX voltages, the PFB alone, the beamformer of legacy
voltages, many beams on the tensor cores, the 8-bit products of several
beams and the per-second tables. Voltages are Gaussian, as MWA voltages are;
calibration matrices are the identity with 10 % scatter; filters are the
sinc x Hann prototype in int16 or scaled to the size of the reference's
FINEPFB coefficients.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "mwa-vcsbeam_gb300"))

import synthetic as SY  # noqa: E402
import vgb  # noqa: E402

K, P, BLOCK, FRAMES = 128, 12, 64000, 500
C = 299792458.0
HREF = SY.MWA_ALTITUDE_METRES


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------
def listed():
    return [
        # one data-second of the whole band on one GPU: 24 coarse channels of
        # the 128-tile array, tracking, PSRFITS and VDIF out (the benchmark)
        dict(name="second_24ch", kind="second", ncc=24, nant=128, nblocks=20, nstokes=4, ipfb=True, filt="int16", track=True),
        # one coarse channel's second, as one of 24 processes has it, with
        # filter coefficients of FINEPFB's size
        dict(name="second_1ch", kind="second", ncc=1, nant=128, nblocks=20, nstokes=4, ipfb=True, filt="fine", track=False),
        # the smallest call: one voltage block of a 16-tile test array
        dict(name="second_small", kind="second", ncc=1, nant=16, nblocks=1, nstokes=4, ipfb=True, filt="int16", track=False),
        # the reference's --smart mode (FPGA rounding, 4-bit voltages) on an
        # odd tile count and an odd number of spectra, Stokes I only
        dict(name="mwax_smart", kind="mwax", ncc=2, nant=119, nspectra=4993, nstokes=1, flags=0x21D, filt="int16"),
        # fine_pfb_offline: the PFB alone to recombined 4+4-bit voltages
        dict(name="fpfb_4bit", kind="fpfb", ncc=1, nant=128, nspectra=10000, flags=0x21D, filt="fine"),
        # ... and to complex doubles, for the beamformer's full-precision input
        dict(name="fpfb_double", kind="fpfb", ncc=1, nant=128, nspectra=4000, flags=0x2D, filt="int16"),
        # legacy recombined voltages: a second of one coarse channel, one beam
        dict(name="legacy_4bit", kind="legacy", nant=128, nsamples=10000, npointing=1, nstokes=4, double=False),
        # ... a few beams of full-precision fine voltages
        dict(name="legacy_double", kind="legacy", nant=128, nsamples=2000, npointing=3, nstokes=4, double=True),
        # 1024 beams, 256 tiles, full Stokes, one coarse channel-second
        dict(name="beams_1024", kind="beams", nant=256, npointing=1024, nsamples=10000, nstokes=4, precision=0, int8=False),
        # a small pulsar census: 20 beams of 8-bit voltages, Stokes I
        dict(name="beams_20", kind="beams", nant=128, npointing=20, nsamples=10000, nstokes=1, precision=2, int8=True),
        # the products of several beams: 8-bit PSRFITS and inverse PFB
        dict(name="products_6", kind="products", npointing=6, nsamples=10000, nstokes=4, floats=True),
        # the per-second tables: primary beam, inverse Jones, phases, weights
        dict(name="tables_8", kind="tables", npointing=8, nant=128, nsets=3),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["second", "second", "mwax", "mwax", "fpfb", "fpfb", "legacy", "legacy", "beams", "products",
                       "tables"])
    nst = rng.choice([1, 4])
    filt = rng.choice(["int16", "fine"])
    if kind == "second":
        return dict(kind=kind, ncc=_log(rng, 1, 12), nant=_log(rng, 8, 144), nblocks=rng.randint(1, 20), nstokes=nst,
                    ipfb=rng.random() < 0.7, filt=filt, track=rng.random() < 0.5)
    if kind == "mwax":
        return dict(kind=kind, ncc=rng.randint(1, 4), nant=_log(rng, 5, 144), nspectra=_log(rng, 300, 10000),
                    nstokes=nst, flags=rng.choice([0x21D, 0x2D]), filt=filt)
    if kind == "fpfb":
        double = rng.random() < 0.5
        return dict(kind=kind, ncc=rng.randint(1, 3), nant=_log(rng, 5, 144), filt=filt,
                    nspectra=_log(rng, 300, 4000 if double else 10000), flags=0x2D if double else 0x21D)
    if kind == "legacy":
        double = rng.random() < 0.5
        return dict(kind=kind, nant=2 * _log(rng, 4, 128), nsamples=_log(rng, 200, 3000 if double else 10000),
                    npointing=_log(rng, 1, 12), nstokes=nst, double=double)
    if kind == "beams":
        return dict(kind=kind, nant=16 * rng.randint(1, 16), npointing=_log(rng, 2, 500),
                    nsamples=10 * _log(rng, 40, 1000), nstokes=nst, precision=rng.choice([0, 0, 1, 2]),
                    int8=rng.random() < 0.5)
    if kind == "products":
        return dict(kind=kind, npointing=_log(rng, 1, 24), nsamples=_log(rng, 300, 10000), nstokes=nst,
                    floats=rng.random() < 0.5)
    return dict(kind=kind, npointing=_log(rng, 1, 24), nant=_log(rng, 8, 256), nsets=rng.randint(1, 8))


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _int8(shape, g, sigma=16.0, bound=127):
    """Gaussian voltages in a new int8 tensor, a slice of the first axis at a time."""
    out = torch.empty(shape, dtype=torch.int8, device="cuda")
    for part in out:
        x = torch.randn(part.shape, generator=g, device="cuda", dtype=torch.float32)
        part.copy_(x.mul_(sigma).round_().clamp_(-bound, bound))
    return out


def _bytes4(shape, g):
    """4+4-bit voltages (high nibble real), clipped Gaussian."""
    out = torch.empty(shape, dtype=torch.uint8, device="cuda")
    step = max(1, (1 << 27) // max(1, out[0].numel()))
    for i in range(0, shape[0], step):
        part = out[i:i + step]
        n = torch.randn((2,) + part.shape, generator=g, device="cuda").mul_(2.0).round_().clamp_(-8, 7).to(torch.int32)
        part.copy_(((n[0] & 15) << 4) | (n[1] & 15))
    return out


def _cn(shape, g):
    return torch.view_as_complex(torch.randn(tuple(shape) + (2,), generator=g, device="cuda", dtype=torch.float64)) / math.sqrt(2)


def _jones_like(shape, g):
    return torch.eye(2, dtype=torch.complex128, device="cuda") + 0.1 * _cn(tuple(shape) + (2, 2), g)


def _weights(shape, g):
    """phi J^-1: near-identity matrices under random phases, complex64."""
    ph = torch.rand(shape, generator=g, device="cuda", dtype=torch.float64) * (2 * math.pi)
    return (_jones_like(shape, g) * torch.polar(torch.ones_like(ph), ph)[..., None, None]).to(torch.complex64)


def _filter(name):
    h = SY.analysis_filter_int16()
    return np.round(h * 3.6).astype(np.int32) if name == "fine" else h


def _synthesis(h):
    return SY.synthesis_filter(scale=SY.synthesis_scale(h)).astype(np.float32)


def _layout(nant, seed):
    """East, north, height, cable of the tiles, and pointing unit vectors from (az, za) in radians."""
    return [torch.from_numpy(x).cuda() for x in SY.tile_layout(nant, seed=seed + 7)]


def _pointings(n, g):
    az = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * 2 * math.pi
    za = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * 0.6
    return az, za


def _unit(az, za):
    return torch.stack([torch.sin(az) * torch.sin(za), torch.cos(az) * torch.sin(za), torch.cos(za)], -1).contiguous()


def _freqs(cc):
    return SY.fine_chan_freqs_hz(SY.coarse_chan_start_hz(cc))


class _View:
    """Device memory at an address, for torch.as_tensor."""

    def __init__(self, ptr, shape, typestr, owner):
        self.__cuda_array_interface__ = dict(data=(ptr, False), shape=shape, typestr=typestr, version=2)
        self.owner = owner


def _inputs(case, seed):
    """What the call takes, on the GPU, from the seed alone."""
    g = _gen(seed)
    k = case["kind"]
    s = {}
    if k == "second":
        n, A = case["ncc"], case["nant"]
        s["v"] = _int8((n, case["nblocks"], 2 * A, BLOCK, 2), g)
        if case["track"]:
            s["D"] = _jones_like((n, A, K), g)
            s["delays"] = torch.from_numpy(np.tile(SY.tile_delays(45.0, 20.0).astype(np.int32), (A, 1))).cuda()
            s["pos"] = _layout(A, seed)
            s["freqs"] = torch.from_numpy(np.stack([_freqs(c) for c in range(n)])).cuda()
            s["bfreqs"] = s["freqs"].mean(1).contiguous()
            s["az"] = torch.tensor([math.radians(45.0)], dtype=torch.float64, device="cuda")
            s["za"] = torch.tensor([math.radians(20.0)], dtype=torch.float64, device="cuda")
        else:
            s["W"] = _weights((n, A, K), g)
    elif k in ("mwax", "fpfb"):
        n, A, nb = case["ncc"], case["nant"], -(-case["nspectra"] // FRAMES)
        s["v"] = _int8((n, nb + 1, 2 * A, BLOCK, 2), g)  # a margin block, then the second
        if k == "mwax":
            s["W"] = _weights((n, A, K), g)
        else:
            s["idx"] = torch.randperm(2 * A, generator=g, device="cuda").to(torch.int32)
    elif k == "legacy":
        A, ns = case["nant"], case["nsamples"]
        if case["double"]:
            s["v"] = torch.randn((ns, K, 2 * A, 2), generator=g, device="cuda", dtype=torch.float32).to(torch.float64)
        else:
            s["v"] = _bytes4((ns, K, 2 * A), g)
        order = torch.randperm(2 * A, generator=g, device="cuda").to(torch.int32)
        s["polQ"], s["polP"] = order[0::2].contiguous(), order[1::2].contiguous()
        s["W"] = _weights((case["npointing"], A, K), g)
    elif k == "beams":
        A, ns, B = case["nant"], case["nsamples"], case["npointing"]
        s["v"] = _int8((ns, K, 2 * A, 2), g) if case["int8"] else _bytes4((ns, K, 2 * A), g)
        order = torch.randperm(2 * A, generator=g, device="cuda").to(torch.int32)
        s["polQ"], s["polP"] = order[0::2].contiguous(), order[1::2].contiguous()
        s["D"], s["B"] = _jones_like((1, A, K), g), _jones_like((1, B, A), g)
        s["pos"] = _layout(A, seed)
        s["unit"] = _unit(*_pointings(B, g))
        s["freqs"] = torch.from_numpy(_freqs(3)[None]).cuda()
    elif k == "products":
        n, ns, nst = case["npointing"], case["nsamples"], case["nstokes"]
        s["S"] = torch.randn((1, n, ns, nst, K), generator=g, device="cuda").mul_(300.0)
        s["S"][..., 0, :].abs_()
        s["e"] = torch.randn((n, ns, K, 2, 2), generator=g, device="cuda").mul_(40.0)
        s["hist"] = torch.randn((n, P, K, 2, 2), generator=g, device="cuda").mul_(40.0)
        hdr = np.stack([vgb.vdif_populate_header(58000 + i, 0.25, threadid=i) for i in range(n)])
        s["hdr"] = torch.from_numpy(hdr.view(np.int32)).cuda()
    else:
        n, A = case["npointing"], case["nant"]
        s["az"], s["za"] = _pointings(n, g)
        sets = torch.from_numpy(SY.tile_delay_sets(case["nsets"], seed=int(seed) % 100000).astype(np.int32)).cuda()
        s["delays"] = sets[torch.randint(0, case["nsets"], (A,), generator=g, device="cuda")].contiguous()
        s["D"] = _jones_like((A, K), g)
        s["pos"] = _layout(A, seed)
        s["unit"] = _unit(s["az"], s["za"])
        s["freqs"] = torch.from_numpy(_freqs(5)).cuda()
        s["bfreq"] = torch.tensor([float(_freqs(5).mean())], dtype=torch.float64, device="cuda")
    return s


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    k = case["kind"]
    new = lambda *shape, t=torch.float32: torch.empty(shape, dtype=t, device="cuda")  # noqa: E731
    if k == "second":
        n, A, nst, ns = case["ncc"], case["nant"], case["nstokes"], case["nblocks"] * FRAMES
        h = _filter(case["filt"])
        p = vgb.Pipeline(n, A, nblocks=case["nblocks"], nstokes=nst, do_ipfb=case["ipfb"])
        p.set_filters(h, _synthesis(h) if case["ipfb"] else None)
        if case["track"]:
            east, north, height, cable = s["pos"]
            p.set_tracking(s["D"], s["delays"], east, north, height, cable, s["freqs"], s["bfreqs"], s["az"], s["za"],
                           href=HREF, latitude=vgb.MWA_LATITUDE_RADIANS)
        else:
            p.stream().wait_stream(torch.cuda.current_stream())  # the copy of W runs on the pipeline's stream
            p.set_weights(s["W"], True)
        if case["ipfb"]:
            p.set_vdif_header(np.stack([vgb.vdif_populate_header(58000, 0.5, threadid=c) for c in range(n)]))
        s["pipe"] = p
    elif k == "mwax":
        h = _filter(case["filt"])
        n, ns = case["ncc"], case["nspectra"]
        s["filt"], s["flags"] = torch.from_numpy(h).cuda(), case["flags"] | vgb.filter_wola_flags(h)
        s["volt"] = vgb.reference_buffer_voltages(s["v"], 2 * case["nant"], s["v"].shape[1] - 1, n, s["v"].stride(0))
        s["S"], s["e"], s["incoh"] = new(n, ns, case["nstokes"], K), new(n, ns, K, 2, 2), new(n, ns, K)
    elif k == "fpfb":
        h = _filter(case["filt"])
        n, ns, I = case["ncc"], case["nspectra"], 2 * case["nant"]
        s["filt"], s["flags"] = torch.from_numpy(h).cuda(), case["flags"] | vgb.filter_wola_flags(h)
        s["volt"] = vgb.reference_buffer_voltages(s["v"], I, s["v"].shape[1] - 1, n, s["v"].stride(0))
        s["out"] = new(n, ns, K, I, t=torch.uint8) if case["flags"] & 0x10 else new(n, ns, K, I, 2, t=torch.float64)
    elif k == "legacy":
        n, ns = case["npointing"], case["nsamples"]
        s["S"], s["e"] = new(n, ns, case["nstokes"], K), new(n, ns, K, 2, 2)
        s["incoh"] = None if case["double"] else new(ns, K)
    elif k == "beams":
        A, B, ns, nst = case["nant"], case["npointing"], case["nsamples"], case["nstokes"]
        mb = vgb.Multibeam(1, K, A, B, ns, nstokes=nst, precision=case["precision"],
                           input=vgb.MB_INT8 if case["int8"] else vgb.MB_INT4)
        east, north, height, cable = s["pos"]
        mb.set_geometry(s["unit"], east, north, height, cable, href=HREF)
        mb.set_jones(s["D"], s["B"], s["freqs"], s["polQ"], s["polP"])
        s["mb"] = mb
        s["S"], s["out"] = new(K, B, nst, ns // 10), new(B, ns // 10, nst, K, t=torch.uint8)
        s["off"], s["scl"] = new(B, nst, K), new(B, nst, K)
    elif k == "products":
        n, ns, nst = case["npointing"], case["nsamples"], case["nstokes"]
        s["coeffs"] = torch.from_numpy(_synthesis(_filter("int16"))).cuda()
        s["out"], s["off"], s["scl"] = new(n, ns, nst, K, t=torch.uint8), new(n, nst, K), new(n, nst, K)
        s["vdif"] = new(n, ns, 544, t=torch.uint8)
        s["outf"] = new(n, ns * K, 2, 2) if case["floats"] else None
    else:
        n, A = case["npointing"], case["nant"]
        s["Bm"], s["J"] = new(1, n, A, 2, 2, 2, t=torch.float64), new(n, A, K, 2, 2, 2, t=torch.float64)
        s["phi"], s["W"] = new(n, A, K, 2, t=torch.float64), new(n, A, K, 2, 2, 2)
    return s


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------
def run(s):
    case = s["case"]
    k = case["kind"]
    if k == "second":
        p, n, ns, nst = s["pipe"], case["ncc"], case["nblocks"] * FRAMES, case["nstokes"]
        p.run_device(s["v"])
        S, e, incoh, ps, vd = p.device_products()
        view = lambda ptr, shape, t: torch.as_tensor(_View(ptr, shape, t, p), device="cuda")  # noqa: E731
        return {"S": view(S, (n, ns, nst, K), "<f4"), "e": view(e, (n, ns, K, 2, 2), "<f4"),
                "incoh": view(incoh, (n, ns, K), "<f4"), "psrfits": view(ps, (ns, nst, n * K), "|u1"),
                "vdif": view(vd, (n, ns, 544), "|u1") if case["ipfb"] else None}
    if k == "mwax":
        A = case["nant"]
        vgb.beamform_mwax(s["volt"], case["ncc"], case["nspectra"], s["filt"], s["flags"], s["W"], A, 1.0 / (2 * A),
                          case["nstokes"], s["S"], s["e"], s["incoh"])
        return {"S": s["S"], "e": s["e"], "incoh": s["incoh"]}
    if k == "fpfb":
        vgb.fpfb(s["volt"], case["ncc"], case["nspectra"], s["filt"], s["idx"], s["flags"], s["out"])
        return {"out": s["out"]}
    if k == "legacy":
        A = case["nant"]
        vgb.beamform_legacy(s["v"], vgb.DBL if case["double"] else vgb.INT4, case["nsamples"], K, A, s["polQ"],
                            s["polP"], s["W"], case["npointing"], 1.0 / (2 * A), case["nstokes"], s["S"], s["e"],
                            s["incoh"])
        return {"S": s["S"], "e": s["e"], "incoh": s["incoh"]}
    if k == "beams":
        s["mb"].run(s["v"], S=s["S"], out=s["out"], offsets=s["off"], scales=s["scl"])
        return {"S": s["S"], "out": s["out"], "offsets": s["off"], "scales": s["scl"]}
    if k == "products":
        n, ns, nst = case["npointing"], case["nsamples"], case["nstokes"]
        vgb.renormalise(s["S"], 1, n, ns, nst, K, s["out"], 0, ns * nst * K, nst * K, K, s["off"], s["scl"])
        vgb.ipfb(s["e"], ns * K * 16, s["hist"], P * K * 16, s["coeffs"], ns, n, out_f=s["outf"], vdif=s["vdif"],
                 hdr=s["hdr"])
        return {"psrfits": s["out"], "offsets": s["off"], "scales": s["scl"], "vdif": s["vdif"], "samples": s["outf"]}
    n, A = case["npointing"], case["nant"]
    east, north, height, cable = s["pos"]
    vgb.primary_beam(s["az"], s["za"], s["bfreq"], s["delays"], s["Bm"])
    vgb.jones(s["D"], s["Bm"], n, A, K, s["J"])
    vgb.phase(s["unit"], east, north, height, cable, s["freqs"], n, A, K, HREF, s["phi"])
    vgb.weights(s["J"], s["phi"], n * A * K, s["W"])
    return {"B": s["Bm"], "J": s["J"], "phi": s["phi"], "W": s["W"]}


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------
def work(case):
    """Each input read once, each output written once; the operations of the
    weighted overlap-add (12 real taps on complex samples), a 5 N log2 N FFT
    and the complex multiply-adds of the beamformer."""
    k = case["kind"]
    pfb = 2 * 2 * P * K + 5 * K * 7  # per (input, fine spectrum)
    beam = 30 * K                    # per (input, fine spectrum) and beam
    if k == "second":
        n, A, ns, nst = case["ncc"], case["nant"], case["nblocks"] * FRAMES, case["nstokes"]
        out = ns * K * (4 * nst + 16 + 4 + nst + 1) + (544 * ns if case["ipfb"] else 0)
        tables = A * K * (64 if case["track"] else 32)
        inv = 2 * ns * (5 * K * 7 + 4 * P * K) if case["ipfb"] else 0
        return dict(bytes=n * (ns * K * 2 * 2 * A + tables + out), flops=n * (ns * 2 * A * (pfb + beam) + inv))
    if k == "mwax":
        n, A, ns, nst = case["ncc"], case["nant"], case["nspectra"], case["nstokes"]
        return dict(bytes=n * (((ns + P - 1) * 4 * A + ns * (4 * nst + 20)) * K + A * K * 32),
                    flops=n * ns * 2 * A * (pfb + beam))
    if k == "fpfb":
        n, I, ns = case["ncc"], 2 * case["nant"], case["nspectra"]
        return dict(bytes=n * I * K * ((ns + P - 1) * 2 + ns * (1 if case["flags"] & 0x10 else 16)), flops=n * ns * I * pfb)
    if k == "legacy":
        n, A, ns, nst = case["npointing"], case["nant"], case["nsamples"], case["nstokes"]
        dbl = case["double"]
        return dict(bytes=ns * K * 2 * A * (16 if dbl else 1) + n * (A * K * 32 + ns * K * (4 * nst + 16)) + (0 if dbl else ns * K * 4),
                    flops=n * ns * K * A * 52)
    if k == "beams":
        A, B, ns, nst = case["nant"], case["npointing"], case["nsamples"], case["nstokes"]
        return dict(bytes=ns * K * 2 * A * (2 if case["int8"] else 1) + (K + B) * A * 64 + B * ns // 10 * nst * K * 5,
                    flops=ns * K * (4 * B * 4 * A * 2 + 12 * B))
    if k == "products":
        n, ns, nst = case["npointing"], case["nsamples"], case["nstokes"]
        return dict(bytes=n * ns * (K * (5 * nst + 16) + 544 + (K * 16 if case["floats"] else 0)),
                    flops=n * ns * (3 * nst * K + 2 * (5 * K * 7 + 4 * P * K)))
    n, A = case["npointing"], case["nant"]
    return dict(bytes=A * K * 64 + n * A * 64 + n * A * K * (64 + 16 + 32), flops=n * A * K * 180)


# --------------------------------------------------------------------------
# the same in 64 bits
# --------------------------------------------------------------------------
def _pfb64(x, h, m0, m1, fpga, demote):
    """x [frames][inputs][K] complex128 windows; fine voltages [m][input][k'] of
    spectra m0 .. m1 - 1 (the reference's fftshift and (im, re) order)."""
    t = torch.from_numpy(h.astype(np.float64)).cuda().flip(0).view(P, K)  # h[KP - Kp - n - 1]
    b = sum(t[p] * x[m0 + p:m1 + p] for p in range(P))
    if fpga:
        b = torch.view_as_real(b)
        b = torch.view_as_complex(torch.floor((b + torch.where(b > 0, 8192.0, 0.0)) / 16384.0))
    else:
        b = b / 16384.0
    X = torch.fft.fftshift(torch.fft.fft(b, dim=-1), dim=-1) / K
    v = torch.stack([X.imag, X.real], -1)
    if demote:
        v = torch.clamp(torch.trunc(v + torch.copysign(torch.full_like(v, 0.5), v)), -8, 7)
    return torch.view_as_complex(v)


def _stokes64(ex, ey, A_dim, invw, nst):
    """Sums over tiles with each tile's own power removed."""
    X, Y = ex.sum(A_dim), ey.sum(A_dim)
    xx = X.abs() ** 2 - (ex.abs() ** 2).sum(A_dim)
    yy = Y.abs() ** 2 - (ey.abs() ** 2).sum(A_dim)
    xy = X * Y.conj() - (ex * ey.conj()).sum(A_dim)
    S = [invw * (xx + yy), invw * (xx - yy), 2 * invw * xy.real, -2 * invw * xy.imag][:nst]
    return S, X, Y


def _beam64(frames, h, W, ns, invw, nst, fpga, demote):
    """One coarse channel: frames [12 + ns (- 1)][inputs][K][2] int8; W [tile][K][2][2]."""
    S = torch.empty((ns, nst, K), dtype=torch.float64, device="cuda")
    e = torch.empty((ns, K, 2), dtype=torch.complex128, device="cuda")
    inc = torch.empty((ns, K), dtype=torch.float64, device="cuda")
    W = W.to(torch.complex128)
    for m0 in range(0, ns, 250):
        m1 = min(ns, m0 + 250)
        x = torch.view_as_complex(frames[m0:m1 + P - 1].to(torch.float64))
        v = _pfb64(x, h, 0, m1 - m0, fpga, demote)
        q, p = v[:, 0::2], v[:, 1::2]
        ex, ey = W[..., 0, 0] * q + W[..., 0, 1] * p, W[..., 1, 0] * q + W[..., 1, 1] * p
        st, X, Y = _stokes64(ex, ey, 1, invw, nst)
        S[m0:m1] = torch.stack(st, 1)
        e[m0:m1] = torch.stack([X, Y], -1)
        inc[m0:m1] = (v.abs() ** 2).sum(1)
    return S, torch.view_as_real(e), inc


def _frames(blocks):
    """[block][input][64000][2] -> [frame][input][K][2]."""
    nb, I = blocks.shape[:2]
    return blocks.view(nb, I, FRAMES, K, 2).transpose(1, 2).reshape(nb * FRAMES, I, K, 2)


def _phase64(unit, pos, freqs):
    """[p][a][c] complex128."""
    east, north, height, cable = pos
    w = unit[:, 0:1] * east + unit[:, 1:2] * north + unit[:, 2:3] * (height - HREF)
    ph = 2 * math.pi * ((w - cable) / C)[..., None] * torch.floor(freqs)
    return torch.polar(torch.ones_like(ph), ph)


def _jinv64(D, B):
    """inv(D B / |D B|_F): D [a][c][2][2], B [p][a][2][2] -> [p][a][c][2][2]."""
    M = D[None] @ B[:, :, None]
    M = M / torch.linalg.matrix_norm(M)[..., None, None]
    m00, m01, m10, m11 = M[..., 0, 0], M[..., 0, 1], M[..., 1, 0], M[..., 1, 1]
    adj = torch.stack([m11, -m01, -m10, m00], -1).view(M.shape)
    return adj / (m00 * m11 - m01 * m10)[..., None, None]


def _tile_beam64(az, za, f, delays, lat):
    """[p][a][2][2]: 16 dipoles over a ground plane, then the parallactic rotation."""
    i = torch.arange(16, device="cuda", dtype=torch.float64)
    x, y = (i % 4 - 1.5) * 1.1, (1.5 - torch.floor(i / 4)) * 1.1
    sza, cza, saz, caz = torch.sin(za), torch.cos(za), torch.sin(az), torch.cos(az)
    tau = (x * (sza * saz)[:, None] + y * (sza * caz)[:, None]) / C
    ph = 2 * math.pi * f * (tau[:, None] - delays.to(torch.float64) * 435e-12)
    af = torch.polar(torch.ones_like(ph), ph).sum(-1) / 16
    w = 2 * math.pi * f * 0.278 / C
    af = af * (torch.sin(w * cza) / math.sin(w))[:, None]
    proj = torch.stack([cza * saz, cza * caz, caz, -saz], -1).view(-1, 1, 2, 2)
    el = math.pi / 2 - za
    hx = -caz * torch.cos(el) * math.sin(lat) + torch.sin(el) * math.cos(lat)
    hy, hz = -saz * torch.cos(el), caz * torch.cos(el) * math.cos(lat) + torch.sin(el) * math.sin(lat)
    ha, dec = torch.atan2(hy, hx), torch.atan2(hz, torch.hypot(hx, hy))
    chi = torch.atan2(math.cos(lat) * torch.sin(ha), math.sin(lat) * torch.cos(dec) - math.cos(lat) * torch.sin(dec) * torch.cos(ha))
    rot = torch.stack([-torch.cos(chi), -torch.sin(chi), torch.sin(chi), -torch.cos(chi)], -1).view(-1, 1, 2, 2)
    return af[..., None, None] * (proj @ rot)


def _nibbles(v):
    b = v.to(torch.int16)
    signed = lambda n: ((n ^ 8) - 8).to(torch.float64)  # noqa: E731
    return torch.complex(signed((b >> 4) & 15), signed(b & 15))


def exact(case, seed):
    k = case["kind"]
    nst = case.get("nstokes")
    if k == "second":
        if case["track"]:
            return None  # the whole band in 64 bits takes too long
        s = _inputs(case, seed)
        got = []
        for c in range(case["ncc"]):
            f = torch.cat([torch.zeros((P, 2 * case["nant"], K, 2), dtype=torch.int8, device="cuda"), _frames(s["v"][c])])
            got.append(_beam64(f, _filter(case["filt"]), s["W"][c], case["nblocks"] * FRAMES, 1.0 / (2 * case["nant"]), nst,
                               False, False))
        S, e, inc = (torch.stack([x[i] for x in got]) for i in range(3))
        return {"S": S, "e": e, "incoh": inc, "psrfits": None, "vdif": None}
    if k == "mwax":
        s = _inputs(case, seed)
        got = [_beam64(_frames(s["v"][c])[FRAMES - P:], _filter(case["filt"]), s["W"][c], case["nspectra"],
                       1.0 / (2 * case["nant"]), nst, bool(case["flags"] & 0x200), bool(case["flags"] & 0x10))
               for c in range(case["ncc"])]
        S, e, inc = (torch.stack([x[i] for x in got]) for i in range(3))
        return {"S": S, "e": e, "incoh": inc}
    if k == "fpfb":
        if case["flags"] & 0x10:
            return None  # bytes
        s = _inputs(case, seed)
        ns, I = case["nspectra"], 2 * case["nant"]
        out = torch.empty((case["ncc"], ns, K, I, 2), dtype=torch.float64, device="cuda")
        h, idx = _filter(case["filt"]), s["idx"].long()
        for c in range(case["ncc"]):
            f = _frames(s["v"][c])[FRAMES - P:]
            for m0 in range(0, ns, 250):
                m1 = min(ns, m0 + 250)
                v = _pfb64(torch.view_as_complex(f[m0:m1 + P - 1].to(torch.float64)), h, 0, m1 - m0, False, False)
                out[c, m0:m1, :, idx] = torch.view_as_real(v).transpose(1, 2)
        return {"out": out}
    if k == "legacy":
        s = _inputs(case, seed)
        n, A, ns = case["npointing"], case["nant"], case["nsamples"]
        S = torch.empty((n, ns, nst, K), dtype=torch.float64, device="cuda")
        e = torch.empty((n, ns, K, 2), dtype=torch.complex128, device="cuda")
        inc = None if case["double"] else torch.empty((ns, K), dtype=torch.float64, device="cuda")
        W = s["W"].to(torch.complex128).transpose(1, 2)  # [p][c][a][2][2]
        q, p = s["polQ"].long(), s["polP"].long()
        for m0 in range(0, ns, 100):
            raw = s["v"][m0:m0 + 100]
            v = torch.view_as_complex(raw) if case["double"] else _nibbles(raw)
            if inc is not None:
                inc[m0:m0 + 100] = (v.abs() ** 2).sum(-1)
            for i in range(n):
                ex = W[i, ..., 0, 0] * v[..., q] + W[i, ..., 0, 1] * v[..., p]
                ey = W[i, ..., 1, 0] * v[..., q] + W[i, ..., 1, 1] * v[..., p]
                st, X, Y = _stokes64(ex, ey, -1, 1.0 / (2 * A), nst)
                S[i, m0:m0 + 100] = torch.stack(st, 1)
                e[i, m0:m0 + 100] = torch.stack([X, Y], -1)
        return {"S": S, "e": torch.view_as_real(e), "incoh": inc}
    if k == "beams":
        A, B, ns = case["nant"], case["npointing"], case["nsamples"]
        if A * B * ns > 1.2e8:
            return None
        s = _inputs(case, seed)
        phi = _phase64(s["unit"], s["pos"], s["freqs"][0])
        J = _jinv64(s["D"][0], s["B"][0])
        S = torch.empty((K, B, nst, ns // 10), dtype=torch.float64, device="cuda")
        q, p = s["polQ"].long(), s["polP"].long()
        for c in range(K):
            raw = s["v"][:, c]
            v = torch.view_as_complex(raw.to(torch.float64)) if case["int8"] else _nibbles(raw)
            v = torch.stack([v[:, q], v[:, p]], -1)                     # [s][a][2]
            j = J[:, :, c]                                              # [p][a][2][2]
            w = (phi[:, :, c, None, None] * j).permute(0, 2, 1, 3).reshape(2 * B, 2 * A)
            E = (w @ v.reshape(ns, 2 * A).T).view(B, 2, ns // 10, 10)
            cov = (v.view(ns // 10, 10, A, 2, 1) * v.conj().view(ns // 10, 10, A, 1, 2)).sum(1)
            own = torch.stack([torch.einsum("paq,taqr,par->pt", j[:, :, x], cov, j[:, :, y].conj())
                               for x, y in ((0, 0), (1, 1), (0, 1))])
            xx = (E[:, 0].abs() ** 2).sum(-1) - own[0].real
            yy = (E[:, 1].abs() ** 2).sum(-1) - own[1].real
            xy = (E[:, 0] * E[:, 1].conj()).sum(-1) - own[2]
            S[c] = torch.stack([xx + yy, xx - yy, 2 * xy.real, -2 * xy.imag][:nst], 1) / (2 * A)
        off = S.amin(-1)
        scl = (S.amax(-1) - off) / 256
        return {"S": S, "out": None, "offsets": off.permute(1, 2, 0).contiguous(), "scales": scl.permute(1, 2, 0).contiguous()}
    if k == "products":
        s = _inputs(case, seed)
        n, ns = case["npointing"], case["nsamples"]
        lo, hi = s["S"][0].amin(1), s["S"][0].amax(1)
        x = None
        if case["floats"]:
            f = torch.from_numpy(_synthesis(_filter("int16"))).cuda().to(torch.float64).view(P, K)
            sign = torch.where(torch.arange(K, device="cuda") % 2 == 0, 1.0, -1.0)[:, None]
            x = torch.empty((n, ns * K, 2, 2), dtype=torch.float64, device="cuda")
            for i in range(n):
                X = torch.view_as_complex(torch.cat([s["hist"][i], s["e"][i]]).to(torch.float64))
                y = torch.fft.ifft(X, dim=1, norm="forward") * sign          # [12 + ns][K][2]
                acc = sum(f[p][:, None] * y[P - p:P - p + ns] for p in range(P))
                x[i] = torch.view_as_real(acc / K).reshape(ns * K, 2, 2)
        return {"psrfits": None, "offsets": lo.double(), "scales": (hi.double() - lo.double()) / 256, "vdif": None, "samples": x}
    s = _inputs(case, seed)
    B = _tile_beam64(s["az"], s["za"], float(s["bfreq"][0]), s["delays"], vgb.MWA_LATITUDE_RADIANS)
    J, phi = _jinv64(s["D"], B), _phase64(s["unit"], s["pos"], s["freqs"])
    return {"B": torch.view_as_real(B)[None], "J": torch.view_as_real(J), "phi": torch.view_as_real(phi),
            "W": torch.view_as_real(phi[..., None, None] * J)}
