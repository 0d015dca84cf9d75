"""Benchmark: real-time factor (data-seconds per wall-second) of the VCSBeam
voltage hot path on GB300.

Workload (one step = one data-second of the full band): 24 coarse channels x
128 tiles x 2 pols of 8-bit MWAX voltages (Gaussian sigma 16, clipped to
+-127, synthetic and seeded), forward fine PFB 12 taps x 128 channels, one
tied-array beam + the incoherent beam, full Stokes at 100 us into channel-
spliced 8-bit PSRFITS rows, and the inverse PFB back to 1.28 MHz 8-bit VDIF,
FP32 throughout. Each step reads 15.7 GB of voltages (> the 129 MB L2, so no
flush is needed); two distinct seconds stay resident and alternate.

  value  device-resident input: voltages already in HBM when timing starts
  e2e    the same through the pipeline's host API: every step copies its
         second of voltages from pinned host memory to the device and its
         PSRFITS + VDIF products back
  multibeam  the many-beam path (vgb_multibeam_*): 256 beams on 128 tiles
         (8-bit, Stokes I) and 1024 beams on 256 tiles (4-bit, full Stokes),
         1 ms integrations into 8-bit PSRFITS, one coarse channel-second per
         step, in four weight precisions: split BF16 and single FP16/BF16 on
         the tensor cores, FP32 on the CUDA cores (the plain baseline)
  reference_cuda  the reference's own CUDA kernels (unmodified, compiled for
         sm_103a) on one coarse channel-second of the same workload, timed on
         the same GPU beside the product (a baseline, like the CPU one)
  --impl reference  the reference's CPU path timed on the host cores: the
         reference has no CPU implementation of its kernels, so this is the
         oracle's OpenMP FP32 transcription of them (oracle/oracle.c).
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import tempfile
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(ROOT, "mwa-vcsbeam_gb300"))

METRIC = "real-time factor (data-s/wall-s) on 1 GB300, 1→1024 beams, vs plain FP32 at ≤1e-3"
UNIT = "data-s/wall-s"
NCC, NANT, NBLK, K, P = 24, 128, 20, 128, 12
NI = 2 * NANT
NSPEC = NBLK * 500
SECOND_BYTES = NBLK * NI * 64000 * 2           # one coarse channel, one second
BEAM_KERNEL_DRAM_BYTES_PER_CC = (1.322368e9 + 86.6944e6) / 2
# the same for the three-CTAs-per-SM shape (variant 5): 1.321426 GB read + 85.7 MB written
BEAM_TM_KERNEL_DRAM_BYTES_PER_CC = (1.321426e9 + 85.663232e6) / 2
# Algorithmic FP32 flops of the fused PFB + beamformer per (RF input, fine
# spectrum): the 12-tap weighted overlap-add of 128 complex samples
# (12 x 2 x 2 x 128 = 6,144), a 128-point complex FFT counted as 5 N log2 N
# (4,480), and the beam back end per input and fine channel -- half of a
# tile's J^-1 v (32), its sums into ex / ey (4), the autocorrelation terms
# (16) and the incoherent power (8) -- (60 / 2) x 128 = 3,840.
BEAM_KERNEL_FLOPS_PER_INPUT_SPECTRUM = 6144 + 4480 + 3840


def out_bytes(ncc):
    """PSRFITS bytes (the tied-array beam's four Stokes and the incoherent
    beam's Stokes I), VDIF bytes and scale/offset bytes per data-second."""
    return NSPEC * 5 * ncc * K, ncc * NSPEC * 544, 2 * ncc * 5 * K * 4


WORKLOAD = ("full band: 24 coarse channels x 128 tiles x 2 pols, 8-bit MWAX voltages (sigma 16), "
            "fine PFB 12x128 -> 1 tied-array beam (full Stokes) + incoherent beam (Stokes I), 100 us -> 8-bit PSRFITS; "
            "inverse PFB -> 8-bit VDIF; FP32")


def dist_env():
    return int(os.environ.get("RANK", 0)), int(os.environ.get("LOCAL_RANK", 0)), int(os.environ.get("WORLD_SIZE", 1))


# --------------------------------------------------------------------------
# clocks
# --------------------------------------------------------------------------
class ClockSampler:
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int):
        self.path = tempfile.mktemp(suffix=".csv")
        self.proc = None
        try:
            self.fh = open(self.path, "w")
            self.proc = subprocess.Popen(["nvidia-smi", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                                          "-lms", "200", "-i", str(gpu_index)], stdout=self.fh,
                                         stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        self.fh.close()
        sm, smax, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in open(self.path):
            parts = [x.strip() for x in line.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                smax.append(float(parts[2]))
            except ValueError:
                continue
            for name, val in zip(names, parts[5:9]):
                if val.lower().startswith("active"):
                    reasons.add(name)
        os.unlink(self.path)
        if not sm:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["no samples"], "samples": 0}
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": max(smax), "reasons": sorted(reasons),
                "samples": len(sm)}


# --------------------------------------------------------------------------
# synthetic workload on the device
# --------------------------------------------------------------------------
def make_voltages(torch, nsec: int, ncc: int, seed: int):
    """[nsec][cc][block][input][sample][2] int8, Gaussian sigma 16 clipped."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    out = torch.empty((nsec, ncc, SECOND_BYTES), dtype=torch.int8, device="cuda")
    for s in range(nsec):
        for cc in range(ncc):
            x = torch.randn(SECOND_BYTES, generator=g, device="cuda", dtype=torch.float32)
            out[s, cc] = x.mul_(16.0).round_().clamp_(-127, 127).to(torch.int8)
            del x
    return out


def make_weights(torch, vgb, SY, ncc):
    """W [cc][tile][128][2][2] complex float = phi * J^-1 built on the device
    in FP64 (vgb_jones, vgb_phase, vgb_weights)."""
    D = SY.calibration_jones(NANT, K, seed=11)
    B = SY.identity_beam(1, NANT)
    east, north, height, cable = SY.tile_layout(NANT, seed=7)
    unit = SY.unit_vectors(45.0, 20.0)

    def d(a):
        a = np.ascontiguousarray(a)
        if np.iscomplexobj(a):
            a = a.view(np.float64)
        return torch.from_numpy(a.copy()).cuda()

    J = torch.empty(NANT * K * 8, dtype=torch.float64, device="cuda")
    vgb.jones(d(D), d(B), 1, NANT, K, J)
    W = torch.empty((ncc, NANT * K, 8), dtype=torch.float32, device="cuda")
    phi = torch.empty(NANT * K * 2, dtype=torch.float64, device="cuda")
    geo = [d(x) for x in (unit, east, north, height, cable)]
    for cc in range(ncc):
        freqs = d(SY.fine_chan_freqs_hz(SY.coarse_chan_start_hz(cc)))
        vgb.phase(*geo, freqs, 1, NANT, K, SY.MWA_ALTITUDE_METRES, phi)
        vgb.weights(J, phi, NANT * K, W[cc])
    torch.cuda.synchronize()
    return W


def make_tracking(torch, SY, ncc, nsec):
    """Device tables for per-second tracking (vgb_pipeline_set_tracking): the
    calibration D of make_weights for every coarse channel, every tile's
    dipole delays pointed at az 45 deg / za 20 deg, the tile layout, the
    fine-channel and beam frequencies, and one pointing per second drifting
    in azimuth at the sidereal rate from (45 deg, 20 deg)."""
    D = np.broadcast_to(SY.calibration_jones(NANT, K, seed=11), (ncc, NANT, K, 2, 2))
    delays = np.broadcast_to(SY.tile_delays(45.0, 20.0), (NANT, 16))
    east, north, height, cable = SY.tile_layout(NANT, seed=7)
    chan_f = np.stack([SY.fine_chan_freqs_hz(SY.coarse_chan_start_hz(cc)) for cc in range(ncc)])
    beam_f = np.array([SY.coarse_chan_start_hz(cc) + 640000 for cc in range(ncc)], np.float64)
    omega = 2.0 * np.pi / 86164.0905
    az = np.radians(45.0) + omega * np.arange(nsec)
    za = np.full(nsec, np.radians(20.0))

    def d(a, dt=None):
        a = np.ascontiguousarray(a, dtype=dt)
        if np.iscomplexobj(a):
            a = a.view(np.float64)
        if a.dtype == np.uint32:
            a = a.view(np.int32)
        return torch.from_numpy(a.copy()).cuda()

    return dict(D=d(D, np.complex128), delays=d(delays, np.uint32), east=d(east), north=d(north), height=d(height),
                cable=d(cable), chan_freqs_hz=d(chan_f), beam_freqs_hz=d(beam_f), az=d(az), za=d(za),
                href=SY.MWA_ALTITUDE_METRES, latitude=-0.4660608448386394, pa_correction=True)


def config_dict(ncc):
    """The workload both arms report (identical keys and values)."""
    return {"workload": WORKLOAD if ncc == NCC else WORKLOAD.replace("24 coarse", f"{ncc} coarse"),
            "ncc": ncc, "ntiles": NANT, "nbeams": 1, "nstokes": 4,
            "tracking": "J^-1, phi and W rebuilt every data-second (vmCalcJonesAndDelays: pointing drifting at "
                        "the sidereal rate, primary beam B, inverse Jones, geometric phase)",
            "l2": "inputs larger than L2: each step reads a different 15.7 GB second"}


# --------------------------------------------------------------------------
# CPU baseline: the oracle's OpenMP FP32 transcription of the reference kernels
# --------------------------------------------------------------------------
def cpu_sample(nspec: int):
    """Time one bounded sample: `nspec` fine spectra of one coarse channel
    through the PFB + beamformer, the renormalise of those spectra and the
    reference-algorithm inverse PFB + VDIF of the same time span."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle as O
    import synthetic as SY

    nblk = (nspec + 11) // 500 + 2
    htr = O.mwax_buffer(5, nblk, NI)
    h = SY.analysis_filter_int16()
    D = SY.calibration_jones(NANT, K, seed=11)
    J = O.calc_j(D, SY.identity_beam(1, NANT))
    e_, n_, h_, c_ = SY.tile_layout(NANT, seed=7)
    phi = O.calc_phi(SY.unit_vectors(45.0, 20.0), e_, n_, h_, c_, SY.fine_chan_freqs_hz(SY.coarse_chan_start_hz(0)))
    W = (phi[0][:, :, None, None] * J[0]).astype(np.complex64)
    coeffs = SY.synthesis_filter(scale=SY.synthesis_scale(h))
    ftr, fti = O.ipfb_table(coeffs, K)
    # the per-second tables of one coarse channel (vmCalcJ + vmCalcPhi, the
    # reference's host code; B from the same beam model stands outside both
    # arms' CPU work here): charged at the sample's share of a second
    t0 = time.perf_counter()
    O.calc_j(D, SY.identity_beam(1, NANT))
    O.calc_phi(SY.unit_vectors(45.0, 20.0), e_, n_, h_, c_, SY.fine_chan_freqs_hz(SY.coarse_chan_start_hz(0)))
    t_tables = time.perf_counter() - t0
    t0 = time.perf_counter()
    S, e, inc, nt = O.pfb_beam32(htr, NI, 0, nspec, h, K, P, False, W, 1.0 / NI)
    _, _, _, nt2 = O.renormalise32(S)
    x = np.concatenate([np.zeros((P, K, 2), np.complex64), e], axis=0)
    _, nt3 = O.ipfb_vdif32(x, ftr, fti, P, 0, nspec * K)
    dt = time.perf_counter() - t0 + t_tables * nspec / NSPEC
    return dt, max(nt, nt2, nt3)


def cpu_baseline_line(target_s: float = 12.0):
    dt, nt = cpu_sample(20)                      # calibrate
    nspec = int(min(NSPEC, max(20, 20 * target_s / max(dt, 1e-3))))
    dt, nt = cpu_sample(nspec)
    data_s = nspec / NSPEC / NCC                 # data-seconds of the full band
    return {"value": data_s / dt, "unit": UNIT, "cores": nt, "kind": "port",
            "sample": f"{nspec} fine spectra of 1 of 24 coarse channels ({nspec / NSPEC * 1e3:.0f} ms of one channel): "
                      f"PFB + beam + renormalise + inverse PFB/VDIF, {dt:.1f} s on {nt} threads"}


# --------------------------------------------------------------------------
# the reference's own CUDA build on the same GPU (a baseline, like the CPU one)
# --------------------------------------------------------------------------
def reference_cuda_section(smart: bool = False, reps: int = 3):
    """The unmodified VCSBeam kernels (oracle/_ref/*.cubin, compiled from the
    reference's pfb.cpp and form_beam.cpp by oracle/build_ref.sh) driven by
    oracle/ref_harness.cu with the reference's launch shapes, memsets and
    cuFFT calls, on one coarse channel-second of the bench workload (128
    tiles, 1 beam, full Stokes): forward PFB (vmWOLAChunk..vmPackChunk),
    beamformer (vmApplyJChunk + vmBeamformChunk), renormalise (the kernel of
    vmSendSToFits) and inverse PFB (the kernel of cu_invert_pfb). Device time
    between CUDA events only, the best of `reps` runs per stage (the
    reference's host repacking loops and synchronous copies are left out,
    which favours it). The reference runs one process per coarse channel, so
    its real-time factor for the 24-channel band on one GPU is 1 / (24 t)."""
    import ctypes

    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle as O
    import synthetic as SY

    path = os.path.join(ROOT, "oracle", "_ref", "libref_harness.so")
    if not os.path.exists(path):
        return {"unavailable": "oracle/_ref/libref_harness.so not built (needs the reference's cubins)"}
    h = ctypes.CDLL(path)
    h.refh_last_error.restype = ctypes.c_char_p
    if h.refh_init(os.path.join(ROOT, "oracle", "_ref").encode()):
        return {"unavailable": h.refh_last_error().decode()}
    V, I = ctypes.c_void_p, ctypes.c_int
    h.refh_fpfb.argtypes = [V, ctypes.c_size_t, I, I, V, I, I, V, I, V, V, V]
    h.refh_beamform.argtypes = [V, I, I, I, I, V, V, V, V, I, ctypes.c_double, I, V, V, V]
    h.refh_ipfb.argtypes = [V, V, V, V, I, I, I, I, V, V]
    h.refh_renormalise_timed.argtypes = [V, I, I, I, I, V, V, V, V]
    p = lambda a: a.ctypes.data_as(V)

    def chk(rc):
        if rc:
            raise RuntimeError(h.refh_last_error().decode())

    clocks = ClockSampler(0)
    htr = O.mwax_buffer(7, NBLK + 1, NI)
    filt = SY.analysis_filter_int16()
    i_idx = SY.legacy_input_order(NANT)
    flags = O.PFB_SMART if smart else O.PFB_FULL_PRECISION
    out = np.empty((NSPEC, K, NI), dtype=np.uint8 if smart else np.complex128)
    ms = ctypes.c_float()
    times = {}

    def best(call):
        vals = []
        for _ in range(reps + 1):          # the first run loads modules and plans cuFFT
            chk(call())
            vals.append(ms.value)
        return min(vals[1:])

    times["pfb"] = best(lambda: h.refh_fpfb(p(htr), htr.nbytes, NI, NSPEC, p(filt), K, P, p(i_idx), flags, None,
                                            p(out), ctypes.byref(ms)))
    J = O.calc_j(SY.calibration_jones(NANT, K, seed=11), SY.identity_beam(1, NANT))
    e_, n_, h_, c_ = SY.tile_layout(NANT, seed=7)
    phi = O.calc_phi(SY.unit_vectors(45.0, 20.0), e_, n_, h_, c_, SY.fine_chan_freqs_hz(SY.coarse_chan_start_hz(0)))
    polQ = np.ascontiguousarray(i_idx[0::2].astype(np.uint32))
    polP = np.ascontiguousarray(i_idx[1::2].astype(np.uint32))
    S = np.empty((1, NSPEC, 4, K), dtype=np.float32)
    e = np.empty((1, NSPEC, K, 2), dtype=np.complex128)
    times["beamform"] = best(lambda: h.refh_beamform(p(out), 0 if smart else 1, NSPEC, K, NANT, p(J), p(phi),
                                                     p(polQ), p(polP), 1, 1.0 / NI, 4, p(S), p(e), ctypes.byref(ms)))
    off = np.empty((1, 4, K), np.float32)
    sc = np.empty((1, 4, K), np.float32)
    u8 = np.empty(S.shape, np.uint8)
    times["renormalise"] = best(lambda: h.refh_renormalise_timed(p(S), 1, NSPEC, 4, K, p(off), p(sc), p(u8),
                                                                 ctypes.byref(ms)))
    coeffs = SY.synthesis_filter(scale=SY.synthesis_scale(filt))
    ftr, fti = O.ipfb_table(coeffs, K)
    x = np.concatenate([np.zeros((P, K, 2), np.complex128), e[0]], axis=0)
    ir = np.ascontiguousarray(x.real.astype(np.float32))
    ii = np.ascontiguousarray(x.imag.astype(np.float32))
    vo = np.empty((NSPEC * K, 2, 2), dtype=np.float32)
    times["ipfb"] = best(lambda: h.refh_ipfb(p(ir), p(ii), p(ftr), p(fti), P, NSPEC, K, 2, p(vo), ctypes.byref(ms)))
    clk = clocks.stop()
    t_cc = sum(times.values()) / 1e3
    return {"what": "the reference's own CUDA kernels (unmodified, compiled for sm_103a), one coarse channel-second, "
                    "128 tiles, 1 beam, full Stokes; device time only (host repacking and copies left out)",
            "mode": "PFB_SMART" if smart else "PFB_FULL_PRECISION", "ms_per_cc_s": times,
            "seconds_per_cc_second": t_cc, "value": 1.0 / (NCC * t_cc), "unit": UNIT, "clocks": clk}


# --------------------------------------------------------------------------
# arms
# --------------------------------------------------------------------------
def reference_arm(args, rank, world):
    if rank != 0:
        return
    for _ in range(args.warmup):
        cpu_sample(args.ref_spectra)
    vals, total_dt, nt = [], 0.0, 1
    for _ in range(args.steps):
        dt, nt = cpu_sample(args.ref_spectra)
        total_dt += dt
        vals.append(dt)
    data_s = args.steps * args.ref_spectra / NSPEC / NCC
    value = data_s / total_dt

    line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": 1e3 * total_dt / args.steps, "higher_is_better": True,
            "scaling": "strong", "vs_baseline": None, "dtype": "f32", "data": "synthetic", "impl": "reference",
            "config": config_dict(NCC),
            "cpu_baseline": {"value": value, "unit": UNIT, "cores": nt, "kind": "port",
                             "sample": f"{args.ref_spectra} fine spectra of 1 of 24 coarse channels per step "
                                       "(the oracle's OpenMP FP32 transcription of the reference kernels; the "
                                       "reference's per-second J/phi host loops charged at the sample's share)"},
            "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


def gb300_arm(args, rank, local_rank, world):
    import torch

    import synthetic as SY
    import vgb

    from sharding import RankContext, gather_splice, shard

    torch.cuda.set_device(local_rank)
    ctx = RankContext()
    vgb.lib()
    if args.pfb_variant:
        vgb.pfb_variant(args.pfb_variant)

    def barrier():
        ctx.barrier()
        torch.cuda.synchronize()

    max_over_ranks = ctx.max

    # one data-second's coarse channels split over the ranks (the reference's
    # one process per coarse channel); one rank takes --ncc of them
    mine = shard(NCC, rank, world) if world > 1 else range(args.ncc)
    ncc = len(mine)
    volt = make_voltages(torch, args.resident, ncc, seed=1234 + rank)
    W = make_weights(torch, vgb, SY, ncc)
    h = SY.analysis_filter_int16()
    syn = SY.synthesis_filter(scale=SY.synthesis_scale(h)).astype(np.float32)
    pipe = vgb.Pipeline(ncc, NANT, NBLK, nstokes=4, pfb_flags=0, do_ipfb=True, invw=1.0 / NI)
    pipe.set_filters(h, syn)
    trk = make_tracking(torch, SY, ncc, nsec=4 * (args.warmup + args.steps) + 64)
    pipe.set_tracking(**trk)
    stream = pipe.stream()

    # ---- device-resident throughput (each second replayed from a captured
    # CUDA graph; stage timing measured separately afterwards) ----------------
    for i in range(args.warmup):
        pipe.run_device(volt[i % args.resident])
    pipe.sync()
    barrier()
    clocks = ClockSampler(local_rank)
    ev0 = torch.cuda.Event(enable_timing=True)
    ev1 = torch.cuda.Event(enable_timing=True)
    ev0.record(stream)
    launches = 0
    for i in range(args.steps):
        pipe.run_device(volt[i % args.resident])
        launches += pipe.launch_count()
    ev1.record(stream)
    ev1.synchronize()
    barrier()
    clk = clocks.stop()
    elapsed_s = max_over_ranks(ev0.elapsed_time(ev1) / 1e3)
    ncc_all = ctx.sum(ncc)                  # channels all ranks process per step
    value = args.steps * ncc_all / NCC / elapsed_s
    # per-stage CUDA-event times (eager launches with events between stages)
    pipe.enable_timing(True)
    stage = np.zeros(5)
    nstage = max(3, min(args.steps, 10))
    for i in range(nstage):
        pipe.run_device(volt[i % args.resident])
        stage += np.array(pipe.stage_ms(5))
    pipe.enable_timing(False)
    stage /= nstage

    # the reference's --smart mode (PFB_SMART: FPGA rounding and 4-bit
    # demotion of the fine channels) through the same stages
    smart = vgb.Pipeline(ncc, NANT, NBLK, nstokes=4, pfb_flags=vgb.PFB_EMULATE_FPGA | vgb.PFB_COMPLEX_INT4,
                         do_ipfb=True, invw=1.0 / NI)
    smart.set_filters(h, syn)
    smart.set_weights(W, on_device=True)
    smart.enable_timing(True)
    sstage = np.zeros(4)
    for i in range(nstage + 1):
        smart.run_device(volt[i % args.resident])
        if i:
            sstage += np.array(smart.stage_ms())
    smart.close()
    sstage /= nstage
    smart_mode = {"pfb_flags": "PFB_EMULATE_FPGA | PFB_COMPLEX_INT4 (the reference's --smart)",
                  "rtf_device_eager": (ncc / NCC) / (sstage.sum() / 1e3),
                  "stage_ms": {"pfb_beam": sstage[0], "renormalise": sstage[1], "ipfb_vdif": sstage[2],
                               "history": sstage[3]}}

    # a filter as large as the reference's FINEPFB (peak tap 117,964): one
    # FP32 sum could pass 2^24, so the weighted overlap-add takes the exact
    # even/odd split sums the library picks for it; the int32 sums beside it
    hbig = (h.astype(np.int64) * 117964 // int(np.abs(h).max())).astype(np.int32)
    assert vgb.filter_wola_flags(hbig) == vgb.WOLA_FP32_SPLIT

    def eager_stages(pfb_flags):
        pl = vgb.Pipeline(ncc, NANT, NBLK, nstokes=4, pfb_flags=pfb_flags, do_ipfb=True, invw=1.0 / NI)
        pl.set_filters(hbig, syn)
        pl.set_weights(W, on_device=True)
        pl.enable_timing(True)
        st = np.zeros(4)
        for i in range(nstage + 1):
            pl.run_device(volt[i % args.resident])
            if i:
                st += np.array(pl.stage_ms())
        pl.close()
        return st / nstage

    bstage = eager_stages(0)
    istage = eager_stages(vgb.WOLA_INT32)
    finepfb_sized = {"filter": "the int16 prototype scaled to a peak tap of 117,964 (the reference's FINEPFB "
                               "range): one FP32 sum is not exact, the even/odd split sums are",
                     "wola": "FP32, even and odd taps summed apart and added once (exact)",
                     "rtf_device_eager": (ncc / NCC) / (bstage.sum() / 1e3),
                     "stage_ms": {"pfb_beam": bstage[0], "renormalise": bstage[1], "ipfb_vdif": bstage[2],
                                  "history": bstage[3]},
                     "int32_wola": {"rtf_device_eager": (ncc / NCC) / (istage.sum() / 1e3),
                                    "pfb_beam_ms": istage[0]}}

    # ---- the PFB alone (fine_pfb_offline: vmExecuteForwardPFB's packed
    # legacy-order output), 8 coarse channels from the reference's read
    # buffer layout, both output types --------------------------------------
    pfb_only = None
    if args.pfb_only:
        npc = min(8, ncc)
        blk = NI * 64000 * 2
        rbuf = torch.randint(-127, 128, (npc, (NBLK + 1) * blk), dtype=torch.int8, device="cuda")
        rv = vgb.reference_buffer_voltages(rbuf, NI, NBLK, npc, (NBLK + 1) * blk)
        dfilt = torch.from_numpy(h.astype(np.int32)).cuda()
        didx = torch.from_numpy(SY.legacy_input_order(NANT).astype(np.int32)).cuda()
        pfb_only = {"workload": f"{npc} coarse channels x 1 s, 128 tiles, packed to the legacy order "
                                "(vgb_fpfb; the reference's fine_pfb_offline)"}
        for name, flags, dt, per in (("smart_int4", vgb.PFB_SMART | vgb.WOLA_FP32, torch.uint8, 1),
                                     ("full_precision_complex_double", vgb.PFB_FULL_PRECISION | vgb.WOLA_FP32,
                                      torch.float64, 2)):
            pout = torch.empty(npc * NSPEC * K * NI * per, dtype=dt, device="cuda")
            for _ in range(2):
                vgb.fpfb(rv, npc, NSPEC, dfilt, didx, flags, pout, stream=stream)
            e0p, e1p = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0p.record(stream)
            for _ in range(3):
                vgb.fpfb(rv, npc, NSPEC, dfilt, didx, flags, pout, stream=stream)
            e1p.record(stream)
            e1p.synchronize()
            ms = e0p.elapsed_time(e1p) / 3 / npc
            nbytes = pout.numel() * pout.element_size() / npc
            pfb_only[name] = {"ms_per_cc_s": ms, "rtf_24cc": 1e3 / (ms * NCC),
                              "write_gbs": nbytes / (ms * 1e-3) / 1e9}
            del pout
        del rbuf
        torch.cuda.empty_cache()

    # ---- end to end through the host API ------------------------------------
    psr_b, vdif_b, stat_b = out_bytes(ncc)
    e2e = None
    if args.e2e_steps > 0:
        hin = torch.empty(ncc * SECOND_BYTES, dtype=torch.int8, pin_memory=True)
        hin.copy_(volt[0].reshape(-1))
        ps = torch.empty(NSPEC * 4 * ncc * K, dtype=torch.uint8, pin_memory=True)
        vd = torch.empty(vdif_b, dtype=torch.uint8, pin_memory=True)
        off = torch.empty(ncc * 4 * K, dtype=torch.float32, pin_memory=True)
        scl = torch.empty(ncc * 4 * K, dtype=torch.float32, pin_memory=True)
        ips = torch.empty(NSPEC * ncc * K, dtype=torch.uint8, pin_memory=True)
        ioff = torch.empty(ncc * K, dtype=torch.float32, pin_memory=True)
        iscl = torch.empty(ncc * K, dtype=torch.float32, pin_memory=True)
        pipe.set_host_outputs(ps, off, scl, vd)
        pipe.set_host_incoh(ips, ioff, iscl)
        del volt
        psv = ps.numpy().reshape(NSPEC, 4, ncc * K)
        offv, sclv = off.numpy().reshape(ncc, 4, K), scl.numpy().reshape(ncc, 4, K)
        vdv = vd.numpy().reshape(ncc, NSPEC, 544)
        ipsv = ips.numpy().reshape(NSPEC, 1, ncc * K)
        ioffv, isclv = ioff.numpy().reshape(ncc, 1, K), iscl.numpy().reshape(ncc, 1, K)

        def e2e_step():
            pipe.run_host(hin)
            if world > 1:                   # the channel splice at the writer rank, host-staged
                pipe.sync()
                gather_splice(ctx, NCC, psv, offv, sclv, vdv)
                gather_splice(ctx, NCC, ipsv, ioffv, isclv)

        # the host link's own rate on this machine: one second of voltages
        # pinned -> device with a single copy, beside the pipeline's numbers
        # (taken before and after the timed steps: the link is shared with
        # the machine's other GPUs)
        def link_rate():
            dst = torch.empty(ncc * SECOND_BYTES, dtype=torch.int8, device="cuda")
            dst.copy_(hin, non_blocking=True)
            torch.cuda.synchronize()
            l0, l1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            l0.record()
            dst.copy_(hin, non_blocking=True)
            l1.record()
            l1.synchronize()
            del dst
            torch.cuda.empty_cache()
            return hin.numel() / (l0.elapsed_time(l1) / 1e3) / 1e9

        link_gbs = link_rate()
        for _ in range(min(args.warmup, 3)):
            e2e_step()
        pipe.sync()
        barrier()
        t0 = time.perf_counter()
        e2e_steps = max(1, min(args.steps, args.e2e_steps))
        done = []                           # each second's completion on the pipeline's stream
        for _ in range(e2e_steps):
            e2e_step()
            ev = torch.cuda.Event(enable_timing=True)
            ev.record(stream)
            done.append(ev)
        pipe.sync()
        barrier()
        e2e_s = max_over_ranks(time.perf_counter() - t0)
        periods = np.array([done[i].elapsed_time(done[i + 1]) for i in range(len(done) - 1)])
        link_after = link_rate()
        e2e = {"value": e2e_steps * ncc_all / NCC / e2e_s, "unit": UNIT,
               "h2d_bytes_per_step": ncc * SECOND_BYTES,
               "d2h_bytes_per_step": psr_b + vdif_b + stat_b,
               "steps": e2e_steps, "ms_per_step": 1e3 * e2e_s / e2e_steps,
               "h2d_link_gbs": link_gbs, "h2d_link_gbs_after": link_after,
               "step_period_ms": ({"median": float(np.median(periods)), "p90": float(np.percentile(periods, 90)),
                                   "max": float(periods.max())} if periods.size else None),
               "link_bound": link_gbs * 1e9 / (ncc * SECOND_BYTES) * ncc_all / NCC,
               "path": "vgb_pipeline_run_host from pinned host memory, products (tied-array PSRFITS rows, "
                       "incoherent PSRFITS rows, VDIF frames, offsets, scales) back to pinned host buffers; "
                       "next second's copy overlaps this second's compute" +
                       ("; each rank's rows gathered and spliced at rank 0 (gloo, host-staged)" if world > 1 else "")}
    pipe.close()

    # ---- roofline of the dominant kernel (fused PFB + beamformer) -----------
    peaks = {}
    try:
        peaks = json.load(open(os.path.join(ROOT, "MEASURED_PEAKS.json")))
    except Exception:
        pass
    peak = float(peaks.get("hbm_gbs", 6800.0))
    alg_bytes = ncc * SECOND_BYTES          # the voltages it must read, per launch
    # DRAM bytes (read + write) of one launch: the ncu capture of a 2-channel
    # launch (1.3224 GB read + 86.7 MB written) scaled by the channels
    # processed, since each channel's voltages are read once and its products
    # written once
    variant = vgb.pfb_variant_last()
    per_cc = BEAM_TM_KERNEL_DRAM_BYTES_PER_CC if variant == 5 else BEAM_KERNEL_DRAM_BYTES_PER_CC
    traffic = args.traffic if args.traffic is not None else ncc * per_cc
    achieved = alg_bytes / (stage[0] / 1e3) / 1e9
    # the compute side: FP32 flops of the launch against this GPU's measured
    # FP32 FMA throughput (scalar FFMA and packed FFMA2, the better of both)
    alg_flops = ncc * NI * NSPEC * BEAM_KERNEL_FLOPS_PER_INPUT_SPECTRUM
    try:
        fp32_ffma = vgb.fp32_peak(False)
        fp32_ffma2 = vgb.fp32_peak(True)
    except Exception:
        fp32_ffma = fp32_ffma2 = None
    fp32_peak = max(fp32_ffma or 0.0, fp32_ffma2 or 0.0) or None
    fp32_achieved = alg_flops / (stage[0] / 1e3) / 1e12
    compute = {"bound": "fp32 (CUDA cores)", "alg_flops_per_launch": alg_flops,
               "alg_flops_per_input_spectrum": {"wola": 6144, "fft_5nlog2n": 4480, "beam_back_end": 3840},
               "achieved": fp32_achieved, "unit": "TFLOP/s",
               "peak_ffma": fp32_ffma, "peak_ffma2": fp32_ffma2, "peak_source": "measured (vgb_fp32_peak)",
               "frac": (fp32_achieved / fp32_peak) if fp32_peak else None,
               # 14,464 flops per 256 voltage bytes: the HBM fraction this kernel
               # would reach running at the FP32 peak (its ceiling on the hbm roofline)
               "flops_per_byte": alg_flops / alg_bytes,
               "hbm_frac_at_fp32_peak": (alg_bytes / (alg_flops / (fp32_peak * 1e12)) / 1e9 / peak)
               if fp32_peak else None}
    if variant == 5:
        kname = "beam_tm_kernel (fused PFB + tied-array/incoherent beam + Stokes; three CTAs per SM)"
        limiter = ("not HBM: the FMA pipe and the shared-memory pipe, each ~60 % busy (ncu of a 2-channel "
                   "launch: issue 64.3 %, FMA pipe 56.5 %, shared-memory pipe 55 % of peak, math-pipe "
                   "throttle the second stall reason; 1.789 ms)")
    else:
        kname = "beam_kernel (fused PFB + tied-array/incoherent beam + Stokes)"
        limiter = ("not HBM: instruction issue, the FMA pipe and the shared-memory pipe, each ~60 % busy "
                   "(ncu of a 2-channel launch: issue 61.0 %, FMA pipe 58.8 %, shared-memory wavefronts "
                   "59.3 % of peak; DRAM 9.4 %)")
    roofline = {"kernel": kname, "bound": "hbm",
                "achieved": achieved, "peak": peak, "unit": "GB/s", "frac": achieved / peak,
                "peak_source": "measured" if "hbm_gbs" in peaks else "fallback",
                "traffic": traffic, "traffic_source": "ncu dram__bytes_read.sum + dram__bytes_write.sum of a "
                "2-channel launch, scaled to the channels of this launch" if args.traffic is None else "--traffic",
                "alg_bytes_per_launch": alg_bytes,
                "limiter": limiter, "pfb_variant": variant,
                "stage_ms": {"pfb_beam": stage[0], "renormalise": stage[1], "ipfb_vdif": stage[2],
                             "history": stage[3], "tracking_tables": stage[4]},
                "compute": compute}

    mb_section = None
    if rank == 0 and not args.no_multibeam:
        mb_section, mb_launches = multibeam_section(torch, vgb, SY, args.mb_iters, stream_iters=args.mb_stream_iters)

    line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": 1e3 * elapsed_s / args.steps, "higher_is_better": True,
            "scaling": "strong", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": config_dict(NCC if world > 1 else ncc),
            "run": {"step": "one data-second (24 coarse channels x 1 s)" +
                            (f"; rank r processes coarse channels shard(24, r, {world})" if world > 1 else ""),
                    "resident_seconds": args.resident,
                    "pfb_variant": vgb.pfb_variant_last(),
                    "cuda_graphs": "each second replayed from a captured CUDA graph (one per resident buffer "
                                   "and second parity), the per-second tracking tables inside it; stage_ms from "
                                   "a separate eager pass with events"},
            "roofline": roofline, "e2e": e2e, "gpu_launches": launches, "clocks": clk,
            "smart_mode": smart_mode, "finepfb_sized": finepfb_sized}
    if pfb_only is not None:
        line["pfb_only"] = pfb_only
    if mb_section is not None:
        mb_section["gpu_launches"] = mb_launches
        line["multibeam"] = mb_section
    if rank == 0 and not args.no_surrogate:
        line["surrogate"] = surrogate_section(torch, vgb, SY, args.sur_steps)
    if rank == 0 and world == 1 and not args.no_cpu:
        line["cpu_baseline"] = cpu_baseline_line(args.cpu_seconds)
    if rank == 0 and world == 1 and not args.no_ref_cuda:
        try:
            rc = reference_cuda_section()
        except Exception as exc:  # the baseline leg must not lose the product's line
            rc = {"unavailable": f"{type(exc).__name__}: {exc}"}
        line["reference_cuda"] = rc
        if "value" in rc:
            # the target: >= 2x the reference's own CUDA build for 1 beam at FP32 accuracy
            line["vs_reference_cuda"] = {"value": value / rc["value"], "e2e": (e2e["value"] / rc["value"]) if e2e
                                         else None, "target": 2.0}
    if rank == 0:
        print(json.dumps(line), flush=True)
    ctx.close()


# --------------------------------------------------------------------------
# many-beam tensor-core path (beams on the tensor cores vs the FP32 CUDA cores)
# --------------------------------------------------------------------------
MB_CASES = {
    # name: (tiles, beams, grid spacing deg, nstokes, 8-bit input, description)
    "C3": (128, 256, 0.02, 1, True, "24 cc x 128 fine ch, 128 tiles x 2 pols, 8-bit voltages, 256 beams "
                                    "(16x16 grid, 0.02 deg), Stokes I at 1 ms"),
    "C4": (256, 1024, 0.02, 4, False, "24 cc x 128 fine ch, 256 tiles x 2 pols, 4-bit voltages, 1024 beams "
                                      "(32x32 grid), full Stokes at 1 ms"),
}
MB_MODES = (("split_bf16", 0), ("fp16", 2), ("bf16", 1), ("fp32_cuda_cores", 3))


def multibeam_section(torch, vgb, SY, iters: int, cases=None, modes=None, nfine=K, stream_iters=3):
    """Each mode runs one coarse channel-second (128 fine channels x 10000
    samples) per step through vgb_multibeam_run on device-resident voltages;
    RTF counts 24 coarse channels per data-second. Stokes go to 8-bit PSRFITS
    bytes (renormalise included)."""
    peaks = {}
    try:
        peaks = json.load(open(os.path.join(ROOT, "MEASURED_PEAKS.json")))
    except Exception:
        pass
    peak_tf = float(peaks.get("bf16_tflops", 1900.0))
    out = {}
    launches = 0
    for name, (nant, npnt, spacing, nst, int8, desc) in MB_CASES.items():
        if cases and name not in cases:
            continue
        ns = 10000
        D = SY.calibration_jones(nant, nfine)
        Bj = SY.identity_beam(npnt, nant)
        e, n, h, c = SY.tile_layout(nant)
        side = int(round(np.sqrt(npnt)))
        az, za = SY.grid_pointings(side, spacing)
        unit = SY.unit_vectors(az, za)
        freqs = SY.fine_chan_freqs_hz(SY.coarse_chan_start_hz(0))[:nfine]
        polQ = np.arange(0, 2 * nant, 2, dtype=np.int32)
        polP = polQ + 1
        to = lambda a: torch.from_numpy(np.ascontiguousarray(
            a.view(np.float64) if a.dtype == np.complex128 else a)).cuda()
        nbytes = ns * nfine * 2 * nant * (2 if int8 else 1)
        g = torch.Generator(device="cuda").manual_seed(77)
        if int8:
            v = torch.randn(nbytes, device="cuda", generator=g).mul_(16).round_().clamp_(-127, 127).to(torch.int8)
        else:
            re = torch.randn(nbytes, device="cuda", generator=g).mul_(2.5).round_().clamp_(-8, 7).to(torch.int32)
            im = torch.randn(nbytes, device="cuda", generator=g).mul_(2.5).round_().clamp_(-8, 7).to(torch.int32)
            v = (((re & 15) << 4) | (im & 15)).to(torch.uint8)
        nint = ns // 10
        psr = torch.empty(npnt * nint * nst * nfine, dtype=torch.uint8, device="cuda")
        off = torch.empty(npnt * nst * nfine, device="cuda")
        scl = torch.empty_like(off)
        case = {"workload": desc, "step": f"one coarse channel-second ({nfine} fine channels x 10000 samples)",
                "alg_tflop_per_cc_s": 32.0 * npnt * nant * ns * nfine / 1e12, "modes": {}}
        S_keep = {}
        for mode, prec in MB_MODES:
            if modes and mode not in modes:
                continue
            mb = vgb.Multibeam(1, nfine, nant, npnt, ns, nstokes=nst, precision=prec,
                               input=vgb.MB_INT8 if int8 else vgb.MB_INT4)
            mb.set_geometry(to(unit), to(e), to(n), to(h), to(c))
            mb.set_jones(to(D), to(Bj), to(freqs), to(polQ), to(polP))
            n_it = iters if prec != 3 else max(1, iters // 4)
            for _ in range(2):
                mb.run(v, out=psr, offsets=off, scales=scl)
            torch.cuda.synchronize()
            st = torch.cuda.current_stream()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record(st)
            for _ in range(n_it):
                mb.run(v, out=psr, offsets=off, scales=scl, stream=st)
                launches += mb.launches()
            e1.record(st)
            e1.synchronize()
            ms = e0.elapsed_time(e1) / n_it
            mb.enable_timing(True)
            # the stage-timed run keeps its Stokes ([chan][beam][stokes][t]) for
            # the comparison of every mode against the plain FP32 path below
            S_mode = torch.empty(nfine * npnt * nst * nint, dtype=torch.float32, device="cuda")
            mb.run(v, S=S_mode, out=psr, offsets=off, scales=scl, stream=st)
            launches += mb.launches()
            stages = mb.stage_ms()
            pair = mb.last_pair()
            S_keep[mode] = S_mode
            mb.close()
            if vgb.check_device_status() != 0:
                raise RuntimeError("device status raised in the many-beam bench")
            alg = case["alg_tflop_per_cc_s"]
            beam_ms = stages["beam_gemm"]
            entry = {"ms_per_cc_s": ms, "rtf_24cc": 1e3 / (NCC * ms), "stage_ms": stages,
                     "beam_gemm_alg_tflops": alg / (beam_ms / 1e3)}
            if prec != 3:
                planes = 2 if prec == 0 else 1
                mma_tf = alg * planes * 256 / 250 / (beam_ms / 1e3)
                entry["roofline"] = {"kernel": f"mb_beam_pair_kernel (cta_group::2 over the two SMs of a TPC, "
                                               f"{pair} pairs)" if pair else "mb_beam_kernel", "bound": "tensor",
                                     "achieved": alg / (beam_ms / 1e3), "peak": peak_tf, "unit": "TFLOP/s",
                                     "frac": alg / (beam_ms / 1e3) / peak_tf,
                                     "mma_issued_tflops": mma_tf, "mma_frac": mma_tf / peak_tf,
                                     "peak_source": "measured" if "bf16_tflops" in peaks else "fallback"}
            case["modes"][mode] = entry
        # end to end: 8 coarse channel-seconds per call from pinned host memory
        # (the caller's stream completes once a call's products are on the
        # host, so the next call's compute waits for the previous call's last
        # download: a batch of 8 spreads that over 8 channel-seconds)
        # through vgb_multibeam_run_host (uploads, compute and downloads overlap)
        if name == "C4" and stream_iters > 0:
            ncs = 8
            for mode, prec in MB_MODES:
                if prec == 3 or (modes and mode not in modes):
                    continue
                mb = vgb.Multibeam(ncs, nfine, nant, npnt, ns, nstokes=nst, precision=prec,
                                   input=vgb.MB_INT8 if int8 else vgb.MB_INT4)
                mb.set_geometry(to(unit), to(e), to(n), to(h), to(c))
                rep = lambda a: np.ascontiguousarray(np.stack([a] * ncs))
                mb.set_jones(to(rep(D)), to(rep(Bj)), to(np.concatenate([freqs] * ncs)), to(polQ), to(polP))
                vh = torch.empty(ncs * nbytes, dtype=torch.uint8).pin_memory()
                vh.view(ncs, nbytes).copy_(v.cpu().view(torch.uint8).expand(ncs, nbytes))
                oh = torch.empty(ncs * npnt * nint * nst * nfine, dtype=torch.uint8).pin_memory()
                offh = torch.empty(ncs * npnt * nst * nfine, dtype=torch.float32).pin_memory()
                sclh = torch.empty_like(offh).pin_memory()
                st = torch.cuda.current_stream()
                mb.run_host(vh, oh, offh, sclh, stream=st)
                st.synchronize()
                t0 = time.perf_counter()
                for _ in range(stream_iters):
                    mb.run_host(vh, oh, offh, sclh, stream=st)
                    launches += mb.launches()
                st.synchronize()
                dt = time.perf_counter() - t0
                mb.close()
                ccs = ncs * stream_iters
                case["modes"][mode]["e2e"] = {
                    "value": ccs / dt / NCC, "unit": UNIT, "ms_per_cc_s": 1e3 * dt / ccs,
                    "h2d_bytes_per_cc_s": nbytes, "d2h_bytes_per_cc_s": int(oh.numel() + 8 * offh.numel()) // ncs,
                    "path": f"vgb_multibeam_run_host, {ncs} coarse channel-seconds per call from pinned host memory, "
                            f"{stream_iters} calls timed (wall clock; {ccs / NCC:g} data-seconds of the full band), "
                            "products back to pinned host memory"}
                del vh, oh, offh, sclh
        m = case["modes"]
        # each tensor mode against the plain FP32 CUDA-core path on the same
        # voltages and tables (Stokes of the whole coarse channel-second,
        # largest |difference| over the largest |FP32 value| per Stokes
        # parameter), and the fastest mode within 1e-3 of it
        if "fp32_cuda_cores" in S_keep:
            ref = S_keep["fp32_cuda_cores"].view(nfine, npnt, nst, nint)
            scale = ref.abs().amax(dim=(0, 1, 3))
            for mode, Sm in S_keep.items():
                if mode == "fp32_cuda_cores":
                    continue
                d = (Sm.view(nfine, npnt, nst, nint) - ref).abs().amax(dim=(0, 1, 3)) / scale
                per = [float(x) for x in d.cpu()]
                m[mode]["vs_plain_fp32"] = {"stokes_rel_err": per, "max": max(per), "within_1e-3": max(per) <= 1e-3}
            ok = [k for k in m if k != "fp32_cuda_cores" and m[k].get("vs_plain_fp32", {}).get("within_1e-3")]
            if ok:
                best = min(ok, key=lambda k: m[k]["ms_per_cc_s"])
                case["fastest_within_1e-3_of_fp32"] = {
                    "mode": best, "rtf_24cc": m[best]["rtf_24cc"],
                    "vs_fp32_cuda_cores": m["fp32_cuda_cores"]["ms_per_cc_s"] / m[best]["ms_per_cc_s"],
                    "definition": "largest |S_mode - S_fp32| / largest |S_fp32| per Stokes parameter over every "
                                  "fine channel, beam and 1-ms integration of the coarse channel-second; the FP32 "
                                  "path is itself within 2e-5 of the FP64 oracle (tests)"}
        del S_keep
        if "fp32_cuda_cores" in m and "split_bf16" in m:
            case["split_bf16_vs_fp32_cuda_cores"] = m["fp32_cuda_cores"]["ms_per_cc_s"] / m["split_bf16"]["ms_per_cc_s"]
        if "fp32_cuda_cores" in m and "fp16" in m:
            case["fp16_vs_fp32_cuda_cores"] = m["fp32_cuda_cores"]["ms_per_cc_s"] / m["fp16"]["ms_per_cc_s"]
        out[name] = case
        del v, psr
        torch.cuda.empty_cache()
    return out, launches


# --------------------------------------------------------------------------
# learned primary-beam surrogate (the beam model's stand-in for many beams)
# --------------------------------------------------------------------------
def beam_sweep(torch, vgb, SY, counts=(1, 4, 16, 64, 256, 1024), nant=256, nfine=K, ns=10000):
    """Beams per coarse channel-second from 1 to 1024: the per-pointing CUDA-core
    beamformer (vgb_beamform_legacy: Stokes at every 100 us sample, the
    reference's own per-pointing structure) against the tensor-core path
    (vgb_multibeam, split BF16 and FP16, Stokes integrated to 1 ms), on one
    coarse channel-second of 4-bit legacy voltages from 256 tiles, full
    Stokes. One timed call each after a warm-up, CUDA events."""
    g = torch.Generator(device="cuda").manual_seed(5)
    nb = ns * nfine * 2 * nant
    re = torch.randn(nb, device="cuda", generator=g).mul_(2.5).round_().clamp_(-8, 7).to(torch.int32)
    im = torch.randn(nb, device="cuda", generator=g).mul_(2.5).round_().clamp_(-8, 7).to(torch.int32)
    v = (((re & 15) << 4) | (im & 15)).to(torch.uint8)
    del re, im
    polQ = torch.arange(0, 2 * nant, 2, dtype=torch.int32, device="cuda")
    polP = polQ + 1
    e, n, h, c = SY.tile_layout(nant)
    to = lambda a: torch.from_numpy(np.ascontiguousarray(
        a.view(np.float64) if a.dtype == np.complex128 else a)).cuda()
    freqs = SY.fine_chan_freqs_hz(SY.coarse_chan_start_hz(0))[:nfine]
    D = SY.calibration_jones(nant, nfine)

    def timed(fn):
        fn()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        fn()
        e1.record()
        e1.synchronize()
        return e0.elapsed_time(e1)

    rows = []
    for B in counts:
        row = {"beams": B}
        W = torch.randn(B * nant * nfine * 8, device="cuda", generator=g)
        S = torch.empty(B * ns * 4 * nfine, device="cuda")
        row["cuda_cores_per_pointing_ms"] = timed(lambda: vgb.beamform_legacy(
            v, 0, ns, nfine, nant, polQ, polP, W, B, 1.0 / (2 * nant), 4, S))
        del W, S
        side = int(np.ceil(np.sqrt(B)))
        az, za = SY.grid_pointings(side, 0.02)
        unit = SY.unit_vectors(az[:B], za[:B])
        for mode, prec in (("split_bf16", vgb.MB_SPLIT_BF16), ("fp16", vgb.MB_FP16)):
            mb = vgb.Multibeam(1, nfine, nant, B, ns, nstokes=4, precision=prec, input=vgb.MB_INT4)
            mb.set_geometry(to(unit), to(e), to(n), to(h), to(c))
            mb.set_jones(to(D), to(SY.identity_beam(B, nant)), to(freqs), polQ, polP)
            row[f"tensor_{mode}_ms"] = timed(lambda: mb.run(v))
            mb.close()
        torch.cuda.empty_cache()
        rows.append(row)
    if vgb.check_device_status() != 0:
        raise RuntimeError("device status raised in the beam sweep")
    return {"workload": f"one coarse channel-second: {nant} tiles x 2 pols, 4-bit legacy voltages, {nfine} fine "
                        f"channels x {ns} samples, full Stokes (per-pointing path at 100 us, tensor path "
                        f"integrated to 1 ms)", "rows": rows}


def sur_feed_beam_run(torch, vgb, SY, Bs, Bp, az, za, f_cc, ntile, nfreq, cc):
    """One coarse channel-second of the 1024-beam run (128 tiles, 4-bit
    voltages, split BF16, full Stokes) with the last tracked second's B (at
    the coarse channel's frequency f_cc) from the surrogate and from the plain
    model: the Stokes difference between the two, and the run's time."""
    nfine, ns, nst = 128, 10000, 4
    npnt = az.size
    D = SY.calibration_jones(ntile, nfine)
    e, n, h, c = SY.tile_layout(ntile)
    freqs = f_cc - 640e3 + 10e3 * np.arange(nfine)  # lower fine-channel edges
    polQ = np.arange(0, 2 * ntile, 2, dtype=np.int32)
    to = lambda a: torch.from_numpy(np.ascontiguousarray(
        a.view(np.float64) if a.dtype == np.complex128 else a)).cuda()
    g = torch.Generator(device="cuda").manual_seed(91)
    nb = ns * nfine * 2 * ntile
    re = torch.randn(nb, device="cuda", generator=g).mul_(2.5).round_().clamp_(-8, 7).to(torch.int32)
    im = torch.randn(nb, device="cuda", generator=g).mul_(2.5).round_().clamp_(-8, 7).to(torch.int32)
    v = (((re & 15) << 4) | (im & 15)).to(torch.uint8)
    mb = vgb.Multibeam(1, nfine, ntile, npnt, ns, nstokes=nst, precision=vgb.MB_SPLIT_BF16, input=vgb.MB_INT4)
    mb.set_geometry(to(SY.unit_vectors(az, za)), to(e), to(n), to(h), to(c))
    S = {}
    ms = 0.0
    for name, B in (("plain", Bp), ("surrogate", Bs)):
        Bcc = B.view(nfreq, -1)[cc].contiguous()
        mb.set_jones(to(D), Bcc, to(freqs), to(polQ), to(polQ + 1))
        S[name] = torch.empty(nfine * npnt * nst * (ns // 10), device="cuda")
        mb.run(v, S=S[name])
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        mb.run(v, S=S[name])
        e1.record()
        e1.synchronize()
        ms = e0.elapsed_time(e1)
    mb.close()
    Sp = S["plain"].view(nfine, npnt, nst, -1).transpose(0, 1).reshape(npnt, -1)
    Ss = S["surrogate"].view(nfine, npnt, nst, -1).transpose(0, 1).reshape(npnt, -1)
    # per beam: largest Stokes difference over channels, parameters and time,
    # relative to the beam's largest Stokes value from the plain model
    rel = ((Ss - Sp).abs().amax(1) / Sp.abs().amax(1).clamp_min(1e-30)).cpu().numpy()
    return {"config": f"{npnt} beams x {ntile} tiles, 4-bit, split BF16, full Stokes, coarse channel {cc}",
            "ms_per_cc_s": ms,
            "per_beam_rel_stokes_diff_vs_plain_model": {
                "median": float(np.median(rel)), "p90": float(np.percentile(rel, 90)), "max": float(rel.max()),
                "beams_within_1e-3": float((rel <= 1e-3).mean()), "beams_within_1e-2": float((rel <= 1e-2).mean())}}


def surrogate_section(torch, vgb, SY, steps: int):
    """Train the surrogate on the plain model (16 delay sets x 24 frequencies
    in 80-300 MHz x 65,536 directions above 10 deg elevation), validate it,
    and time B for 1024 beams x 128 tiles x 24 frequencies from the
    surrogate (with fallback) and from the plain model on the device."""
    nsets, nfreq = 16, 24
    delays, set_az, set_za = SY.tile_delay_sets(nsets, seed=11, return_dirs=True)
    freqs = np.linspace(80e6, 300e6, nfreq)
    s = vgb.Surrogate(nsets, batch=8192, seed=1)
    s.set_training(delays, freqs, ndir=65536)
    t0 = time.perf_counter()
    loss = s.train(steps, lr_max=2e-3, lr_min=1e-4)
    train_s = time.perf_counter() - t0
    val = {}
    for tol in (3e-2, 1e-2, 1e-3):
        mx, frac = s.validate(2_000_000, tol=tol)
        val[f"{tol:g}"] = {"cells_within": frac, "max_jones_error": mx}
    # the observation: all 128 tiles on trained delay set 0 (one analogue
    # pointing), 1024 tied-array beams on a 32 x 32 grid of 0.4 deg inside
    # that tile beam's main lobe
    npnt, ntile = 1024, 128
    gaz, gza = SY.grid_pointings(32, 0.4, np.degrees(set_az[0]), np.degrees(set_za[0]))
    az = torch.tensor(np.radians(gaz), device="cuda")
    za = torch.tensor(np.radians(gza), device="cuda")
    f = torch.tensor(freqs, device="cuda")
    tset = np.zeros(ntile, dtype=np.int64)
    ts = torch.tensor(tset, dtype=torch.int32, device="cuda")
    td = torch.tensor(delays[tset].astype(np.int32), device="cuda")
    Bs = torch.empty(nfreq * npnt * ntile * 8, dtype=torch.float64, device="cuda")
    Bp = torch.empty_like(Bs)

    def timed(fn, n=5):
        fn()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(n):
            r = fn()
        e1.record()
        e1.synchronize()
        return e0.elapsed_time(e1) / n, r

    out = {"workload": "MLP 6 -> 4 x 256 GELU -> 8, BF16 weights, FP32 accumulate; trained on the analytic tile "
                       "model that stands in for the FEE model (FEE parity unpinned: mwa_hyperbeam and its HDF5 "
                       "table are not available) (16 delay sets x 24 frequencies 80-300 MHz x 65,536 directions "
                       "above 10 deg); "
                       "queries: 1024 beams (32 x 32 grid, 0.4 deg, around the tiles' pointing) x 128 tiles "
                       "(trained delay set 0) x 24 frequencies, re-pointed every second for 10 s",
           "train_steps": steps, "train_s": train_s, "ms_per_train_step": 1e3 * train_s / max(steps, 1),
           "final_loss": float(loss[-100:].mean()), "validation": val}
    # 10 s of tracking: the pointings drift with the sky (azimuth advancing at
    # the sidereal rate, zenith angles held) and B is re-evaluated each second
    omega = 2.0 * np.pi / 86164.0905
    az_sec = [torch.remainder(az + omega * sec, 2.0 * np.pi).contiguous() for sec in range(10)]
    for tol in (1e-3, 3e-2):
        s.validate(2_000_000, tol=tol)
        ms_s, nfb = timed(lambda: sum(s.beam(a, za, f, ts, td, Bs) for a in az_sec), n=2)
        ms_p, _ = timed(lambda: [vgb.primary_beam(a, za, f, td, Bp) for a in az_sec], n=2)
        err = (Bs - Bp).abs().max().item()
        cc = 11
        run = sur_feed_beam_run(torch, vgb, SY, Bs, Bp, az_sec[-1].cpu().numpy(), za.cpu().numpy(), float(freqs[cc]),
                                ntile, nfreq, cc)
        out[f"inference_tol_{tol:g}"] = {"tracking_seconds": 10, "surrogate_ms_10s": ms_s,
                                         "plain_model_device_ms_10s": ms_p,
                                         "fallback_fraction": nfb / (10 * nfreq * npnt * ntile),
                                         "max_abs_B_difference": err, "beam_run": run}
    s.close()
    return out


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=100)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="gb300", choices=["gb300", "reference"])
    ap.add_argument("--resident", type=int, default=2, help="distinct seconds kept in HBM")
    ap.add_argument("--ncc", type=int, default=NCC, help="coarse channels (24 = the full band; fewer for "
                    "profiling captures; value stays in full-band data-seconds)")
    ap.add_argument("--e2e-steps", type=int, default=40)
    ap.add_argument("--cpu-seconds", type=float, default=12.0)
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--no-ref-cuda", action="store_true", help="skip timing the reference's own CUDA build")
    ap.add_argument("--ref-spectra", type=int, default=400, help="reference arm: spectra per step")
    ap.add_argument("--no-multibeam", action="store_true", help="skip the many-beam (C3/C4) section")
    ap.add_argument("--no-surrogate", action="store_true", help="skip the beam-surrogate section")
    ap.add_argument("--sur-steps", type=int, default=96000, help="surrogate training steps")
    ap.add_argument("--mb-iters", type=int, default=5, help="many-beam timed runs per mode")
    ap.add_argument("--mb-only", default=None, help="profiling: run only these many-beam cases (e.g. C4 or C3,C4) "
                    "and print their JSON; no bench line")
    ap.add_argument("--mb-modes", default=None, help="profiling: comma-separated precision modes")
    ap.add_argument("--mb-nfine", type=int, default=K, help="profiling: fine channels per case")
    ap.add_argument("--mb-beam-variant", type=int, default=0, choices=[0, 1, 2],
                    help="many-beam GEMM kernel: 0 automatic, 1 single CTA, 2 CTA pairs")
    ap.add_argument("--mb-stream-iters", type=int, default=30,
                    help="many-beam host-streaming calls timed, 8 coarse channel-seconds each (30: 10 data-seconds "
                         "of the full band; 0: skip)")
    ap.add_argument("--no-pfb-only", dest="pfb_only", action="store_false",
                    help="skip the PFB-only (fine_pfb_offline) section")
    ap.add_argument("--pfb-variant", type=int, default=0, choices=[0, 3, 4, 5, 8],
                    help="profiling: force the fused front end's variant (4 or 8 inputs per step, 5 the 4-input "
                         "shape at three CTAs per SM, 3 the warp-specialised kernel; 0 = timed choice)")
    ap.add_argument("--beam-sweep", action="store_true",
                    help="time 1..1024 beams per coarse channel-second on both beamformers and print their JSON")
    ap.add_argument("--traffic", type=float, default=None,
                    help="DRAM bytes per beam_kernel launch from an ncu capture (profiles/)")
    args = ap.parse_args()
    args.warmup = max(args.warmup, 3)
    rank, local_rank, world = dist_env()
    if args.beam_sweep:
        import torch

        import synthetic as SY
        import vgb

        vgb.lib()
        print(json.dumps(beam_sweep(torch, vgb, SY)), flush=True)
        return
    if args.mb_only:
        import torch

        import synthetic as SY
        import vgb

        vgb.lib()
        vgb.multibeam_beam_variant(args.mb_beam_variant)
        sec, nl = multibeam_section(torch, vgb, SY, args.mb_iters, cases=args.mb_only.split(","),
                                    modes=args.mb_modes.split(",") if args.mb_modes else None, nfine=args.mb_nfine,
                                    stream_iters=args.mb_stream_iters)
        sec["gpu_launches"] = nl
        print(json.dumps(sec), flush=True)
        return
    if args.impl == "reference":
        reference_arm(args, rank, world)
    else:
        gb300_arm(args, rank, local_rank, world)


if __name__ == "__main__":
    main()
