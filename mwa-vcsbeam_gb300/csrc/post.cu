// Table builders, detection post-processing and the legacy-input beamformer.
//
//  * tables: geometric phase (geometry.c:40-101), inverse Jones
//    (jones.c:97-157) and their product, the per-(tile, channel) weight
//    W = phi J^-1 the beam kernels apply. FP64 on the device, W rounded to FP32.
//  * renormalise: per-channel min/max scale-and-offset to 8 bits
//    (form_beam.cpp:408-449), writing the spliced multi-channel layout
//    directly when asked.
//  * incoherent beam of 4+4-bit legacy voltages (form_beam.cpp:60-87).
//  * beamformer for fine-channel voltages already in legacy layout
//    (v_IDX [s][c][i], 4+4-bit or complex FP64): vmApplyJ_kernel followed by
//    vmBeamform_kernel (form_beam.cpp:122-371) in one pass.
#include <algorithm>
#include <type_traits>

#include <cooperative_groups.h>

#include "vgb_launch.cuh"

namespace vgb {

// ---------------------------------------------------------------------------
// FP64 complex helpers with cuCmul's operation order.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double2 zmul(double2 a, double2 b)
{
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 zadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 zsub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }

// (float)d, round to nearest even, in integer operations. `bad` is set where
// the result is not a normal number (zero, infinities and NaN among them).
__device__ __forceinline__ float narrow(double d, bool &bad)
{
    const uint32_t hi = (uint32_t)__double2hiint(d), lo = (uint32_t)__double2loint(d);
    const uint32_t h = 2u * hi - 0x70000000u;                      // sign out, exponent bias 1023 -> 127
    bad |= h - 0x00200000u >= 0x1FC00000u;                         // FP32 exponent not in 1 .. 254
    uint32_t u = __funnelshift_l(lo, h >> 1, 3);                   // truncated to 23 bits
    u += ((lo << 3) | (u & 1u)) > 0x80000000u;                     // above half, or half and odd
    return __uint_as_float(u | (hi & 0x80000000u));
}

// A call, so that the conversion instructions are never issued predicated off.
__device__ __noinline__ float4 narrow4_slow(double x, double y, double z, double w)
{
    return make_float4((float)x, (float)y, (float)z, (float)w);
}

__device__ __forceinline__ float4 narrow4(double x, double y, double z, double w)
{
    bool bad = false;
    const float4 f = make_float4(narrow(x, bad), narrow(y, bad), narrow(z, bad), narrow(w, bad));
    return bad ? narrow4_slow(x, y, z, w) : f;
}

// geometry.c:40-101 for one (pointing, tile, channel): phase terms use the
// reference's order of operations, 2*pi*dt*f. `u` is the pointing's (E, N, H)
// unit vector; the frequency is cast to whole Hz as the reference's is.
__device__ __forceinline__ double2 geometric_phase(const double *u, double east, double north, double height,
                                                   double cable, double href, double freq)
{
    const double L = cable - 0.0;
    const double w = (east - 0.0) * u[0] + (north - 0.0) * u[1] + (height - href) * u[2];
    const double dt = (w - L) / 299792458.0;
    const double f = (double)(uint32_t)freq;
    const double phase = 2.0 * 3.14159265358979323846 * dt * f;
    double s, co;
    sincos(phase, &s, &co);
    return make_double2(co, s);
}

__global__ void phase_kernel(const double *unit, const double *east, const double *north, const double *height,
                             const double *cable, const double *freqs, int npointing, int nant, int nchan,
                             double href, double2 *phi)
{
    const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long n = (long long)npointing * nant * nchan;
    if (idx >= n) return;
    const int c = idx % nchan;
    const int a = (idx / nchan) % nant;
    const int p = idx / ((long long)nchan * nant);
    phi[idx] = geometric_phase(unit + 3 * p, east[a], north[a], height[a], cable[a], href, freqs[c]);
}

// geometry.c:440-467 (calc_array_factor; Eq. A4 of Meyers et al. 2017): the
// tied-array response of the look direction's phases w at test direction
// psi, |sum_a conj(w_a) psi_a|^2 / nant^2. One block per test direction, the
// phases in FP64 with the geometric-delay kernel's operation order, the sum
// as the reference's sequential complex additions (thread 0 adds the tiles in
// order after each thread formed its products).
__global__ void array_factor_kernel(const double *look, const double *dirs, int npix, double freq,
                                    const double *east, const double *north, const double *height,
                                    const double *cable, double href, int nant, double *af)
{
    extern __shared__ double2 prod[];
    const int pix = blockIdx.x;
    if (pix >= npix) return;
    const double f = (double)(uint32_t)freq;
    for (int a = threadIdx.x; a < nant; a += blockDim.x) {
        double2 ph[2];
        for (int k = 0; k < 2; k++) {
            const double *u = k == 0 ? look : dirs + 3 * pix;
            const double L = cable[a] - 0.0;
            const double w = (east[a] - 0.0) * u[0] + (north[a] - 0.0) * u[1] + (height[a] - href) * u[2];
            const double dt = (w - L) / 299792458.0;
            const double phase = 2.0 * 3.14159265358979323846 * dt * f;
            double sn, cs;
            sincos(phase, &sn, &cs);
            ph[k] = make_double2(cs, sn);
        }
        // conj(w) * psi
        prod[a] = make_double2(ph[0].x * ph[1].x + ph[0].y * ph[1].y, ph[0].x * ph[1].y - ph[0].y * ph[1].x);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double2 s = make_double2(0.0, 0.0);
        for (int a = 0; a < nant; a++) s = make_double2(s.x + prod[a].x, s.y + prod[a].y);
        const double m = hypot(s.x, s.y) / nant;
        af[pix] = m * m;
    }
}

int launch_array_factor(const double *look, const double *dirs, int npix, double freq, const double *east,
                        const double *north, const double *height, const double *cable, double href, int nant,
                        double *af, cudaStream_t st)
{
    if (npix <= 0) return VGB_SUCCESS;
    array_factor_kernel<<<npix, 128, sizeof(double2) * nant, st>>>(look, dirs, npix, freq, east, north, height,
                                                                    cable, href, nant, af);
    return check_launch("array_factor_kernel");
}

// jones.c:97-157: J = inv2x2S(D[a][c] B[p][a] / ||D B||_F), zero if the norm is 0.
// jones.c:97-157 for one (pointing, tile, channel): J = D B normalised by
// its Frobenius norm, then inverted (zero when the norm is zero).
__device__ __forceinline__ void inverse_jones(const double2 *d, const double2 *b, double2 (&o)[4])
{
    double2 m[4];
    m[0] = zadd(zmul(d[0], b[0]), zmul(d[1], b[2]));
    m[1] = zadd(zmul(d[0], b[1]), zmul(d[1], b[3]));
    m[2] = zadd(zmul(d[2], b[0]), zmul(d[3], b[2]));
    m[3] = zadd(zmul(d[2], b[1]), zmul(d[3], b[3]));
    double F = 0.0;
    for (int i = 0; i < 4; i++) F += zmul(m[i], make_double2(m[i].x, -m[i].y)).x;
    F = sqrt(F);
    if (F == 0.0) {
        for (int i = 0; i < 4; i++) o[i] = make_double2(0.0, 0.0);
        return;
    }
    // one FP64 division instead of eight (FP64 is this GPU's slow pipe;
    // the products differ from the quotients by at most an ulp)
    const double rF = 1.0 / F;
    for (int i = 0; i < 4; i++) m[i] = make_double2(m[i].x * rF, m[i].y * rF);
    const double2 det = zsub(zmul(m[0], m[3]), zmul(m[1], m[2]));
    const double scale = 1.0 / (det.x * det.x + det.y * det.y);
    const double2 inv = make_double2(scale * det.x, -scale * det.y);
    const double2 ninv = make_double2(-inv.x, -inv.y);
    o[0] = zmul(inv, m[3]);
    o[1] = zmul(ninv, m[1]);
    o[2] = zmul(ninv, m[2]);
    o[3] = zmul(inv, m[0]);
}

// W = phi J in FP64, rounded to FP32 and stored as two float4:
// (w00, w01), (w10, w11). The rounding stays off the FP64 pipe, which the
// products keep busy (131,072 weights: 12.9 -> 10.9 us).
__device__ __forceinline__ void store_weight(double2 ph, const double2 (&j)[4], float4 *W)
{
    double2 w[4];
    for (int i = 0; i < 4; i++) w[i] = zmul(ph, j[i]);
    W[0] = narrow4(w[0].x, w[0].y, w[1].x, w[1].y);
    W[1] = narrow4(w[2].x, w[2].y, w[3].x, w[3].y);
}

__global__ void jones_kernel(const double2 *D, const double2 *B, int npointing, int nant, int nchan, double2 *J)
{
    const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long n = (long long)npointing * nant * nchan;
    if (idx >= n) return;
    const int c = idx % nchan;
    const int a = (idx / nchan) % nant;
    const int p = idx / ((long long)nchan * nant);
    double2 o[4];
    inverse_jones(D + 4 * ((long long)a * nchan + c), B + 4 * ((long long)p * nant + a), o);
    for (int i = 0; i < 4; i++) J[4 * idx + i] = o[i];
}

// W[p][a][c] = phi[p][a][c] * J[p][a][c].
__global__ void weights_kernel(const double2 *J, const double2 *phi, long long n, float4 *W)
{
    const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (idx >= n) return;
    const double2 j[4] = {J[4 * idx], J[4 * idx + 1], J[4 * idx + 2], J[4 * idx + 3]};
    store_weight(phi[idx], j, W + 2 * idx);
}

// ---------------------------------------------------------------------------
// Per-second tracking (vmCalcJonesAndDelays, jones.c:170-188): the pointing
// of the current second, then B (primary-beam kernel), then J^-1, phi and
// W = phi J^-1 for every (coarse channel, tile, fine channel) in one pass.
// ---------------------------------------------------------------------------

// One thread: the second's pointing from the per-second table (the last entry
// holds past its end), its (E, N, H) unit vector as calc_beam_geom sets it
// (geometry.c:226-286, from az and el = pi/2 - za), and the counter stepped
// for the next second.
__global__ void track_select_kernel(const double *az_tab, const double *za_tab, int nseconds,
                                    long long *counter, double *cur)
{
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const long long s = *counter;
    const int i = (int)(s < nseconds ? s : nseconds - 1);
    const double az = az_tab[i], za = za_tab[i];
    const double el = 0.5 * 3.14159265358979323846 - za;
    double saz, caz, sel, cel;
    sincos(az, &saz, &caz);
    sincos(el, &sel, &cel);
    cur[0] = az;
    cur[1] = za;
    cur[2] = cel * saz; // E
    cur[3] = cel * caz; // N
    cur[4] = sel;       // H
    *counter = s + 1;
}

// One thread per (cc, tile, fine channel): D [cc][a][c][2][2], B [cc][a][2][2]
// (one pointing, the coarse channel's beam frequency), freqs [cc][c].
__global__ void track_weights_kernel(const double2 *D, const double2 *B, const double *unit, const double *east,
                                     const double *north, const double *height, const double *cable,
                                     const double *freqs, int ncc, int nant, int nchan, double href, float4 *W)
{
    const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long n = (long long)ncc * nant * nchan;
    if (idx >= n) return;
    const int c = idx % nchan;
    const int a = (idx / nchan) % nant;
    const int cc = idx / ((long long)nchan * nant);
    double2 j[4];
    inverse_jones(D + 4 * idx, B + 4 * ((long long)cc * nant + a), j);
    const double2 ph = geometric_phase(unit, east[a], north[a], height[a], cable[a], href,
                                       freqs[(long long)cc * nchan + c]);
    store_weight(ph, j, W + 2 * idx);
}

int launch_track_select(const double *az_tab, const double *za_tab, int nseconds, long long *counter, double *cur,
                        cudaStream_t st)
{
    track_select_kernel<<<1, 32, 0, st>>>(az_tab, za_tab, nseconds, counter, cur);
    return check_launch("track_select_kernel");
}

int launch_track_weights(const double2 *D, const double2 *B, const double *unit, const double *east,
                         const double *north, const double *height, const double *cable, const double *freqs,
                         int ncc, int nant, int nchan, double href, float4 *W, cudaStream_t st)
{
    const long long n = (long long)ncc * nant * nchan;
    if (n == 0) return VGB_SUCCESS;
    track_weights_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(D, B, unit, east, north, height, cable, freqs,
                                                                      ncc, nant, nchan, href, W);
    return check_launch("track_weights_kernel");
}

int launch_phase(const double *unit, const double *east, const double *north, const double *height,
                 const double *cable, const double *freqs, int npointing, int nant, int nchan, double href,
                 double2 *phi, cudaStream_t st)
{
    const long long n = (long long)npointing * nant * nchan;
    if (n == 0) return VGB_SUCCESS;
    phase_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(unit, east, north, height, cable, freqs, npointing,
                                                               nant, nchan, href, phi);
    return check_launch("phase_kernel");
}

int launch_jones(const double2 *D, const double2 *B, int npointing, int nant, int nchan, double2 *J,
                 cudaStream_t st)
{
    const long long n = (long long)npointing * nant * nchan;
    if (n == 0) return VGB_SUCCESS;
    jones_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(D, B, npointing, nant, nchan, J);
    return check_launch("jones_kernel");
}

int launch_weights(const double2 *J, const double2 *phi, long long n, float4 *W, cudaStream_t st)
{
    if (n == 0) return VGB_SUCCESS;
    weights_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(J, phi, n, W);
    return check_launch("weights_kernel");
}

// ---------------------------------------------------------------------------
// renormalise_channels (form_beam.cpp:408-449)
// ---------------------------------------------------------------------------

// The float -> uint8 conversion of form_beam.cpp:443, (uint8_t)(val + 0.5)
// with val + 0.5 in FP64, as the reference's GPU build performs it: truncate
// to an integer and keep the low 8 bits, so a channel's maximum sample
// (256.5) becomes 0; NaN becomes 0. val is never negative here.
// One warp lane per channel; the 8 warps of a block split the samples.
constexpr int kRenormSplit = 8; // CTAs (one thread-block cluster) per (cc, pointing, stokes, 32 channels)

// Cluster of kRenormSplit CTAs over one (cc, pointing, stokes, 32 channels):
// CTA r scans samples [r n / 8, (r + 1) n / 8). Sequential-scan semantics of
// the reference: every partial starts from sample 0 and uses the same
// comparisons, so combining them in any order gives the same extremes (a NaN
// first sample makes the result NaN; other NaNs are skipped). The partials
// meet through distributed shared memory; each CTA then quantises its samples.
__global__ void __launch_bounds__(256) renorm_kernel(const RenormArgs a)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ float smin[8][32], smax[8][32];
    __shared__ float cmin[32], cmax[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int part = (int)cluster.block_rank();
    const int c = (blockIdx.x / kRenormSplit) * 32 + lane;
    const int st = blockIdx.y % a.nstokes, p = blockIdx.y / a.nstokes;
    const int cc = blockIdx.z;
    const bool live = c < a.nchan;
    const long long sstride = (long long)a.nstokes * a.nchan;
    const float *S = a.S + cc * a.S_cc + ((long long)p * a.nstep * a.nstokes + st) * a.nchan + (live ? c : 0);
    const int sb = (int)((long long)a.nstep * part / kRenormSplit);
    const int se = (int)((long long)a.nstep * (part + 1) / kRenormSplit);

    float mn, mx;
    if (a.st_mn) {
        // extremes gathered by the beam kernel: one pass over the samples
        const long long si = cc * a.stat_cc + ((long long)p * a.nstokes + st) * a.nchan + (live ? c : 0);
        if (a.st_nan0[si]) {
            mn = mx = __int_as_float(0x7fffffff);
        } else {
            mn = fkey_inv(a.st_mn[si]);
            mx = fkey_inv(a.st_mx[si]);
        }
    } else {
        const float s0 = S[0];
        mn = s0;
        mx = s0;
        // four independent loads in flight per lane (the scan order does not
        // change the extremes: a NaN first value stays, later NaNs are skipped)
        int s = sb + wid;
        for (; s + 24 < se; s += 32) {
            float v[4];
#pragma unroll
            for (int u = 0; u < 4; u++) v[u] = S[(long long)(s + 8 * u) * sstride];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                mn = (v[u] < mn ? v[u] : mn);
                mx = (v[u] > mx ? v[u] : mx);
            }
        }
        for (; s < se; s += 8) {
            const float v = S[(long long)s * sstride];
            mn = (v < mn ? v : mn);
            mx = (v > mx ? v : mx);
        }
        smin[wid][lane] = mn;
        smax[wid][lane] = mx;
        __syncthreads();
        if (wid == 0) {
            for (int w = 1; w < 8; w++) {
                const float v0 = smin[w][lane], v1 = smax[w][lane];
                mn = (v0 < mn ? v0 : mn);
                mx = (v1 > mx ? v1 : mx);
            }
            cmin[lane] = mn;
            cmax[lane] = mx;
        }
        cluster.sync(); // every CTA's partial is in its shared memory
        mn = s0;
        mx = s0;
        for (int r = 0; r < kRenormSplit; r++) {
            const float v0 = *cluster.map_shared_rank(&cmin[lane], r);
            const float v1 = *cluster.map_shared_rank(&cmax[lane], r);
            mn = (v0 < mn ? v0 : mn);
            mx = (v1 > mx ? v1 : mx);
        }
        cluster.sync(); // no CTA leaves while another still reads its partials
    }
    const float scale = (float)((double)(mx - mn) / 256.0);
    const float offset = mn;
    if (live) {
        uint8_t *o = a.out + cc * a.out_cc + p * a.out_p + st * a.out_st + c;
        const float rcp = 1.f / scale;
        int s = sb + wid;
        for (; s + 24 < se; s += 32) {
            float v[4];
#pragma unroll
            for (int u = 0; u < 4; u++) v[u] = S[(long long)(s + 8 * u) * sstride];
#pragma unroll
            for (int u = 0; u < 4; u++) o[(long long)(s + 8 * u) * a.out_s] = quant_u8(v[u], offset, scale, rcp);
        }
        for (; s < se; s += 8) o[(long long)s * a.out_s] = quant_u8(S[(long long)s * sstride], offset, scale, rcp);
        if (part == 0 && wid == 0) {
            const long long si = cc * a.stat_cc + ((long long)p * a.nstokes + st) * a.nchan + c;
            a.scales[si] = scale;
            a.offsets[si] = offset;
        }
    }
}

// Four adjacent channels per thread (16-byte reads, 4-byte writes), for Stokes
// and bytes aligned to that. A block takes kCh channels of one (cc, pointing,
// stokes) and a share of the samples.
//
// kStats: the extremes come from the beam kernel and a block reads its samples
// once (a second of one channel 38 -> 12 us). Otherwise a cluster of
// kRenormSplit blocks covers the samples, each keeps its share in shared memory
// (asynchronous copies, all in flight at once), the extremes meet through
// distributed shared memory and the bytes are formed from there, so the Stokes
// are read from memory once (six beams' second, 123 MB: 76 -> 54 us, now bound
// by the latencies between the phases; the incoherent beam's second of one
// channel 37 -> 9.5 us). kCh is the largest of 32, 16 and 8 whose share leaves
// five blocks per SM: with 100 KB and two the six beams took 71 us. The scan's
// semantics are renorm_kernel's, which serves the rest.
constexpr int kRenormTile = 44 * 1024; // bytes of samples a block may keep: five blocks per SM

__device__ __forceinline__ float4 min4(float4 a, float4 b)
{
    return make_float4(fminf(a.x, b.x), fminf(a.y, b.y), fminf(a.z, b.z), fminf(a.w, b.w));
}
__device__ __forceinline__ float4 max4(float4 a, float4 b)
{
    return make_float4(fmaxf(a.x, b.x), fmaxf(a.y, b.y), fmaxf(a.z, b.z), fmaxf(a.w, b.w));
}
__device__ __forceinline__ float4 shfl4(float4 v, int o)
{
    return make_float4(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o),
                       __shfl_xor_sync(0xffffffffu, v.z, o), __shfl_xor_sync(0xffffffffu, v.w, o));
}

template <int kCh, bool kStats> __global__ void __launch_bounds__(256, 5) renorm4_kernel(const RenormArgs a)
{
    namespace cg = cooperative_groups;
    constexpr int kThr = 256, kQ = kCh / 4, kRows = kThr / kQ; // threads per row, rows per pass
    extern __shared__ __align__(16) float4 rsm[];
    __shared__ float4 smin[kThr / 32][kQ], smax[kThr / 32][kQ];
    __shared__ __align__(16) float s_par[3][kCh]; // offset, scale, 1 / scale
    const int tid = threadIdx.x, q = tid % kQ, row = tid / kQ;
    const int nparts = kStats ? (int)gridDim.x / (a.nchan / kCh) : kRenormSplit;
    const int part = blockIdx.x % nparts, c0 = (blockIdx.x / nparts) * kCh, c = c0 + 4 * q;
    const int st = blockIdx.y % a.nstokes, p = blockIdx.y / a.nstokes, cc = blockIdx.z;
    const long long sstride = (long long)a.nstokes * a.nchan;
    const float *S = a.S + cc * a.S_cc + ((long long)p * a.nstep * a.nstokes + st) * a.nchan + c;
    const int sb = (int)((long long)a.nstep * part / nparts), se = (int)((long long)a.nstep * (part + 1) / nparts);
    const long long si = cc * a.stat_cc + ((long long)p * a.nstokes + st) * a.nchan + c0;

    float lo = 0.f, hi = 0.f; // thread t < kCh: the extremes of channel c0 + t
    if (kStats) {
        if (tid < kCh) {
            const bool nan0 = a.st_nan0[si + tid] != 0;
            lo = nan0 ? __int_as_float(0x7fffffff) : fkey_inv(a.st_mn[si + tid]);
            hi = nan0 ? __int_as_float(0x7fffffff) : fkey_inv(a.st_mx[si + tid]);
        }
    } else {
        cg::cluster_group cluster = cg::this_cluster();
        for (int s = sb + row; s < se; s += kRows)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(&rsm[(s - sb) * kQ + q])),
                         "l"(S + s * sstride)
                         : "memory");
        asm volatile("cp.async.commit_group;" ::: "memory");
        float4 mn = *reinterpret_cast<const float4 *>(S), mx = mn;
        asm volatile("cp.async.wait_group 0;" ::: "memory"); // each thread scans what it copied
        for (int s = sb + row; s < se; s += kRows) {
            const float4 v = rsm[(s - sb) * kQ + q];
            mn = min4(mn, v);
            mx = max4(mx, v);
        }
        // the warp's rows, then the block's warps, then the cluster's blocks
#pragma unroll
        for (int o = kQ; o < 32; o <<= 1) {
            mn = min4(mn, shfl4(mn, o));
            mx = max4(mx, shfl4(mx, o));
        }
        if ((tid & 31) < kQ) {
            smin[tid >> 5][q] = mn;
            smax[tid >> 5][q] = mx;
        }
        __syncthreads();
        float *bmin = &smin[0][0].x, *bmax = &smax[0][0].x;
        if (tid < kCh)
            for (int w = 1; w < kThr / 32; w++) {
                bmin[tid] = fminf(bmin[tid], bmin[w * kCh + tid]);
                bmax[tid] = fmaxf(bmax[tid], bmax[w * kCh + tid]);
            }
        cluster.sync(); // every block's partials are in its shared memory
        if (tid < kCh) {
            // a NaN first value makes both extremes NaN, other NaN are skipped
            const float s0 = a.S[(S - a.S) - 4 * q + tid];
            lo = hi = s0;
#pragma unroll
            for (int r = 0; r < kRenormSplit; r++) {
                lo = fminf(lo, cluster.map_shared_rank(bmin, r)[tid]);
                hi = fmaxf(hi, cluster.map_shared_rank(bmax, r)[tid]);
            }
            if (isnan(s0)) lo = hi = s0;
        }
    }
    if (tid < kCh) {
        const float scale = (float)((double)(hi - lo) / 256.0);
        s_par[0][tid] = lo;
        s_par[1][tid] = scale;
        s_par[2][tid] = 1.f / scale;
        if (part == 0) {
            a.scales[si + tid] = scale;
            a.offsets[si + tid] = lo;
        }
    }
    __syncthreads();
    if (!kStats) {
        // no block leaves while another still reads its partials: arrive here, wait at the
        // end. The first warp read the others' and arrives with a release, which orders
        // those reads (a relaxed arrival would not, and a block without samples could be
        // gone while they are in flight); ahead of the parameters it held up all warps
        // (six beams' second, with the inverse PFB: 135.6 against 133.2 us)
        static_assert(kCh <= 32, "the readers of other blocks are one warp");
        if (tid < 32) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        else asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    }
    const float4 off = *reinterpret_cast<const float4 *>(&s_par[0][4 * q]);
    const float4 scl = *reinterpret_cast<const float4 *>(&s_par[1][4 * q]);
    const float4 rcp = *reinterpret_cast<const float4 *>(&s_par[2][4 * q]);
    uint8_t *o = a.out + cc * a.out_cc + p * a.out_p + st * a.out_st + c;
    auto put = [&](int s, float4 v) { *reinterpret_cast<uint32_t *>(o + (long long)s * a.out_s) = quant4_u8(v, off, scl, rcp); };
    if (kStats) {
        int s = sb + row;
        for (; s + 3 * kRows < se; s += 4 * kRows) { // four loads in flight
            float4 v[4];
#pragma unroll
            for (int u = 0; u < 4; u++) v[u] = __ldcs(reinterpret_cast<const float4 *>(S + (s + u * kRows) * sstride));
#pragma unroll
            for (int u = 0; u < 4; u++) put(s + u * kRows, v[u]);
        }
        for (; s < se; s += kRows) put(s, *reinterpret_cast<const float4 *>(S + s * sstride));
    } else {
#pragma unroll 2
        for (int s = sb + row; s < se; s += kRows) put(s, rsm[(s - sb) * kQ + q]);
        __syncwarp();
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}

template <int kCh, bool kStats> static int launch_renorm4(const RenormArgs &a, int ncc, cudaStream_t st)
{
    auto kern = renorm4_kernel<kCh, kStats>;
    cudaLaunchConfig_t cfg = {};
    // with the extremes given: about eight blocks per SM
    const long long groups = (long long)(a.nchan / kCh) * a.npointing * a.nstokes * ncc;
    const long long parts = kStats ? std::max(1LL, std::min<long long>(a.nstep / 256 + 1, (8 * sm_count() + groups - 1) / groups))
                                   : kRenormSplit;
    cfg.gridDim = dim3((unsigned)(parts * (a.nchan / kCh)), a.npointing * a.nstokes, ncc);
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kStats ? 1 : kRenormSplit;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (!kStats) {
        cfg.dynamicSmemBytes = sizeof(float) * kCh * (size_t)((a.nstep + kRenormSplit - 1) / kRenormSplit);
        const int rc = check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kRenormTile),
                                  "cudaFuncSetAttribute(renorm4)");
        if (rc) return rc;
    }
    const int rc = check_cuda(cudaLaunchKernelEx(&cfg, kern, a), "cudaLaunchKernelEx(renorm4_kernel)");
    return rc ? rc : check_launch("renorm4_kernel");
}

int launch_renorm(const RenormArgs &a, int ncc, cudaStream_t st)
{
    if (a.nstep <= 0 || ncc <= 0) return VGB_SUCCESS;
    const auto low = [](const void *p) { return reinterpret_cast<uintptr_t>(p) & 15; };
    const bool aligned = !low(a.S) && !low(a.scales) && !low(a.offsets) && a.nchan % 32 == 0 && (low(a.out) & 3) == 0 &&
                         ((a.out_cc | a.out_p | a.out_s | a.out_st) & 3) == 0 && a.S_cc % 4 == 0 && a.stat_cc % 4 == 0;
    if (aligned && a.st_mn) return launch_renorm4<32, true>(a, ncc, st);
    const long long share = (long long)((a.nstep + kRenormSplit - 1) / kRenormSplit) * 4; // bytes per channel
    if (aligned && share * 32 <= kRenormTile) return launch_renorm4<32, false>(a, ncc, st);
    if (aligned && share * 16 <= kRenormTile) return launch_renorm4<16, false>(a, ncc, st);
    if (aligned && share * 8 <= kRenormTile) return launch_renorm4<8, false>(a, ncc, st);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kRenormSplit * ((a.nchan + 31) / 32), a.npointing * a.nstokes, ncc);
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kRenormSplit;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const int rc = check_cuda(cudaLaunchKernelEx(&cfg, renorm_kernel, a), "cudaLaunchKernelEx(renorm_kernel)");
    return rc ? rc : check_launch("renorm_kernel");
}

// ---------------------------------------------------------------------------
// Incoherent beam of 4+4-bit voltages (form_beam.cpp:60-87): exact integer
// sums of |v|^2 over all inputs. Eight lanes per (s, c) row of ninput bytes.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int nib(uint32_t x) { return ((int)(x << 28)) >> 28; }

__device__ __forceinline__ int power4(uint32_t w)
{
    int acc = 0;
#pragma unroll
    for (int b = 0; b < 4; b++) {
        const uint32_t byte = (w >> (8 * b)) & 0xFFu;
        const int re = nib(byte >> 4), im = nib(byte);
        acc += re * re + im * im;
    }
    return acc;
}

__global__ void incoh_kernel(const uint8_t *data, long long nrows, int ninput, float *incoh)
{
    const long long row = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 3;
    const int sub = threadIdx.x & 7;
    int acc = 0;
    if (row < nrows) {
        const uint8_t *r = data + row * ninput;
        if ((ninput & 31) == 0) {
            for (int off = sub * 4; off < ninput; off += 32)
                acc += power4(*reinterpret_cast<const uint32_t *>(r + off));
        } else {
            for (int off = sub; off < ninput; off += 8) acc += power4(r[off]);
        }
    }
    acc += __shfl_xor_sync(0xffffffffu, acc, 1);
    acc += __shfl_xor_sync(0xffffffffu, acc, 2);
    acc += __shfl_xor_sync(0xffffffffu, acc, 4);
    if (row < nrows && sub == 0) incoh[row] = (float)acc;
}

int launch_incoh(const uint8_t *data, long long nrows, int ninput, float *incoh, cudaStream_t st)
{
    if (nrows <= 0) return VGB_SUCCESS;
    const long long threads = nrows * 8;
    incoh_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, st>>>(data, nrows, ninput, incoh);
    return check_launch("incoh_kernel");
}

// ---------------------------------------------------------------------------
// Beamformer for legacy-layout fine voltages v[s][c][i].
// ---------------------------------------------------------------------------
// One (tile, sample) of one pointing costs 28 multiply-adds (the two Jones
// rows times the (Q, P) voltages, the sums, the tile's own power), so the FP32
// pipe bounds the kernels once the weights are read from registers rather
// than per sample. Sums are kept for pairs of samples in FP32x2, so one issue
// slot covers two multiply-adds and half of the slots are left for the loads
// and the widening of the voltages. One beam of 128 tiles x 128 channels x
// 10,000 samples of 4+4-bit voltages: 1,060 -> 252 us against the row kernel
// below (issue 63 %, ALU pipe 50 %); three beams of 2,000 samples of complex
// doubles: 1,440 -> 283 us (shared-memory pipe 57 %, DRAM 47 %, the FP64
// voltages read once instead of once per beam).

constexpr int kLS = 4; // samples of a row kernel's block: a call takes 65,535 times as many

// The 8 sums of a pair of samples over a tile: a[0..3] += ex, ey (re, im);
// a[4..7] += |ex|^2, |ey|^2, ex ey* (re, im). w: the two Jones rows with each
// value doubled into a pair; nw: minus the imaginary parts of w.
struct LegacyW {
    float2 xr0, xi0, xr1, xi1, yr0, yi0, yr1, yi1; // row x: (w00, w01), row y: (w10, w11)
    float2 nxi0, nxi1, nyi0, nyi1;
    __device__ __forceinline__ void set(float4 a, float4 b)
    {
        xr0 = make_float2(a.x, a.x); xi0 = make_float2(a.y, a.y); xr1 = make_float2(a.z, a.z); xi1 = make_float2(a.w, a.w);
        yr0 = make_float2(b.x, b.x); yi0 = make_float2(b.y, b.y); yr1 = make_float2(b.z, b.z); yi1 = make_float2(b.w, b.w);
        nxi0 = make_float2(-a.y, -a.y); nxi1 = make_float2(-a.w, -a.w);
        nyi0 = make_float2(-b.y, -b.y); nyi1 = make_float2(-b.w, -b.w);
    }
};

__device__ __forceinline__ void legacy_pair(float2 (&a)[8], const LegacyW &w, float2 qr, float2 qi, float2 pr, float2 pi)
{
    const float2 exr = __ffma2_rn(w.nxi1, pi, __ffma2_rn(w.xr1, pr, __ffma2_rn(w.nxi0, qi, __fmul2_rn(w.xr0, qr))));
    const float2 exi = __ffma2_rn(w.xi1, pr, __ffma2_rn(w.xr1, pi, __ffma2_rn(w.xi0, qr, __fmul2_rn(w.xr0, qi))));
    const float2 eyr = __ffma2_rn(w.nyi1, pi, __ffma2_rn(w.yr1, pr, __ffma2_rn(w.nyi0, qi, __fmul2_rn(w.yr0, qr))));
    const float2 eyi = __ffma2_rn(w.yi1, pr, __ffma2_rn(w.yr1, pi, __ffma2_rn(w.yi0, qr, __fmul2_rn(w.yr0, qi))));
    const float2 nexr = make_float2(-exr.x, -exr.y);
    a[0] = padd(a[0], exr);
    a[1] = padd(a[1], exi);
    a[2] = padd(a[2], eyr);
    a[3] = padd(a[3], eyi);
    a[4] = __ffma2_rn(exr, exr, __ffma2_rn(exi, exi, a[4]));
    a[5] = __ffma2_rn(eyr, eyr, __ffma2_rn(eyi, eyi, a[5]));
    a[6] = __ffma2_rn(exr, eyr, __ffma2_rn(exi, eyi, a[6]));
    a[7] = __ffma2_rn(exi, eyr, __ffma2_rn(nexr, eyi, a[7]));
}

// Stokes and e of one (pointing, sample, channel) from its 8 sums.
__device__ __forceinline__ void legacy_store(const LegacyArgs &a, int p, int s, int c, const float (&acc)[8])
{
    const float bnXX = acc[0] * acc[0] + acc[1] * acc[1] - acc[4];
    const float bnYY = acc[2] * acc[2] + acc[3] * acc[3] - acc[5];
    const float bxr = acc[0] * acc[2] + acc[1] * acc[3] - acc[6];
    const float bxi = acc[1] * acc[2] - acc[0] * acc[3] - acc[7];
    float *S = a.S + (((long long)p * a.nsamples + s) * a.nstokes) * a.nchan + c;
    S[0] = a.invw * (bnXX + bnYY);
    if (a.nstokes == 4) {
        S[a.nchan] = a.invw * (bnXX - bnYY);
        S[2 * a.nchan] = 2.0f * a.invw * bxr;
        S[3 * a.nchan] = -2.0f * a.invw * bxi;
    }
    if (a.e) a.e[((long long)p * a.nsamples + s) * a.nchan + c] = make_float4(acc[0], acc[1], acc[2], acc[3]);
}

// The tiles' (Q, P) input pairs into shared memory, checked against the row.
__device__ __forceinline__ void legacy_inputs(const LegacyArgs &a, uint32_t *pq)
{
    const uint32_t ni = 2u * a.nant;
    for (int ant = threadIdx.x; ant < a.nant; ant += blockDim.x) {
        uint32_t iq = __ldg(a.polQ + ant), ip = __ldg(a.polP + ant);
        if (iq >= ni || ip >= ni) {
            if (blockIdx.x == 0 && blockIdx.y == 0) atomicOr(a.status, kErrBadInput);
            iq = ip = 0;
        }
        pq[ant] = iq | (ip << 16);
    }
}

// 4+4-bit voltages. A block covers 32 channels x kG groups of kS samples; the
// 8 / kG warps of a group take tiles part, part + 8 / kG, ...: each weight is
// read once for kS samples. The voltages are staged transposed,
// [group][input][channel][kS samples] bytes, so that a warp's reads are
// contiguous and one read brings an input's kS samples; channels are rotated
// by the input's word so that the staging writes fall on all banks too. The
// warps' partial sums meet in shared memory, four samples of each group at a
// time.
constexpr int kL4C = 32, kLWarps = 8;
constexpr int kL4Red = kLWarps * 4 * 8 * kL4C; // floats of partial sums

template <int kS, int kG> static size_t legacy4_smem(int nant)
{
    return (size_t)2 * nant * kL4C * kS * kG + sizeof(float) * kL4Red + (size_t)nant * 4;
}

__device__ __forceinline__ uint32_t legacy4_slot(uint32_t i, uint32_t c)
{
    return i * kL4C + ((c + 4 * ((i >> 2) & 7)) & (kL4C - 1));
}

// Four samples' nibbles (bytes x + 8, x = -8 .. 7) as two pairs of floats.
__device__ __forceinline__ void legacy4_widen(uint32_t u, float2 &a, float2 &b)
{
    const float2 bias = make_float2(-8388616.0f, -8388616.0f); // 2^23 + 8
    a = padd(make_float2(__uint_as_float(__byte_perm(u, 0x4B000000u, 0x7540)),
                         __uint_as_float(__byte_perm(u, 0x4B000000u, 0x7541))),
             bias);
    b = padd(make_float2(__uint_as_float(__byte_perm(u, 0x4B000000u, 0x7542)),
                         __uint_as_float(__byte_perm(u, 0x4B000000u, 0x7543))),
             bias);
}

template <int kS, int kG> __global__ void __launch_bounds__(256, 2) legacy4_kernel(const LegacyArgs a)
{
    constexpr int kParts = kLWarps / kG;
    using Word = typename std::conditional<kS == 8, uint2, uint32_t>::type; // kS samples of one input
    extern __shared__ __align__(16) unsigned char lsm[];
    const int ni = 2 * a.nant, nw = ni / 4;
    float *red = reinterpret_cast<float *>(lsm);
    Word *vt = reinterpret_cast<Word *>(red + kL4Red);
    uint32_t *pq = reinterpret_cast<uint32_t *>(vt + (size_t)kG * ni * kL4C);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int c0 = blockIdx.x * kL4C, s0 = blockIdx.y * kS * kG;

    legacy_inputs(a, pq);
    // stage: lane = (channel 4 warp + lane % 4, word lane / 4 of 8), so 8 lanes
    // read a whole 32-byte sector of a row
    for (int g = 0; g < kG; g++) {
        const int cl = 4 * warp + (lane & 3), c = c0 + cl, sg = s0 + g * kS;
        const uint32_t *v32 = static_cast<const uint32_t *>(a.v) + ((long long)sg * a.nchan + c) * nw;
        const long long sstep = (long long)a.nchan * nw;
        const int ns = c < a.nchan ? min(kS, a.nsamples - sg) : 0;
        Word *vg = vt + (size_t)g * ni * kL4C;
        int power[kS];
#pragma unroll
        for (int s = 0; s < kS; s++) power[s] = 0;
#pragma unroll 2
        for (int wd = lane >> 2; wd < nw; wd += 8) {
            uint32_t w[kS];
#pragma unroll
            for (int s = 0; s < kS; s++) w[s] = s < ns ? __ldg(v32 + s * sstep + wd) : 0u;
            uint32_t t[kS / 4][4];
#pragma unroll
            for (int h = 0; h < kS / 4; h++) { // bytes [sample][input] -> [input][sample]
                const uint32_t l0 = __byte_perm(w[4 * h], w[4 * h + 1], 0x5140);
                const uint32_t l1 = __byte_perm(w[4 * h + 2], w[4 * h + 3], 0x5140);
                const uint32_t h0 = __byte_perm(w[4 * h], w[4 * h + 1], 0x7362);
                const uint32_t h1 = __byte_perm(w[4 * h + 2], w[4 * h + 3], 0x7362);
                t[h][0] = __byte_perm(l0, l1, 0x5410);
                t[h][1] = __byte_perm(l0, l1, 0x7632);
                t[h][2] = __byte_perm(h0, h1, 0x5410);
                t[h][3] = __byte_perm(h0, h1, 0x7632);
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if constexpr (kS == 8) vg[legacy4_slot(4 * wd + q, cl)] = make_uint2(t[0][q], t[1][q]);
                else vg[legacy4_slot(4 * wd + q, cl)] = t[0][q];
            }
            if (a.incoh) {
                // |16 v|^2 of four inputs per product (bytes 16 re, 16 im)
#pragma unroll
                for (int s = 0; s < kS; s++) {
                    const int re = (int)(w[s] & 0xF0F0F0F0u), im = (int)((w[s] << 4) & 0xF0F0F0F0u);
                    power[s] = __dp4a(im, im, __dp4a(re, re, power[s]));
                }
            }
        }
        if (a.incoh && blockIdx.z == 0) {
#pragma unroll
            for (int s = 0; s < kS; s++) {
                for (int o = 4; o < 32; o <<= 1) power[s] += __shfl_xor_sync(0xffffffffu, power[s], o);
                if (lane < 4 && s < ns) a.incoh[(long long)(sg + s) * a.nchan + c] = (float)(power[s] >> 8);
            }
        }
    }
    __syncthreads();

    const int c = c0 + lane, part = warp % kParts;
    const bool live = c < a.nchan;
    const Word *vg = vt + (size_t)(warp / kParts) * ni * kL4C;
    for (int p = blockIdx.z; p < a.npointing; p += gridDim.z) {
        float2 acc[kS / 2][8];
#pragma unroll
        for (int k = 0; k < kS / 2; k++)
#pragma unroll
            for (int q = 0; q < 8; q++) acc[k][q] = make_float2(0.f, 0.f);
        const float4 *Wp = a.W + ((long long)p * a.nant * a.nchan + (live ? c : 0)) * 2;
        const long long wstep = (long long)a.nchan * 2;
        float4 na = make_float4(0.f, 0.f, 0.f, 0.f), nb = na;
        if (part < a.nant) {
            na = __ldg(Wp + part * wstep);
            nb = __ldg(Wp + part * wstep + 1);
        }
        for (int ant = part; ant < a.nant; ant += kParts) {
            LegacyW w;
            w.set(na, nb);
            if (ant + kParts < a.nant) {
                na = __ldg(Wp + (ant + kParts) * wstep);
                nb = __ldg(Wp + (ant + kParts) * wstep + 1);
            }
            const uint32_t iqp = pq[ant];
            const Word bq = vg[legacy4_slot(iqp & 0xFFFFu, lane)], bp = vg[legacy4_slot(iqp >> 16, lane)];
#pragma unroll
            for (int h = 0; h < kS / 4; h++) {
                uint32_t wq, wp;
                if constexpr (kS == 8) {
                    wq = h ? bq.y : bq.x;
                    wp = h ? bp.y : bp.x;
                } else {
                    wq = bq;
                    wp = bp;
                }
                float2 qr[2], qi[2], pr[2], pi[2];
                legacy4_widen(((wq >> 4) & 0x0F0F0F0Fu) ^ 0x08080808u, qr[0], qr[1]);
                legacy4_widen((wq & 0x0F0F0F0Fu) ^ 0x08080808u, qi[0], qi[1]);
                legacy4_widen(((wp >> 4) & 0x0F0F0F0Fu) ^ 0x08080808u, pr[0], pr[1]);
                legacy4_widen((wp & 0x0F0F0F0Fu) ^ 0x08080808u, pi[0], pi[1]);
#pragma unroll
                for (int k = 0; k < 2; k++) legacy_pair(acc[2 * h + k], w, qr[k], qi[k], pr[k], pi[k]);
            }
        }
#pragma unroll
        for (int h = 0; h < kS / 4; h++) {
            if (h > 0 || p > 0) __syncthreads(); // the previous sums have been read
#pragma unroll
            for (int k = 0; k < 2; k++)
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    red[((warp * 4 + 2 * k) * 8 + q) * kL4C + lane] = acc[2 * h + k][q].x;
                    red[((warp * 4 + 2 * k + 1) * 8 + q) * kL4C + lane] = acc[2 * h + k][q].y;
                }
            __syncthreads();
            // (group, sample of the four) pairs over the warps; with one group
            // the warps 4 h .. 4 h + 3 take them
            for (int e = kG == 1 ? warp - 4 * h : warp; e >= 0 && e < 4 * kG; e += kLWarps) {
                const int g = e / 4, sl = e % 4, s = s0 + g * kS + 4 * h + sl;
                if (!live || s >= a.nsamples) continue;
                float sum[8];
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    sum[q] = 0.f;
#pragma unroll
                    for (int w = 0; w < kParts; w++) sum[q] += red[(((g * kParts + w) * 4 + sl) * 8 + q) * kL4C + lane];
                }
                legacy_store(a, p, s, c, sum);
            }
        }
    }
}

// Complex FP64 voltages. A block covers 8 channels x kG groups of kS samples:
// each row is read from memory once for all pointings and kept as FP32, pairs
// of samples together; thread = (channel lane % 8, tiles part, part + 32 / kG,
// ... of its group), and the partial sums of a (sample, channel) meet through
// shuffles, then shared memory. The voltages are narrowed in integer operations:
// the conversion instruction issues on the FP64 pipe, 2 per clock per SM here,
// which takes longer than reading them.
constexpr int kLdC = 8;

__device__ __forceinline__ float2 shfl2(float2 x, int mask)
{
    return make_float2(__shfl_xor_sync(0xffffffffu, x.x, mask), __shfl_xor_sync(0xffffffffu, x.y, mask));
}

template <int kS, int kG> static size_t legacyd_smem(int nant)
{
    return sizeof(float4) * (size_t)(kS / 2) * kG * kLdC * (2 * nant + 1) + sizeof(float) * kLWarps * kS * 8 * kLdC +
           (size_t)nant * 4;
}

template <int kS, int kG> __global__ void __launch_bounds__(256, 3) legacyd_kernel(const LegacyArgs a)
{
    constexpr int kGroupWarps = kLWarps / kG, kParts = 4 * kGroupWarps, kPairs = kS / 2, kV = 8 * kPairs;
    extern __shared__ __align__(16) unsigned char lsm[];
    const int ni = 2 * a.nant, stride = ni + 1;   // odd: the rows of 8 channels fall on different banks
    float4 *vt = reinterpret_cast<float4 *>(lsm); // [sample pair][channel][input]: re, re, im, im
    float *red = reinterpret_cast<float *>(vt + (size_t)kPairs * kG * kLdC * stride); // partial sums
    uint32_t *pq = reinterpret_cast<uint32_t *>(red + kLWarps * kS * 8 * kLdC);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int c0 = blockIdx.x * kLdC, s0 = blockIdx.y * kS * kG + (kS * kG < kLS ? a.s_first : 0);

    legacy_inputs(a, pq);
    // warp w stages channel w's rows, two sample pairs in flight
    if (c0 + warp < a.nchan) {
        const double2 *v = static_cast<const double2 *>(a.v) + ((long long)s0 * a.nchan + c0 + warp) * ni;
        const long long sstep = (long long)a.nchan * ni;
        const int ns = min(kS * kG, a.nsamples - s0);
        constexpr int kRows = kPairs * kG;
        if (((ni + 31) & ~31) * 8 <= ni * 9) {
            constexpr int kFly = kRows >= 2 ? 2 : 1;
            for (int k0 = 0; k0 < kRows; k0 += kFly)
#pragma unroll 2
                for (int i = lane; i < ni; i += 32) {
                    double2 d[kFly][2];
#pragma unroll
                    for (int k = 0; k < kFly; k++)
#pragma unroll
                        for (int q = 0; q < 2; q++) {
                            const int sl = 2 * (k0 + k) + q;
                            d[k][q] = sl < ns ? __ldcs(v + sl * sstep + i) : make_double2(0.0, 0.0);
                        }
#pragma unroll
                    for (int k = 0; k < kFly; k++)
                        vt[((k0 + k) * kLdC + warp) * stride + i] = narrow4(d[k][0].x, d[k][1].x, d[k][0].y, d[k][1].y);
                }
        } else {
            // more than an eighth of the lanes would idle at the rows' ends: the rows as one run over
            // the lanes (20 tiles, 3,000 samples, one beam: 95 -> 60 us; whole rows of 128 tiles the
            // other way, 283 -> 311 us for the work around it)
            constexpr int kFly = 4;
            const int dk = 32 / ni, di = 32 - dk * ni;
            int k = lane / ni, i = lane - k * ni;
            while (k < kRows) {
                double2 d[kFly][2];
                int at[kFly];
#pragma unroll
                for (int f = 0; f < kFly; f++) {
                    at[f] = k < kRows ? (k * kLdC + warp) * stride + i : -1;
#pragma unroll
                    for (int q = 0; q < 2; q++)
                        d[f][q] = 2 * k + q < ns ? __ldcs(v + (2 * k + q) * sstep + i) : make_double2(0.0, 0.0);
                    i += di;
                    const int next = i >= ni;
                    i -= next ? ni : 0;
                    k += dk + next;
                }
#pragma unroll
                for (int f = 0; f < kFly; f++)
                    if (at[f] >= 0) vt[at[f]] = narrow4(d[f][0].x, d[f][1].x, d[f][0].y, d[f][1].y);
            }
        }
    }
    __syncthreads();

    const int cl = lane & (kLdC - 1), c = c0 + cl, group = warp / kGroupWarps;
    const int part = 4 * (warp % kGroupWarps) + (lane >> 3);
    const bool live = c < a.nchan;
    const float4 *vc = vt + (group * kPairs * kLdC + cl) * stride;
    for (int p = blockIdx.z; p < a.npointing; p += gridDim.z) {
        float2 acc[kPairs][8];
#pragma unroll
        for (int k = 0; k < kPairs; k++)
#pragma unroll
            for (int q = 0; q < 8; q++) acc[k][q] = make_float2(0.f, 0.f);
        const float4 *Wp = a.W + ((long long)p * a.nant * a.nchan + (live ? c : 0)) * 2;
        const long long wstep = (long long)a.nchan * 2;
        float4 na = make_float4(0.f, 0.f, 0.f, 0.f), nb = na;
        if (part < a.nant) {
            na = __ldg(Wp + part * wstep);
            nb = __ldg(Wp + part * wstep + 1);
        }
        for (int ant = part; live && ant < a.nant; ant += kParts) {
            LegacyW w;
            w.set(na, nb);
            if (ant + kParts < a.nant) {
                na = __ldg(Wp + (ant + kParts) * wstep);
                nb = __ldg(Wp + (ant + kParts) * wstep + 1);
            }
            const uint32_t iqp = pq[ant], iq = iqp & 0xFFFFu, ip = iqp >> 16;
#pragma unroll
            for (int k = 0; k < kPairs; k++) {
                const float4 q = vc[k * kLdC * stride + iq], r = vc[k * kLdC * stride + ip];
                legacy_pair(acc[k], w, make_float2(q.x, q.y), make_float2(q.z, q.w), make_float2(r.x, r.y),
                            make_float2(r.z, r.w));
            }
        }
        // the four lanes of a channel exchange halves twice: each ends with a
        // quarter `sel` of the kV pairs of sums, added over the four
        const bool up = lane & 16, right = lane & 8;
        float2 half[kV / 2], quarter[kV / 4];
#pragma unroll
        for (int j = 0; j < kV / 2; j++) {
            const float2 lo = acc[j / 8][j % 8], hi = acc[(j + kV / 2) / 8][(j + kV / 2) % 8];
            half[j] = padd(up ? hi : lo, shfl2(up ? lo : hi, 16));
        }
#pragma unroll
        for (int j = 0; j < kV / 4; j++)
            quarter[j] = padd(right ? half[j + kV / 4] : half[j], shfl2(right ? half[j] : half[j + kV / 4], 8));
        if (p > 0) __syncthreads(); // the previous pointing's partial sums have been read
#pragma unroll
        for (int j = 0; j < kV / 4; j++) {
            const int sel = (up ? 2 : 0) + (right ? 1 : 0);
            red[(((warp * 2 + 0) * (kV / 4) + j) * 4 + sel) * kLdC + cl] = quarter[j].x;
            red[(((warp * 2 + 1) * (kV / 4) + j) * 4 + sel) * kLdC + cl] = quarter[j].y;
        }
        __syncthreads();
        // thread = (sample, channel)
        const int sl = tid / kLdC, s = s0 + sl;
        if (sl < kS * kG && live && s < a.nsamples) {
            float sum[8];
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const int v = (sl % kS / 2) * 8 + q; // the pair of sums; the sample is its half sl % 2
                sum[q] = 0.f;
#pragma unroll
                for (int w = 0; w < kGroupWarps; w++)
                    sum[q] += red[((((sl / kS * kGroupWarps + w) * 2 + sl % 2) * (kV / 4) + v % (kV / 4)) * 4 + v / (kV / 4)) * kLdC + cl];
            }
            legacy_store(a, p, s, c, sum);
        }
    }
}

// The tile: as many sample groups as leave two (4-bit) or three (FP64) blocks'
// shared memory per SM and still give every SM a block (4-bit, pointings counted:
// they can go to different blocks) or two (FP64): groups spend less on the partial
// sums, but a short run needs its samples spread (4-bit, 8 tiles, 200 samples, one
// beam: 10.9 us in 16-sample tiles, 8.8 in 8; 3,000 samples: 21.2 and 24.2; FP64,
// 8 tiles, one beam, 3,000 samples: 31 us with eight groups, 70 with one). The row
// kernel takes 8.8 and 35.5 us for the 4-bit runs, 40 us for the FP64 one. Where
// one group of the larger kS leaves room for one block only, the smaller kS (256
// tiles of 4+4-bit voltages, 4,000 samples: 224 us, row kernel 840 us). Arrays past
// that (more than 768 tiles of 4+4-bit or 877 of FP64 voltages) take the row kernel.
struct LegacyTile {
    void (*kern)(LegacyArgs);
    size_t smem;
    int channels, samples;
};

static LegacyTile legacy_tile(const LegacyArgs &a, bool int4, int nsm)
{
    const int nant = a.nant;
    const LegacyTile t4[] = {{legacy4_kernel<8, 2>, legacy4_smem<8, 2>(nant), kL4C, 16},
                             {legacy4_kernel<8, 1>, legacy4_smem<8, 1>(nant), kL4C, 8},
                             {legacy4_kernel<4, 1>, legacy4_smem<4, 1>(nant), kL4C, 4}};
    const LegacyTile td[] = {{legacyd_kernel<4, 8>, legacyd_smem<4, 8>(nant), kLdC, 32},
                             {legacyd_kernel<4, 4>, legacyd_smem<4, 4>(nant), kLdC, 16},
                             {legacyd_kernel<4, 2>, legacyd_smem<4, 2>(nant), kLdC, 8},
                             {legacyd_kernel<4, 1>, legacyd_smem<4, 1>(nant), kLdC, 4},
                             {legacyd_kernel<2, 1>, legacyd_smem<2, 1>(nant), kLdC, 2}};
    const LegacyTile *t = int4 ? t4 : td;
    const int n = int4 ? 3 : 5;
    for (int k = 0; k < n - 1; k++) {
        const long long blocks = (long long)((a.nchan + t[k].channels - 1) / t[k].channels) *
                                 ((a.nsamples + t[k].samples - 1) / t[k].samples);
        const bool enough = k == n - 2 || (int4 ? blocks * a.npointing >= nsm : blocks >= 2 * nsm);
        if (enough && t[k].smem <= (size_t)(int4 || k == n - 2 ? 113 : 75) * 1024) return t[k];
    }
    return t[n - 1];
}

// ---------------------------------------------------------------------------
// Arrays too large for the tiles above. A block covers 16 channels x 4 samples = 64 voltage rows, four threads per
// row splitting the tiles (tile = part, part + 4, ...) and combining their
// sums with two shuffles; the 4+4-bit rows are staged in shared memory with a
// 4-byte pad (33 KB for 256 tiles, so several blocks share an SM).
// ---------------------------------------------------------------------------

constexpr int kLC = 16;          // channels per block
constexpr int kLParts = 4;       // threads per row

template <bool kInt4>
__global__ void __launch_bounds__(256) legacy_beam_kernel(const LegacyArgs a)
{
    extern __shared__ __align__(16) unsigned char lsm[];
    const int ni = 2 * a.nant;
    const int tid = threadIdx.x;
    const int r = tid / kLParts, part = tid % kLParts;
    const int c0 = blockIdx.x * kLC, s0 = blockIdx.y * kLS;
    const int c = c0 + r % kLC, s = s0 + r / kLC;
    const bool live = c < a.nchan && s < a.nsamples;
    const int wpr = ni / 4 + 1;

    // Stage the 4+4-bit rows (s, c) of this block. Complex FP64 voltages are
    // read straight from global memory.
    if (kInt4) {
        // 4-byte asynchronous copies, all in flight before one wait (rows
        // outside the block's samples or channels are zero-filled)
        uint32_t *rows = reinterpret_cast<uint32_t *>(lsm);
        const int nw = ni / 4;
        const uint32_t *v32 = static_cast<const uint32_t *>(a.v);
        for (int idx = tid; idx < kLS * kLC * nw; idx += blockDim.x) {
            const int rr = idx / nw, wdx = idx % nw;
            const int rs = s0 + rr / kLC, rc = c0 + rr % kLC;
            const bool in = rs < a.nsamples && rc < a.nchan;
            const uint32_t *src = in ? v32 + ((long long)rs * a.nchan + rc) * (ni / 4) + wdx : v32;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(&rows[rr * wpr + wdx])),
                         "l"(src), "r"(in ? 4u : 0u)
                         : "memory");
        }
        asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    }
    // the tiles' (Q, P) input pairs, checked against the row once per block
    uint32_t *pq = reinterpret_cast<uint32_t *>(lsm + (kInt4 ? (size_t)kLS * kLC * wpr * 4 : 0));
    for (int ant = tid; ant < a.nant; ant += blockDim.x) {
        uint32_t iq = __ldg(a.polQ + ant), ip = __ldg(a.polP + ant);
        if (iq >= (uint32_t)ni || ip >= (uint32_t)ni) {
            if (blockIdx.x == 0 && blockIdx.y == 0) atomicOr(a.status, kErrBadInput);
            iq = ip = 0;
        }
        pq[ant] = iq | (ip << 16);
    }
    __syncthreads();
    const uint8_t *row8 = lsm + 4 * (r * wpr);

    for (int p = 0; p < a.npointing; p++) {
        float acc[8];
#pragma unroll
        for (int q = 0; q < 8; q++) acc[q] = 0.f;
        const float4 *Wp = a.W + ((long long)p * a.nant * a.nchan + (live ? c : 0)) * 2;
        if (live) {
#pragma unroll 4
            for (int ant = part; ant < a.nant; ant += kLParts) {
                const uint32_t iqp = pq[ant], iq = iqp & 0xFFFFu, ip = iqp >> 16;
                float2 vq, vp;
                if (kInt4) {
                    const uint32_t bq = row8[iq], bp = row8[ip];
                    vq = make_float2((float)nib(bq >> 4), (float)nib(bq));
                    vp = make_float2((float)nib(bp >> 4), (float)nib(bp));
                } else {
                    const double2 *row = static_cast<const double2 *>(a.v) + ((long long)s * a.nchan + c) * ni;
                    const double2 dq = __ldg(row + iq), dp = __ldg(row + ip);
                    vq = make_float2((float)dq.x, (float)dq.y);
                    vp = make_float2((float)dp.x, (float)dp.y);
                }
                const float4 wa = __ldg(Wp + (long long)ant * a.nchan * 2);
                const float4 wb = __ldg(Wp + (long long)ant * a.nchan * 2 + 1);
                const float exr = wa.x * vq.x - wa.y * vq.y + wa.z * vp.x - wa.w * vp.y;
                const float exi = wa.x * vq.y + wa.y * vq.x + wa.z * vp.y + wa.w * vp.x;
                const float eyr = wb.x * vq.x - wb.y * vq.y + wb.z * vp.x - wb.w * vp.y;
                const float eyi = wb.x * vq.y + wb.y * vq.x + wb.z * vp.y + wb.w * vp.x;
                acc[0] += exr;
                acc[1] += exi;
                acc[2] += eyr;
                acc[3] += eyi;
                acc[4] = fmaf(exr, exr, fmaf(exi, exi, acc[4]));
                acc[5] = fmaf(eyr, eyr, fmaf(eyi, eyi, acc[5]));
                acc[6] = fmaf(exr, eyr, fmaf(exi, eyi, acc[6]));
                acc[7] = fmaf(exi, eyr, fmaf(-exr, eyi, acc[7]));
            }
        }
        // the row's four partial sums (lanes 4k .. 4k+3 of a warp)
#pragma unroll
        for (int q = 0; q < 8; q++) {
            acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], 1);
            acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], 2);
        }
        if (!live || part != 0) continue;
        const float bnXX = acc[0] * acc[0] + acc[1] * acc[1] - acc[4];
        const float bnYY = acc[2] * acc[2] + acc[3] * acc[3] - acc[5];
        const float bxr = acc[0] * acc[2] + acc[1] * acc[3] - acc[6];
        const float bxi = acc[1] * acc[2] - acc[0] * acc[3] - acc[7];
        float *S = a.S + (((long long)p * a.nsamples + s) * a.nstokes) * a.nchan + c;
        S[0] = a.invw * (bnXX + bnYY);
        if (a.nstokes == 4) {
            S[a.nchan] = a.invw * (bnXX - bnYY);
            S[2 * a.nchan] = 2.0f * a.invw * bxr;
            S[3 * a.nchan] = -2.0f * a.invw * bxi;
        }
        if (a.e) a.e[((long long)p * a.nsamples + s) * a.nchan + c] = make_float4(acc[0], acc[1], acc[2], acc[3]);
    }
    if (kInt4 && a.incoh && live && part == 0) {
        const uint32_t *row = reinterpret_cast<const uint32_t *>(lsm) + r * wpr;
        int accp = 0;
        for (int wdx = 0; wdx < ni / 4; wdx++) accp += power4(row[wdx]);
        a.incoh[(long long)s * a.nchan + c] = (float)accp;
    }
}

int launch_legacy_beam(const LegacyArgs &a, cudaStream_t st)
{
    if (a.nsamples <= 0) return VGB_SUCCESS;
    const int ni = 2 * a.nant;
    const bool int4 = a.datatype == VGB_INT4;
    if (int4 && (ni % 4) != 0) return set_error(VGB_ERR_INVALID, "legacy beamformer: 2*nant must be a multiple of 4");
    if (ni > 65535) return set_error(VGB_ERR_INVALID, "legacy beamformer: at most 65535 inputs");
    const size_t smem = (int4 ? (size_t)kLS * kLC * (ni / 4 + 1) * 4 : 0) + (size_t)a.nant * 4;
    if (smem > 227 * 1024)
        return set_error(VGB_ERR_INVALID, "legacy beamformer: %d inputs do not fit the shared-memory tile", ni);
    if ((a.nsamples + kLS - 1) / kLS > 65535)
        return set_error(VGB_ERR_INVALID, "legacy beamformer: at most %d samples per call", 65535 * kLS);
    const int nsm = sm_count();
    const LegacyTile t = legacy_tile(a, int4, nsm);
    if (t.smem <= 227 * 1024) {
        const int rc = check_cuda(cudaFuncSetAttribute(t.kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)t.smem),
                                  "cudaFuncSetAttribute(legacy tile)");
        if (rc) return rc;
        const unsigned gx = (a.nchan + t.channels - 1) / t.channels, gy = (a.nsamples + t.samples - 1) / t.samples;
        // the pointings over blocks too where the rest is short of two (4-bit) or one (FP64) per SM: each
        // share reads the voltages again (4-bit, 20 tiles, 200 samples, 12 beams: 74 -> 21 us)
        const long long shares = (int4 ? 2 : 1) * nsm / ((long long)gx * gy);
        const unsigned gz = (unsigned)std::min<long long>(a.npointing, std::max<long long>(1, shares));
        // grid y counts 65,535 tiles of samples; those of two (FP64, 208 to 877 tiles) can be twice as many
        // and come in two launches. (A first sample in the other kernels too, or both directions on grid x
        // with a division a block: 4-bit 252 -> 256 us.)
        LegacyArgs part = a;
        for (unsigned y = 0; y < gy; y += 65535) {
            part.s_first = (int)y * t.samples;
            t.kern<<<dim3(gx, std::min(gy - y, 65535u), gz), 256, t.smem, st>>>(part);
        }
        return check_launch("legacy beam kernel");
    }
    dim3 grid((a.nchan + kLC - 1) / kLC, (a.nsamples + kLS - 1) / kLS);
    if (int4) {
        int rc = check_cuda(cudaFuncSetAttribute(legacy_beam_kernel<true>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                            "cudaFuncSetAttribute(legacy)");
        if (rc) return rc;
        legacy_beam_kernel<true><<<grid, 256, smem, st>>>(a);
    } else {
        int rc = check_cuda(cudaFuncSetAttribute(legacy_beam_kernel<false>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                            "cudaFuncSetAttribute(legacy)");
        if (rc) return rc;
        legacy_beam_kernel<false><<<grid, 256, smem, st>>>(a);
    }
    return check_launch("legacy_beam_kernel");
}

} // namespace vgb
