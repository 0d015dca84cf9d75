// Primary-beam matrices B [pointing][tile][2][2] (vmCalcB,
// primary_beam.c:79-191) on the device, FP64, evaluated once per distinct
// delay set (tiles sharing a dipole configuration share B, as vmCalcB's
// per-configuration cache) and copied to the other tiles.
//
// The reference evaluates the MWA FEE model (mwa_hyperbeam's calc_jones, a
// Rust crate reading an HDF5 table of spherical-wave coefficients) once per
// distinct dead-dipole configuration and pointing, then multiplies the
// parallactic-angle rotation on the right. The FEE model is not available to
// this build; the model evaluated here is an analytic MWA tile:
//
//   * 16 dipoles on a 4 x 4 grid of 1.1 m pitch (row 0 north, column 0 west),
//     each delayed by d_i x 435 ps by the tile beamformer (d_i = 0..31, 32 =
//     dead dipole, amplitude 0: create_delays_amps_from_metafits,
//     primary_beam.c:260-284);
//   * array factor AF = (1/16) sum_i a_i exp(2 pi i f (tau_i - d_i 435 ps)),
//     tau_i = (x_i sin(za) sin(az) + y_i sin(za) cos(az)) / c;
//   * a ground plane 0.278 m below the dipoles,
//     G = sin(2 pi f h cos(za) / c) / sin(2 pi f h / c);
//   * short-dipole projections onto the sky basis (theta, phi) for the E-W (X)
//     and N-S (Y) dipoles: [[cos za sin az, cos za cos az], [cos az, -sin az]].
//
//   J = AF G [[cos za sin az, cos za cos az], [cos az, -sin az]]   (zenith-normalised)
//
// Parallactic angle (primary_beam.c:436-456, the spherical-triangle identity
// of the reference's doc/Definitions.md): horizon (az, el) -> (ha, dec) at
// latitude lat, chi = atan2(cos lat sin ha, sin lat cos dec - cos lat sin dec
// cos ha), P = [[-cos chi, -sin chi], [sin chi, -cos chi]], B = J P.
#include "beam_model.cuh"
#include "vgb_launch.cuh"

namespace vgb {

// Distinct delay sets, as vmCalcB evaluates the beam once per distinct dipole
// configuration (primary_beam.c:119-160).
__device__ __forceinline__ bool same_delays(const uint32_t *delays, int t, int u)
{
    const uint4 *dt = reinterpret_cast<const uint4 *>(delays + 16 * (long long)t);
    const uint4 *du = reinterpret_cast<const uint4 *>(delays + 16 * (long long)u);
    for (int i = 0; i < 4; i++) {
        const uint4 a = dt[i], b = du[i];
        if (a.x != b.x || a.y != b.y || a.z != b.z || a.w != b.w) return false;
    }
    return true;
}

// B = J P (complex x real, as mult2x2d_CxR), or J without the rotation.
__device__ __forceinline__ void bm_store(double2 *o, const double2 (&J)[4], const double *P)
{
    if (!P) {
        for (int e = 0; e < 4; e++) o[e] = J[e];
        return;
    }
    for (int r = 0; r < 2; r++)
        for (int c = 0; c < 2; c++) {
            const double2 a = J[2 * r], b = J[2 * r + 1];
            // explicit contraction: every caller gets the same bits
            o[2 * r + c] = make_double2(fma(b.x, P[2 + c], __dmul_rn(a.x, P[c])), fma(b.y, P[2 + c], __dmul_rn(a.y, P[c])));
        }
}

// bm_jones by 16 lanes (l = 0 .. 15 of `mask`), one dipole each: the same
// operations, the dipoles' terms added in dipole order. Every lane returns J.
__device__ __forceinline__ void bm_jones16(int l, unsigned mask, double az, double za, double f, const uint32_t *d,
                                           double2 (&J)[4])
{
    double s, c;
    sincos(l == 0 ? az : za, &s, &c);
    const double saz = __shfl_sync(mask, s, 0, 16), caz = __shfl_sync(mask, c, 0, 16);
    const double sza = __shfl_sync(mask, s, 1, 16), cza = __shfl_sync(mask, c, 1, 16);
    const double k = 2.0 * kBmPi * f;
    const uint32_t di = d[l];
    bm_dipole(l, di, sza, saz, caz, k, s, c);
    double re = 0.0, im = 0.0;
    int live = 0;
    for (int i = 0; i < 16; i++) {
        const double ci = __shfl_sync(mask, c, i, 16), si = __shfl_sync(mask, s, i, 16);
        if (__shfl_sync(mask, di, i, 16) == 32u) continue;
        live++;
        re += ci;
        im += si;
    }
    const double gl = sin(l == 0 ? k * kBmHeight * cza / kBmC : k * kBmHeight / kBmC);
    bm_project(live, re, im, __shfl_sync(mask, gl, 0, 16) / __shfl_sync(mask, gl, 1, 16), saz, caz, cza, J);
}

// Everything in one launch: block b takes (frequency, pointing) pairs b *
// per_block ... and writes their B for all tiles. A chain of FP64
// transcendentals (about 2 us each at this GPU's FP64 latency) bounds a small
// call, so a delay set's 16 dipoles take 16 lanes, the parallactic rotations
// one lane each of the last warp beside them, and the tiles' sets are found in
// shared memory by every block instead of a kernel of its own: 8 to 152
// pointings x 128 tiles in 3 sets, 78-88 us in three launches -> 19 us. The
// lanes repeat the per-direction work, 6.1 ns per (pair, set) against 4.3 ns
// with one thread each, so past 304 pairs (24,576 pairs: 453 against 317 us) the
// three launches take over.
constexpr int kBmThreads = 256, kBmPairs = 2, kBmMaxTiles = 2048, kBmMaxPairs = 304;

__global__ void __launch_bounds__(kBmThreads) beam_kernel_fused(const PbArgs a, int per_block)
{
    extern __shared__ int bm_smem[];
    int *rep = bm_smem, *list = rep + a.ntile;
    uint32_t *hash = reinterpret_cast<uint32_t *>(list + a.ntile);
    __shared__ double P[kBmPairs][4];
    __shared__ int warp_count[kBmThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long pairs = (long long)a.nfreq * a.npointing;
    const long long p0 = (long long)blockIdx.x * per_block;
    const int np = (int)min((long long)per_block, pairs - p0);

    for (int t = tid; t < a.ntile; t += kBmThreads) {
        uint32_t h = 2166136261u;
        for (int i = 0; i < 16; i++) h = (h ^ a.delays[16 * (long long)t + i]) * 16777619u;
        hash[t] = h;
    }
    __syncthreads();
    // rep[t]: the first tile with tile t's delays; list: those first tiles
    int count = 0;
    for (int t0 = 0; t0 < a.ntile; t0 += kBmThreads) {
        const int t = t0 + tid;
        int r = t;
        if (t < a.ntile) {
            for (int u = 0; u < t; u++)
                if (hash[u] == hash[t] && same_delays(a.delays, t, u)) {
                    r = u;
                    break;
                }
            rep[t] = r;
        }
        const bool first = t < a.ntile && r == t;
        const unsigned b = __ballot_sync(0xffffffffu, first);
        if (lane == 0) warp_count[warp] = __popc(b);
        __syncthreads();
        int at = count;
        for (int w = 0; w < kBmThreads / 32; w++) {
            if (w < warp) at += warp_count[w];
            count += warp_count[w];
        }
        if (first) list[at + __popc(b & ((1u << lane) - 1))] = t;
        __syncthreads();
    }

    if (a.pa && warp == kBmThreads / 32 - 1) {
        if (lane < np) {
            double p[4];
            const int pt = (int)((p0 + lane) % a.npointing);
            bm_pa(a.lat, a.az[pt], a.za[pt], p);
            for (int e = 0; e < 4; e++) P[lane][e] = p[e];
        }
    }
    // items: (pair, set), 16 lanes each
    const int groups = 2 * (kBmThreads / 32 - (a.pa ? 1 : 0)), group = tid >> 4, l = tid & 15;
    const unsigned mask = 0xFFFFu << (lane & 16);
    const int items = np * count;
    double2 *out = a.B + 4 * p0 * a.ntile;
    for (int e0 = 0; e0 < items; e0 += groups) {
        const int e = e0 + group;
        const bool mine = group < groups && e < items;
        double2 J[4];
        if (mine) {
            const int pt = (int)((p0 + e / count) % a.npointing), fi = (int)((p0 + e / count) / a.npointing);
            bm_jones16(l, mask, a.az[pt], a.za[pt], a.freq[fi], a.delays + 16 * (long long)list[e % count], J);
        }
        if (e0 == 0) __syncthreads(); // the rotations
        if (mine && l == 0)
            bm_store(out + 4 * ((long long)(e / count) * a.ntile + list[e % count]), J, a.pa ? P[e / count] : nullptr);
    }
    __syncthreads();
    // every other tile copies its set's matrix, 16 bytes per thread
    for (int i = tid; i < np * a.ntile * 4; i += kBmThreads) {
        const int t = (i / 4) % a.ntile, r = rep[t];
        if (r != t) out[i] = out[i + 4 * (r - t)];
    }
}

// Callers with scratch of their own (the pipeline's tracking, 24 channels x one
// pointing beside a second's other work), more pairs, and more tiles than a
// block's shared memory lists: rep[t] = the first tile with
// tile t's 16 delays, list[k] = the k-th such first tile, count = their number.
// One block; O(ntile^2) comparisons of 16 words, early exit on the first match.
__global__ void beam_configs_kernel(const uint32_t *delays, int ntile, int *rep, int *list, int *count)
{
    __shared__ int s_first[1024];
    __shared__ int s_base;
    if (threadIdx.x == 0) s_base = 0;
    __syncthreads();
    for (int t0 = 0; t0 < ntile; t0 += blockDim.x) {
        const int t = t0 + threadIdx.x;
        int r = t;
        if (t < ntile) {
            for (int u = 0; u < t; u++)
                if (same_delays(delays, t, u)) {
                    r = u;
                    break;
                }
            rep[t] = r;
        }
        s_first[threadIdx.x] = t < ntile && r == t;
        __syncthreads();
        if (threadIdx.x == 0) { // compact this chunk's first tiles in tile order
            int k = s_base;
            for (int i = 0; i < (int)blockDim.x && t0 + i < ntile; i++)
                if (s_first[i]) list[k++] = t0 + i;
            s_base = k;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) *count = s_base;
}

// B for (frequency, pointing, the k-th distinct delay set), written at that
// set's first tile. Threads with k >= count leave at once.
__global__ void beam_model_kernel(const PbArgs a, const int *list, const int *count)
{
    const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long per_k = (long long)a.nfreq * a.npointing;
    const int k = (int)(idx / per_k);
    if (k >= *count || k >= a.ntile) return;
    const int p = (int)(idx % a.npointing);
    const int fi = (int)((idx / a.npointing) % a.nfreq);
    const int t = list[k];
    double2 J[4];
    bm_jones(a.az[p], a.za[p], a.freq[fi], a.delays + 16 * (long long)t, J);
    double P[4];
    if (a.pa) bm_pa(a.lat, a.az[p], a.za[p], P);
    bm_store(a.B + 4 * (((long long)fi * a.npointing + p) * a.ntile + t), J, a.pa ? P : nullptr);
}

// Every other tile copies its set's matrix (32 bytes per thread, two uint4).
__global__ void beam_expand_kernel(const PbArgs a, const int *rep)
{
    const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long n = (long long)a.nfreq * a.npointing * a.ntile;
    if (idx >= n) return;
    const int t = (int)(idx % a.ntile);
    const int r = rep[t];
    if (r == t) return;
    const uint4 *src = reinterpret_cast<const uint4 *>(a.B + 4 * (idx - t + r));
    uint4 *dst = reinterpret_cast<uint4 *>(a.B + 4 * idx);
    dst[0] = src[0];
    dst[1] = src[1];
    dst[2] = src[2];
    dst[3] = src[3];
}

int launch_beam_model(const PbArgs &a, cudaStream_t st, int *given)
{
    const long long n = (long long)a.nfreq * a.npointing * a.ntile;
    if (n <= 0) return VGB_SUCCESS;
    const long long pairs = (long long)a.nfreq * a.npointing;
    if (!given && a.ntile <= kBmMaxTiles && pairs <= kBmMaxPairs) {
        const int per_block = pairs <= 152 ? 1 : 2; // one per SM, then two
        beam_kernel_fused<<<(unsigned)((pairs + per_block - 1) / per_block), kBmThreads, 3 * sizeof(int) * a.ntile, st>>>(
            a, per_block);
        return check_launch("beam_kernel_fused");
    }
    int *scratch = given; // rep [ntile], list [ntile], count
    int rc = VGB_SUCCESS;
    if (!given)
        rc = check_cuda(cudaMallocAsync(reinterpret_cast<void **>(&scratch), (2 * (size_t)a.ntile + 1) * sizeof(int),
                                        st),
                        "cudaMallocAsync(beam configurations)");
    if (rc) return rc;
    int *rep = scratch, *list = scratch + a.ntile, *count = scratch + 2 * a.ntile;
    beam_configs_kernel<<<1, 1024, 0, st>>>(a.delays, a.ntile, rep, list, count);
    rc = check_launch("beam_configs_kernel");
    if (!rc) {
        beam_model_kernel<<<(unsigned)((n + 127) / 128), 128, 0, st>>>(a, list, count);
        rc = check_launch("beam_model_kernel");
    }
    if (!rc) {
        beam_expand_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(a, rep);
        rc = check_launch("beam_expand_kernel");
    }
    if (given) return rc;
    const int rf = check_cuda(cudaFreeAsync(scratch, st), "cudaFreeAsync(beam configurations)");
    return rc ? rc : rf;
}

} // namespace vgb

using namespace vgb;

// primary_beam.c:355-414: index of a live/dead dipole pattern among the 138
// cached configurations (0 all live, 1-16 one dead, 17-136 two dead, 137 all
// dead), or -1 for more than two (but not all) dead.
extern "C" int vgb_hash_dipole_config(const double *amps)
{
    if (!amps) {
        set_error(VGB_ERR_INVALID, "hash_dipole_config: NULL amps");
        return -2;
    }
    int dead[16], ndead = 0;
    for (int i = 0; i < 16; i++)
        if (amps[i] == 0.0) dead[ndead++] = i;
    switch (ndead) {
    case 0: return 0;
    case 1: return dead[0] + 1;
    case 2: return 16 * dead[0] - ((dead[0] + 2) * (dead[0] + 1)) / 2 + dead[1] + 17;
    case 16: return 137;
    default: return -1;
    }
}

extern "C" int vgb_primary_beam(const double *az, const double *za, int npointing, const double *freq_hz, int nfreq,
                                const uint32_t *delays, int ntile, double latitude, int pa_correction, void *B,
                                void *stream)
{
    if (!az || !za || !freq_hz || !delays || !B) return set_error(VGB_ERR_INVALID, "primary_beam: NULL argument");
    if (npointing <= 0 || nfreq <= 0 || ntile <= 0) return set_error(VGB_ERR_INVALID, "primary_beam: empty shape");
    if ((reinterpret_cast<uintptr_t>(delays) | reinterpret_cast<uintptr_t>(B)) & 15)
        return set_error(VGB_ERR_INVALID, "primary_beam: delays and B must be 16-byte aligned");
    PbArgs a{az, za, npointing, freq_hz, nfreq, delays, ntile, latitude, pa_correction, static_cast<double2 *>(B)};
    return launch_beam_model(a, static_cast<cudaStream_t>(stream));
}
