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
#include <algorithm>

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

// What bm_jones computes once per direction and frequency: p holds bm_project's
// projections in its order.
struct BmDir {
    double saz, caz, sza, k, g, p[4];
};

// By two lanes (l = 0, 1) of `mask`'s pairs, a sine each; both return it.
__device__ __forceinline__ BmDir bm_dir2(int l, unsigned mask, double az, double za, double f)
{
    double s, c;
    sincos(l == 0 ? az : za, &s, &c);
    BmDir v;
    v.saz = __shfl_sync(mask, s, 0, 2), v.caz = __shfl_sync(mask, c, 0, 2);
    v.sza = __shfl_sync(mask, s, 1, 2);
    const double cza = __shfl_sync(mask, c, 1, 2);
    v.k = 2.0 * kBmPi * f;
    const double gl = sin(l == 0 ? v.k * kBmHeight * cza / kBmC : v.k * kBmHeight / kBmC);
    v.g = __shfl_sync(mask, gl, 0, 2) / __shfl_sync(mask, gl, 1, 2);
    v.p[0] = cza * v.saz, v.p[1] = cza * v.caz, v.p[2] = v.caz, v.p[3] = -v.saz;
    return v;
}

// bm_jones and bm_store by 16 lanes (l = 0 .. 15 of `mask`) with the same
// operations: a dipole's phase term each, the terms added in dipole order (real
// parts on even lanes, imaginary parts on odd ones), then lanes 0 .. 7 write one
// of the matrix's eight values each.
__device__ __forceinline__ void bm_write16(int l, unsigned mask, const BmDir &v, const uint32_t *d, const double *P,
                                           double2 *o)
{
    const uint32_t di = d[l];
    double s, c, sum = 0.0;
    bm_dipole(l, di, v.sza, v.saz, v.caz, v.k, s, c);
    const unsigned live = __ballot_sync(mask, di != 32u) >> (__ffs(mask) - 1);
    for (int i = 0; i < 16; i++) {
        const double ci = __shfl_sync(mask, c, i, 16), si = __shfl_sync(mask, s, i, 16);
        if (live >> i & 1u) sum += l & 1 ? si : ci;
    }
    if (l >= 8) return;
    const int r = l >> 2, col = l >> 1 & 1;
    const double q = sum / 16.0 * v.g;
    const double ja = live ? q * v.p[2 * r] : 0.0, jb = live ? q * v.p[2 * r + 1] : 0.0;
    reinterpret_cast<double *>(o)[l] = P ? fma(jb, P[2 + col], __dmul_rn(ja, P[col])) : col ? jb : ja;
}

// Everything in one launch: block (b, y) takes (frequency, pointing) pairs b *
// per_block ... and the distinct delay sets y, y + gridDim.y, ...; it writes B for
// the tiles of those sets. A chain of FP64 transcendentals (about 2 us each at this
// GPU's FP64 latency) bounds a small call, so a delay set's 16 dipoles take 16
// lanes, and the directions and the parallactic rotations a warp each while the
// others find the sets in shared memory, which every block does instead of a kernel
// of its own. With many sets the FP64 pipe bounds it (2 per clock per SM): what
// depends on the direction only is computed once per pair, no sum or product is
// formed by two lanes, and the sets go to as many blocks as there are SMs (how many
// sets there are is not known to the host, so blocks past them leave). With 3 / all
// tiles different, against the three launches (us):
//   8 pointings, 128 tiles    17 / 19    63 / 75     152, 128 tiles    17 / 51    68 / 77
//   1 pointing, 2,048 tiles   44 / 109  145 / 382    304, 256 tiles    19 / 159   76 / 217
// Measured up to 304 pairs; many more fill the GPU with a thread per (pair, set).
constexpr int kBmThreads = 256, kBmPairs = 2, kBmMaxTiles = 2048, kBmMaxPairs = 304;
constexpr int kBmFinders = kBmThreads - 64, kBmGroups = kBmThreads / 16;

__host__ __device__ constexpr int bm_hashes(int ntile) { return (ntile + 15) / 16 * 16; }

// The first tile with tile t's delays.
__device__ __forceinline__ int bm_first_equal(const uint32_t *hash, const uint32_t *delays, int t)
{
    const uint32_t h = hash[t];
    for (int u = 0; u < t; u += 16) {
        bool any = false;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const uint4 q = reinterpret_cast<const uint4 *>(hash + u)[j];
            any |= q.x == h || q.y == h || q.z == h || q.w == h;
        }
        if (any)
            for (int w = u; w < min(u + 16, t); w++)
                if (hash[w] == h && same_delays(delays, t, w)) return w;
    }
    return t;
}

__global__ void __launch_bounds__(kBmThreads) beam_kernel_fused(const PbArgs a, int per_block)
{
    extern __shared__ __align__(16) int bm_smem[];
    uint32_t *hash = reinterpret_cast<uint32_t *>(bm_smem);
    int *rep = bm_smem + bm_hashes(a.ntile), *list = rep + a.ntile, *rank = list + a.ntile;
    __shared__ double P[kBmPairs][4];
    __shared__ BmDir dir[kBmPairs];
    __shared__ int warp_count[kBmFinders / 32], nlist;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long pairs = (long long)a.nfreq * a.npointing;
    const long long p0 = (long long)blockIdx.x * per_block;
    const int np = (int)min((long long)per_block, pairs - p0);

    if (tid < kBmFinders) {
        for (int t = tid; t < a.ntile; t += kBmFinders) {
            uint32_t h = 2166136261u;
            for (int i = 0; i < 16; i++) h = (h ^ a.delays[16 * (long long)t + i]) * 16777619u;
            hash[t] = h;
        }
        auto meet = [] { asm volatile("bar.sync 1, %0;" ::"n"(kBmFinders) : "memory"); };
        meet();
        // rep[t]: the first tile with tile t's delays; list: those first tiles; rank: their places in it
        int count = 0;
        for (int t0 = 0; t0 < a.ntile; t0 += kBmFinders) {
            const int t = t0 + tid;
            const int r = t < a.ntile ? bm_first_equal(hash, a.delays, t) : -1;
            if (t < a.ntile) rep[t] = r;
            const bool first = r == t;
            __syncwarp();
            const unsigned b = __ballot_sync(0xffffffffu, first);
            if (lane == 0) warp_count[warp] = __popc(b);
            meet();
            int at = count;
            for (int w = 0; w < kBmFinders / 32; w++) {
                if (w < warp) at += warp_count[w];
                count += warp_count[w];
            }
            if (first) {
                rank[t] = at + __popc(b & ((1u << lane) - 1));
                list[rank[t]] = t;
            }
            meet();
        }
        if (tid == 0) nlist = count;
    } else if (warp == kBmFinders / 32) {
        if (lane < 2 * np) {
            const long long pr = p0 + lane / 2;
            const int pt = (int)(pr % a.npointing), fi = (int)(pr / a.npointing);
            const BmDir v = bm_dir2(lane & 1, np == 2 ? 0xFu : 0x3u, a.az[pt], a.za[pt], a.freq[fi]);
            if ((lane & 1) == 0) dir[lane / 2] = v;
        }
    } else if (a.pa && lane < np) {
        double p[4];
        const int pt = (int)((p0 + lane) % a.npointing);
        bm_pa(a.lat, a.az[pt], a.za[pt], p);
        for (int e = 0; e < 4; e++) P[lane][e] = p[e];
    }
    __syncthreads();
    const int share = blockIdx.y, shares = gridDim.y;
    if (share >= nlist) return;
    const int nsets = (nlist - share + shares - 1) / shares; // list[share + shares i]

    // items: (pair, set), 16 lanes each
    const int items = np * nsets;
    double2 *out = a.B + 4 * p0 * a.ntile;
    for (int e = tid >> 4; e < items; e += kBmGroups) {
        const int j = e / nsets, t = list[share + shares * (e - j * nsets)];
        bm_write16(tid & 15, 0xFFFFu << (lane & 16), dir[j], a.delays + 16 * (long long)t, a.pa ? P[j] : nullptr,
                   out + 4 * ((long long)j * a.ntile + t));
    }
    __syncthreads();
    // every other tile of these sets copies its set's matrix, 16 bytes per thread
    for (int i = tid; i < np * a.ntile * 4; i += kBmThreads) {
        const int t = (i / 4) % a.ntile, r = rep[t];
        if (r != t && rank[r] % shares == share) out[i] = out[i + 4 * (r - t)];
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
        const int sms = sm_count(), per_block = pairs <= sms ? 1 : 2;
        const int blocks = (int)((pairs + per_block - 1) / per_block);
        // shares of the sets: down to one round of a block's lanes each, as long as each block has an SM to itself
        const int shares = std::max(1, std::min((a.ntile + kBmGroups - 1) / kBmGroups, sms / blocks));
        beam_kernel_fused<<<dim3(blocks, shares), kBmThreads, sizeof(int) * (bm_hashes(a.ntile) + 3 * a.ntile), st>>>(a, per_block);
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
