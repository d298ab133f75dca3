// hb_predict_pot.cu -- predictor, potential and the FMA-peak probe.
#include <algorithm>
#include <type_traits>
#include "hb_internal.h"
#include "hb_math.cuh"

namespace hb {

// ---------------------------------------------------------------------------
// Predictor (replaces predict_kernel, SRC/hermite4-titan.cu:80-99,
// SRC/hermite6-titan.cu:113-133, SRC/hermite8-titan.cu:153-172).
// One thread per slot.  The CTA's 128 contiguous AoS records are brought into
// shared memory by one bulk async copy; the outputs are written per
// component into the AoSoA32 predicted layout (full 128/256-byte stores).
// Slots in [n, npad) are written as zero-mass far-away padding.
constexpr int kPredThreads = 128;

template <int ORDER, bool MIXED>
__global__ void __launch_bounds__(kPredThreads)
predict_kernel(const double *__restrict__ jp, int n, int npad, double tsys,
               void *__restrict__ pred, int *err)
{
    constexpr int R = Rec<ORDER>::words;
    __shared__ __align__(128) double rec[kPredThreads * R];
    __shared__ __align__(8) uint64_t bar;
    pdl_enter();
    const int tid = threadIdx.x;
    const int base = blockIdx.x * kPredThreads;
    const int cnt = min(kPredThreads, n - base);

    if (cnt > 0) {
        if (tid == 0) {
            mbar_init(&bar, 1);
            fence_mbar_init();
        }
        __syncthreads();
        if (tid == 0) {
            // a bulk copy moves a multiple of 16 bytes: with 29-word records
            // (ORDER 9) a partial last block rounds up by 8 bytes, which stay
            // inside the padded record array and the staging buffer
            const uint32_t bytes = (uint32_t)((cnt * R * 8 + 15) & ~15);
            mbar_arrive_expect_tx(&bar, bytes);
            bulk_load(rec, jp + (size_t)base * R, bytes, &bar);
        }
        const bool ok = mbar_wait_bounded(&bar, 0);
        if (!__syncthreads_and(ok)) {
            if (tid == 0) {
                raise_error(err, kErrWaitTimeout);
                mbar_wait_bounded(&bar, 0);
            }
            return;
        }
    }
    const int slot = base + tid;
    if (slot >= npad) return;
    double x[3], v[3], a[3] = {0, 0, 0}, jk[3] = {0, 0, 0}, xl[3] = {0, 0, 0}, m;
    if (tid < cnt) {
        const double *r = rec + tid * R;
        predict_slot<ORDER>(r, tsys, x, v, a, jk, xl);
        m = r[3];
    } else {
        for (int k = 0; k < 3; ++k) { x[k] = pad_position(slot, k); v[k] = 0.0; }
        m = 0.0;
    }
    const int ci = slot >> 5, lane = slot & 31;
    if constexpr (MIXED) {
        constexpr int NC = PredMx<ORDER>::ncomp;
        float *c = static_cast<float *>(pred) + (size_t)ci * NC * 32 + lane;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float hi = __double2float_rn(x[k]);
            c[(PMX_XH + k) * 32] = hi;
            c[(PMX_XL + k) * 32] = __double2float_rn(x[k] - (double)hi);
            c[(PMX_V + k) * 32] = __double2float_rn(v[k]);
            if constexpr (ORDER >= 6) c[(PMX_A + k) * 32] = __double2float_rn(a[k]);
            if constexpr (ORDER == 8) c[(PMX_J + k) * 32] = __double2float_rn(jk[k]);
        }
        c[PMX_M * 32] = __double2float_rn(m);
    } else {
        constexpr int NC = Pred64<ORDER>::ncomp;
        double *c = static_cast<double *>(pred) + (size_t)ci * NC * 32 + lane;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            c[(P64_X + k) * 32] = x[k];
            c[(P64_V + k) * 32] = v[k];
            if constexpr (ORDER >= 6) c[(P64_A + k) * 32] = a[k];
            if constexpr (ORDER >= 8) c[(P64_J + k) * 32] = jk[k];
            if constexpr (ORDER == 9) c[(P64_XL + k) * 32] = xl[k];
        }
        c[P64_M * 32] = m;
    }
}

template <int ORDER, bool MIXED>
static cudaError_t launch_predict_t(const double *jp, int n, int npad, double tsys,
                                    void *pred, int *err, cudaStream_t s)
{
    const int grid = npad / kPredThreads;   // npad is a multiple of 256
    predict_kernel<ORDER, MIXED><<<grid, kPredThreads, 0, s>>>(jp, n, npad, tsys, pred, err);
    return cudaGetLastError();
}

cudaError_t launch_predict(int order, bool mixed, const double *jp, int n, int npad,
                           double tsys, void *pred, int *err, cudaStream_t s)
{
    switch (order * 2 + (mixed ? 1 : 0)) {
    case 8:  return launch_predict_t<4, false>(jp, n, npad, tsys, pred, err, s);
    case 9:  return launch_predict_t<4, true>(jp, n, npad, tsys, pred, err, s);
    case 12: return launch_predict_t<6, false>(jp, n, npad, tsys, pred, err, s);
    case 13: return launch_predict_t<6, true>(jp, n, npad, tsys, pred, err, s);
    case 16: return launch_predict_t<8, false>(jp, n, npad, tsys, pred, err, s);
    case 17: return launch_predict_t<8, true>(jp, n, npad, tsys, pred, err, s);
    case 18: return launch_predict_t<9, false>(jp, n, npad, tsys, pred, err, s);
    }
    return cudaErrorInvalidValue;
}

// ---------------------------------------------------------------------------
// Sum of the j-slices' partial forces (replaces reduce_kernel,
// SRC/hermite4-titan.cu:303-327 and its 6th/8th-order counterparts).
// A block takes 32 consecutive values and G groups of a warp each: group g adds slices
// g, g + G, ... in 8 interleaved sums (8 loads in flight), combined pairwise;
// the groups' sums likewise: at most log2(G) + 2 roundings in a row there, where group
// order had 31.
template <int G>
__global__ void __launch_bounds__(G * 32)
reduce_kernel(const double *__restrict__ partial, size_t stride, int S, int v,
              double *__restrict__ force)
{
    pdl_enter();
    __shared__ double red[G][32];
    const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
    const int e = blockIdx.x * 32 + lane;
    double acc[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    if (e < v) {
        const double *p = partial + e;
        int s = g;
        for (; s + 7 * G < S; s += 8 * G)
#pragma unroll
            for (int u = 0; u < 8; ++u) acc[u] += __ldcg(p + (size_t)(s + u * G) * stride);
#pragma unroll
        for (int u = 0; u < 7; ++u)
            if (s + u * G < S) acc[u] += __ldcg(p + (size_t)(s + u * G) * stride);
    }
    red[g][lane] = ((acc[0] + acc[1]) + (acc[2] + acc[3])) + ((acc[4] + acc[5]) + (acc[6] + acc[7]));
    __syncthreads();
    if (g == 0 && e < v) {
        constexpr int W = G < 8 ? G : 8;
        double sum[W];
#pragma unroll
        for (int u = 0; u < W; ++u) {
            sum[u] = red[u][lane];
#pragma unroll
            for (int k = u + W; k < G; k += W) sum[u] += red[k][lane];
        }
#pragma unroll
        for (int w = W / 2; w > 0; w /= 2)
#pragma unroll
            for (int u = 0; u < w; ++u) sum[u] += sum[u + w];
        force[e] = sum[0];
    }
}

cudaError_t launch_reduce(const double *partial, size_t stride, int S, int v, double *force,
                          cudaStream_t s)
{
    const dim3 grid((v + 31) / 32);
    if (S <= 16) return launch_pdl(reduce_kernel<2>, grid, 64, 0, s, partial, stride, S, v, force);
    if (S <= 64) return launch_pdl(reduce_kernel<8>, grid, 256, 0, s, partial, stride, S, v, force);
    return launch_pdl(reduce_kernel<32>, grid, 1024, 0, s, partial, stride, S, v, force);
}

// ---------------------------------------------------------------------------
// Potential (replaces pot_kernel + calc_potential, SRC/pot-titan.hu:80-171).
// Pass 1 packs (x, y, z, m) of the un-predicted records into AoSoA32;
// pass 2 sums phi_i = -sum_{j != i} m_j / sqrt(r^2 + eps2) in FP64 with the
// same bulk-copy ring as the force kernel.  Each 32-slot chunk is summed
// separately and then added to the running total (two-level blocked sum;
// the reference uses a four-level cascade, SRC/pot-titan.hu:103-114).
// ORDER 9 (double-double positions) packs (x, y, z, m, xL, yL, zL) and takes
// the separation as (xj - xi) + (xLj - xLi) (calc_potential,
// SRC/hermite8dd.h:397-416).
template <int ORDER> constexpr int posm_comps() { return ORDER == 9 ? 7 : 4; }

template <int ORDER>
__global__ void pack_posm_kernel(const double *__restrict__ jp, int n, int npad,
                                 double *__restrict__ posm)
{
    pdl_enter();
    constexpr int R = Rec<ORDER>::words, NC = posm_comps<ORDER>();
    const int slot = blockIdx.x * blockDim.x + threadIdx.x;
    if (slot >= npad) return;
    double *c = posm + (size_t)(slot >> 5) * NC * 32 + (slot & 31);
    if (slot < n) {
        const double *r = jp + (size_t)slot * R;
        for (int k = 0; k < 4; ++k) c[k * 32] = r[k];
        if constexpr (NC == 7)
            for (int k = 0; k < 3; ++k) c[(4 + k) * 32] = r[kRecPosL + k];
    } else {
        for (int k = 0; k < 3; ++k) c[k * 32] = pad_position(slot, k);
        c[3 * 32] = 0.0;
        if constexpr (NC == 7)
            for (int k = 0; k < 3; ++k) c[(4 + k) * 32] = 0.0;
    }
}

constexpr int kPotThreads = 128;
constexpr int kPotTileChunks = 8;

// j-slice blockIdx.y of gridDim.y writes its sums to row blockIdx.y of pot (row
// stride `stride`).
template <int NC>
__global__ void __launch_bounds__(kPotThreads)
potential_kernel(const double *__restrict__ posm, int nchunk, int n, double eps2,
                 double *__restrict__ pot, size_t stride, int *err)
{
    pdl_enter();
    constexpr int kPosmChunkBytes = NC * 32 * 8;
    constexpr int TB = kPotTileChunks * kPosmChunkBytes;
    __shared__ __align__(128) unsigned char ring[2 * TB];
    __shared__ __align__(8) uint64_t bar[2];
    const int tid = threadIdx.x, lane = tid & 31;
    const int i = blockIdx.x * kPotThreads + tid;   // < npad always
    const double *ci = posm + (size_t)(i >> 5) * NC * 32 + (i & 31);
    const double xi = ci[0], yi = ci[32], zi = ci[64];
    double xli = 0.0, yli = 0.0, zli = 0.0;
    if constexpr (NC == 7) {
        xli = ci[128];
        yli = ci[160];
        zli = ci[192];
    }
    const int c0 = (int)((long long)blockIdx.y * nchunk / gridDim.y);
    const int c1 = (int)((long long)(blockIdx.y + 1) * nchunk / gridDim.y);
    const int ntile = (c1 - c0 + kPotTileChunks - 1) / kPotTileChunks;

    if (tid == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        fence_mbar_init();
    }
    __syncthreads();
    auto issue = [&](int t) {
        const int cnt = min(kPotTileChunks, c1 - c0 - t * kPotTileChunks);
        const uint32_t bytes = (uint32_t)(cnt * kPosmChunkBytes);
        mbar_arrive_expect_tx(&bar[t & 1], bytes);
        bulk_load(ring + (t & 1) * TB,
                  reinterpret_cast<const unsigned char *>(posm) + (size_t)c0 * kPosmChunkBytes + (size_t)t * TB,
                  bytes, &bar[t & 1]);
    };
    if (tid == 0) {
        issue(0);
        if (ntile > 1) issue(1);
    }
    double total = 0.0;
    for (int t = 0; t < ntile; ++t) {
        const bool got = mbar_wait_bounded(&bar[t & 1], (uint32_t)((t >> 1) & 1));
        if (!__syncthreads_and(got)) {
            if (tid == 0) {
                raise_error(err, kErrWaitTimeout);
                for (int u = t; u < ntile && u < t + 2; ++u)
                    mbar_wait_bounded(&bar[u & 1], (uint32_t)((u >> 1) & 1));
            }
            return;
        }
        const int cnt = min(kPotTileChunks, c1 - c0 - t * kPotTileChunks);
        const double *tile = reinterpret_cast<const double *>(ring + (t & 1) * TB);
        for (int q = 0; q < cnt; ++q) {
            const double *cp = tile + q * NC * 32;
            // The self pair is left out, by index, in the one chunk that holds it.
            // (Looking for it in every chunk, by a branch around the rsqrt, took
            // 48 us instead of 34 at N = 100, and 24.1 ms instead of 20.4 at N =
            // 131072 in double-double.)
            auto pairs = [&](auto diag) {
                double part = 0.0;
#pragma unroll 8
                for (int jl = 0; jl < 32; ++jl) {
                    double dx = cp[jl] - xi, dy = cp[32 + jl] - yi, dz = cp[64 + jl] - zi;
                    if constexpr (NC == 7) {
                        dx = dx + (cp[128 + jl] - xli);
                        dy = dy + (cp[160 + jl] - yli);
                        dz = dz + (cp[192 + jl] - zli);
                    }
                    double r2 = fma(dz, dz, fma(dy, dy, fma(dx, dx, eps2)));
                    double mj = cp[96 + jl];
                    if (diag.value && jl == lane) {      // any finite rsqrt, no mass
                        r2 = 1.0;
                        mj = 0.0;
                    }
                    part = fma(-mj, rsqrt_fp64(r2), part);
                }
                total += part;
            };
            if (c0 + t * kPotTileChunks + q == (i >> 5)) pairs(std::true_type());
            else pairs(std::false_type());
        }
        __syncthreads();
        if (tid == 0 && t + 2 < ntile) issue(t + 2);
    }
    if (i < n) pot[blockIdx.y * stride + i] = total;
}

// Each pair once: a pair's rsqrt serves both particles (13 FP64 instructions
// for two interactions instead of 24).
//
// Groups of 1024 slots (8 warps x 4 chunks of i-particles, one per lane and
// chunk) meet every later chunk: lane l of a warp takes j = l + s of the chunk
// in step s, the chunk's running sums moving one lane per step by a shuffle
// (the states moving along instead of being read again measured 4 % slower).
// So a step adds to 4 i-sums and to one j-sum of every lane with no collisions,
// and after 32 steps the j-sums are home.  The 8 warps' j-sums meet in shared
// memory and go out once per (group, j).  The group's own chunks are summed
// one-sided, as ordered pairs; the self pair is step 0 of a chunk with itself.
//
// A launch takes a band of groups, as many as `partial` has rows for, cut into
// slices of `lc` chunks; pot_band_kernel then adds rows and slices to the
// potentials in a fixed order, so results are deterministic.
//
// N = 100003: 5.08 ms (11.0 ms with ordered pairs and no slices); the FP64 pipe
// is 80 % busy, its 13 instructions per pair and little else; 8 i-chunks a warp, 2 of
// 16 warps, three CTAs per SM and other unrollings measured 0-10 % slower.
constexpr int kSymWarps = 8, kSymI = 4, kSymTile = 16;
constexpr int kSymChunks = kSymWarps * kSymI, kSymSlots = kSymChunks * 32;

struct PotBand {
    const double *posm;
    double *rows, *cols;   // j-sums [group][npad]; i-sums [group][smax][kSymSlots]
    int g0, ng, smax, lc, nchunk;
    double eps2;
    int *err;
};

__host__ __device__ __forceinline__ int pot_slices(int nchunk, int g, int lc)
{
    return (nchunk - g * kSymChunks + lc - 1) / lc;
}

template <bool DIAG>
__device__ __forceinline__ void pot_chunk(const double *cp, int lane, const double (&xi)[kSymI][3],
                                          const double (&mi)[kSymI], const bool (&own)[kSymI],
                                          double eps2, double (&total)[kSymI], double &fj)
{
    double part[kSymI];
#pragma unroll
    for (int k = 0; k < kSymI; ++k) part[k] = 0.0;
    fj = 0.0;
    const int next = (lane + 1) & 31;
    int jl = lane;
#pragma unroll 4
    for (int s = 0; s < 32; ++s) {
        const double x = cp[jl], y = cp[32 + jl], z = cp[64 + jl], m = cp[96 + jl];
#pragma unroll
        for (int k = 0; k < kSymI; ++k) {
            const double dx = x - xi[k][0], dy = y - xi[k][1], dz = z - xi[k][2];
            double ri = rsqrt_fp64(fma(dz, dz, fma(dy, dy, fma(dx, dx, eps2))));
            if (DIAG && s == 0 && own[k]) ri = 0.0;
            part[k] = fma(-m, ri, part[k]);
            if (!DIAG) fj = fma(-mi[k], ri, fj);
        }
        jl = (jl + 1) & 31;
        if (!DIAG) fj = __shfl_sync(0xffffffffu, fj, next);
    }
#pragma unroll
    for (int k = 0; k < kSymI; ++k) total[k] += part[k];
}

__global__ void __launch_bounds__(kSymWarps * 32, 2)
potential_sym_kernel(const PotBand a)
{
    pdl_enter();
    constexpr int CB = 4 * 32 * 8, TB = kSymTile * CB, T = kSymWarps * 32;
    extern __shared__ __align__(128) unsigned char smem[];
    double *accj = reinterpret_cast<double *>(smem + 2 * TB);      // [warp][tile chunk][32]
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem + 2 * TB + kSymWarps * kSymTile * 32 * 8);
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    int g = a.g0, s = blockIdx.x;
    while (s >= pot_slices(a.nchunk, g, a.lc)) s -= pot_slices(a.nchunk, g++, a.lc);
    const int own0 = g * kSymChunks, own1 = min(own0 + kSymChunks, a.nchunk);
    const int c0 = own0 + s * a.lc, c1 = min(c0 + a.lc, a.nchunk);

    double xi[kSymI][3], mi[kSymI], total[kSymI];
#pragma unroll
    for (int k = 0; k < kSymI; ++k) {
        const int ci = own0 + w * kSymI + k;
        const double *p = a.posm + (size_t)min(ci, a.nchunk - 1) * 4 * 32 + lane;
        for (int d = 0; d < 3; ++d) xi[k][d] = p[d * 32];
        mi[k] = ci < a.nchunk ? p[96] : 0.0;       // past the last chunk: adds nothing
        total[k] = 0.0;
    }
    if (tid == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        fence_mbar_init();
    }
    __syncthreads();
    const int ntile = (c1 - c0 + kSymTile - 1) / kSymTile;
    auto issue = [&](int t) {
        const uint32_t bytes = (uint32_t)(min(kSymTile, c1 - c0 - t * kSymTile) * CB);
        mbar_arrive_expect_tx(&bar[t & 1], bytes);
        bulk_load(smem + (t & 1) * TB, a.posm + (size_t)(c0 + t * kSymTile) * 4 * 32, bytes, &bar[t & 1]);
    };
    if (tid == 0) {
        issue(0);
        if (ntile > 1) issue(1);
    }
    for (int t = 0; t < ntile; ++t) {
        const bool got = mbar_wait_bounded(&bar[t & 1], (uint32_t)((t >> 1) & 1));
        if (!__syncthreads_and(got)) {
            if (tid == 0) {
                raise_error(a.err, kErrWaitTimeout);
                for (int u = t; u < ntile && u < t + 2; ++u)
                    mbar_wait_bounded(&bar[u & 1], (uint32_t)((u >> 1) & 1));
            }
            return;
        }
        // lc and the groups are whole tiles: a tile is in the group or past it
        const int ct = c0 + t * kSymTile, cnt = min(kSymTile, c1 - ct);
        const double *tile = reinterpret_cast<const double *>(smem + (t & 1) * TB);
        const bool diag = ct < own1;
        for (int q = 0; q < cnt; ++q) {
            double fj;
            bool own[kSymI];
            if (diag) {
#pragma unroll
                for (int k = 0; k < kSymI; ++k) own[k] = ct + q == own0 + w * kSymI + k;
                pot_chunk<true>(tile + q * 4 * 32, lane, xi, mi, own, a.eps2, total, fj);
            } else {
                pot_chunk<false>(tile + q * 4 * 32, lane, xi, mi, own, a.eps2, total, fj);
                accj[(w * kSymTile + q) * 32 + lane] = fj;
            }
        }
        __syncthreads();
        if (tid == 0 && t + 2 < ntile) issue(t + 2);
        if (!diag) {
            double *row = a.rows + (size_t)(g - a.g0) * a.nchunk * 32 + (size_t)ct * 32;
            for (int e = tid; e < cnt * 32; e += T) {
                double v = accj[e];
#pragma unroll
                for (int ww = 1; ww < kSymWarps; ++ww) v += accj[ww * kSymTile * 32 + e];
                row[e] = v;
            }
            __syncthreads();
        }
    }
    double *col = a.cols + ((size_t)(g - a.g0) * a.smax + s) * kSymSlots;
#pragma unroll
    for (int k = 0; k < kSymI; ++k) col[(w * kSymI + k) * 32 + lane] = total[k];
}

// Adds a band's sums to the potentials of the slots from its first group on.
__global__ void __launch_bounds__(256)
pot_band_kernel(const PotBand a, int n, double *__restrict__ pot)
{
    pdl_enter();
    const int j = a.g0 * kSymSlots + blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const int gj = j / kSymSlots, before = min(gj - a.g0, a.ng);   // groups below j's own
    double acc[8] = {a.g0 > 0 ? pot[j] : 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    auto add = [&](const double *p, size_t stride, int cnt) {
        int k = 0;
        for (; k + 8 <= cnt; k += 8)
#pragma unroll
            for (int u = 0; u < 8; ++u) acc[u] += __ldcg(p + (size_t)(k + u) * stride);
#pragma unroll
        for (int u = 0; u < 7; ++u)
            if (k + u < cnt) acc[u] += __ldcg(p + (size_t)(k + u) * stride);
    };
    add(a.rows + j, (size_t)a.nchunk * 32, before);
    if (gj - a.g0 < a.ng)
        add(a.cols + (size_t)(gj - a.g0) * a.smax * kSymSlots + j % kSymSlots, kSymSlots,
            pot_slices(a.nchunk, gj, a.lc));
    pot[j] = ((acc[0] + acc[1]) + (acc[2] + acc[3])) + ((acc[4] + acc[5]) + (acc[6] + acc[7]));
}

// Each-pair-once potential in bands; *launches counts them.  Returns
// cudaErrorInvalidValue when `cap` doubles hold no band of one group.
static cudaError_t launch_potential_sym(int n, int npad, double eps2, const double *posm, double *pot,
                                        double *partial, size_t cap, int nsm, int *err,
                                        cudaStream_t s, int *launches)
{
    constexpr int smem = 2 * kSymTile * 4 * 32 * 8 + kSymWarps * kSymTile * 32 * 8 + 16;
    cudaError_t e = cudaFuncSetAttribute(potential_sym_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    PotBand a{};
    a.posm = posm;
    a.nchunk = npad / 32;
    a.eps2 = eps2;
    a.err = err;
    const int groups = (a.nchunk + kSymChunks - 1) / kSymChunks;
    for (int g0 = 0; g0 < groups; g0 += a.ng) {
        // about 8 waves of two CTAs per SM: a CTA's chunks, in whole tiles
        const long long wide = std::min((long long)groups - g0, (long long)(cap / npad));
        const long long units = std::max(1LL, wide) * (a.nchunk - (long long)g0 * kSymChunks);
        const long long lc = units / (16LL * nsm);
        a.g0 = g0;
        a.lc = (int)std::max(1LL, (lc + kSymTile - 1) / kSymTile) * kSymTile;
        a.smax = pot_slices(a.nchunk, g0, a.lc);
        const long long per = (long long)npad + (long long)a.smax * kSymSlots;
        a.ng = (int)std::min((long long)(groups - g0), (long long)cap / per);
        if (a.ng < 1) return cudaErrorInvalidValue;
        a.rows = partial;
        a.cols = partial + (size_t)a.ng * npad;
        int ctas = 0;
        for (int g = g0; g < g0 + a.ng; ++g) ctas += pot_slices(a.nchunk, g, a.lc);
        e = launch_pdl(potential_sym_kernel, dim3(ctas), kSymWarps * 32, smem, s, a);
        if (e == cudaSuccess)
            e = launch_pdl(pot_band_kernel, dim3((n - g0 * kSymSlots + 255) / 256), 256, 0, s, a, n, pot);
        if (e != cudaSuccess) return e;
        *launches += 2;
    }
    return cudaSuccess;
}

// From this many slots on the pairs are taken once: 16384: 191 against 283 us
// with ordered pairs, 100003: 5.08 against 8.90 ms, 262144: 34.3 against 60.8;
// 12000: 189 against 171 us, too few groups to fill the GPU evenly.
// Double-double positions keep the ordered pairs.
constexpr int kPotSymMin = 14336;

cudaError_t launch_potential(int order, const double *jp, int n, int npad, double eps2,
                             double *posm, double *pot, double *partial, size_t cap, int nsm,
                             int *err, cudaStream_t s, int *launches)
{
    const int g = npad / 128;
    switch (order) {
    case 4: pack_posm_kernel<4><<<g, 128, 0, s>>>(jp, n, npad, posm); break;
    case 6: pack_posm_kernel<6><<<g, 128, 0, s>>>(jp, n, npad, posm); break;
    case 8: pack_posm_kernel<8><<<g, 128, 0, s>>>(jp, n, npad, posm); break;
    case 9: pack_posm_kernel<9><<<g, 128, 0, s>>>(jp, n, npad, posm); break;
    default: return cudaErrorInvalidValue;
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    ++*launches;
    if (order != 9 && n >= kPotSymMin && (size_t)npad * 2 <= cap)
        return launch_potential_sym(n, npad, eps2, posm, pot, partial, cap, nsm, err, s, launches);
    // j-slices of at least one tile, about 4 waves of 12 CTAs per SM
    const int nchunk = npad / 32, gx = npad / kPotThreads;
    int S = std::max(1, std::min(nchunk / kPotTileChunks, 48 * nsm / gx));
    S = (int)std::min<size_t>(S, cap / npad);
    S = std::max(S, 1);
    double *out = S > 1 ? partial : pot;
    if (order == 9)
        e = launch_pdl(potential_kernel<7>, dim3(gx, S), kPotThreads, 0, s, (const double *)posm, nchunk, n,
                       eps2, out, (size_t)npad, err);
    else
        e = launch_pdl(potential_kernel<4>, dim3(gx, S), kPotThreads, 0, s, (const double *)posm, nchunk, n,
                       eps2, out, (size_t)npad, err);
    if (e != cudaSuccess) return e;
    ++*launches;
    if (S == 1) return cudaSuccess;
    ++*launches;
    return launch_reduce(partial, (size_t)npad, S, n, pot, s);
}

// ---------------------------------------------------------------------------
// FMA-pipe peak probe: independent register-resident FMA chains, no memory
// traffic inside the timed loop.  mode 0 = FP64 (DFMA), 1 = FP32 (FFMA),
// 2 = packed FP32 (f32x2 FMA, two FMAs per instruction).
constexpr int kPeakChains = 8;
constexpr int kPeakIters = 4096;

template <int MODE>
__global__ void __launch_bounds__(256) fma_peak_kernel(float seed, double *sink)
{
    if constexpr (MODE == 0) {
        double r[kPeakChains];
        for (int c = 0; c < kPeakChains; ++c) r[c] = seed + threadIdx.x + c;
        const double a = 0.999999, b = 1e-7;
#pragma unroll 4
        for (int it = 0; it < kPeakIters; ++it)
#pragma unroll
            for (int c = 0; c < kPeakChains; ++c) r[c] = fma(r[c], a, b);
        double s = 0;
        for (int c = 0; c < kPeakChains; ++c) s += r[c];
        if (s == 12345.678) sink[0] = s;
    } else if constexpr (MODE == 1) {
        float r[kPeakChains];
        for (int c = 0; c < kPeakChains; ++c) r[c] = seed + threadIdx.x + c;
        const float a = 0.999999f, b = 1e-7f;
#pragma unroll 4
        for (int it = 0; it < kPeakIters; ++it)
#pragma unroll
            for (int c = 0; c < kPeakChains; ++c) r[c] = fmaf(r[c], a, b);
        float s = 0;
        for (int c = 0; c < kPeakChains; ++c) s += r[c];
        if (s == 12345.678f) sink[0] = s;
    } else {
        float2 r[kPeakChains];
        for (int c = 0; c < kPeakChains; ++c) r[c] = make_float2(seed + threadIdx.x + c, seed - c);
        const float2 a = f2(0.999999f), b = f2(1e-7f);
#pragma unroll 4
        for (int it = 0; it < kPeakIters; ++it)
#pragma unroll
            for (int c = 0; c < kPeakChains; ++c) r[c] = fma2(r[c], a, b);
        float s = 0;
        for (int c = 0; c < kPeakChains; ++c) s += r[c].x + r[c].y;
        if (s == 12345.678f) sink[0] = s;
    }
}

cudaError_t run_fma_peak(int mode, int nsm, double *gflops)
{
    double *sink = nullptr;
    cudaError_t e = cudaMalloc(&sink, sizeof(double));
    if (e != cudaSuccess) return e;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    const int grid = nsm * 8, block = 256;
    auto launch = [&]() {
        if (mode == 0) fma_peak_kernel<0><<<grid, block>>>(1.0f, sink);
        else if (mode == 1) fma_peak_kernel<1><<<grid, block>>>(1.0f, sink);
        else fma_peak_kernel<2><<<grid, block>>>(1.0f, sink);
    };
    for (int w = 0; w < 3; ++w) launch();
    float best_ms = 1e30f;
    for (int rep = 0; rep < 5; ++rep) {
        cudaEventRecord(e0);
        launch();
        cudaEventRecord(e1);
        cudaEventSynchronize(e1);
        float ms = 0;
        cudaEventElapsedTime(&ms, e0, e1);
        if (ms < best_ms) best_ms = ms;
    }
    e = cudaGetLastError();
    const double fmas = (double)grid * block * kPeakIters * kPeakChains * (mode == 2 ? 2 : 1);
    *gflops = 2.0 * fmas / (best_ms * 1e-3) * 1e-9;
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(sink);
    return e;
}

}  // namespace hb
