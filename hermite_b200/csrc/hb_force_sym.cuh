// hb_force_sym.cuh -- FP64 force with every pair of active particles taken once
// (4th and 6th order).
//
// Newton's third law holds for every derivative of the pair force: one
// evaluation of the pair algebra (interact64, hb_math.cuh) serves both
// particles, 63 FP64 instructions instead of 2 x 53 at 6th order, 38 instead of
// 2 x 31 at 4th.  It pays where a large part of all pairs is between active
// particles: the start-up passes and the steps in which most particles move.
// (The reference sums ordered pairs: SRC/hermite4-titan.cu:189-238,
// SRC/hermite6-titan.cu:245-299.)
//
// Groups of 512 slots at 4th order, 384 at 6th (4 warps x 4 or 3 chunks of
// i-particles, one per lane and chunk) meet every later chunk of active
// particles: lane l of a warp takes j = l + s of the chunk in step s, and the
// chunk's running sums move one lane per step by shuffles, so that a step adds to
// 4 or 3 i-sums and one j-sum of every lane with no collisions and the j-sums are
// home after 32 steps.  The group's
// own chunks and the inactive particles are summed one-sided.
//
// The warps' j-sums meet in shared memory and go out as a row per group; a
// launch takes a band of groups, as many as the scratch has rows for, cut into
// j-slices; sym_band_kernel adds a band's rows and slices to the forces in a fixed
// order, so results are deterministic.
//
// What bounds it: the FP64 pipe (76 % busy while an SM has CTAs) beside the
// j-states' loads and the shuffles, 20 + 18 shared-memory cycles per step at 6th
// order for 3 x 63 FP64 instructions: with one i-chunk per warp those bound it (339
// Gint/s at N = 131072), with two 401, three 415, four 418, five 389 (spills), all
// with 6 waves and 16 rows; 440 with 20 and 64.  Ordered pairs 292.  4th order, N =
// 65536: 741 against 505.  A band's sums and its last CTAs are 2-3 % of the time.
#pragma once
#include "hb_common.cuh"
#include "hb_force.cuh"
#include "hb_internal.h"
#include "hb_math.cuh"

namespace hb {

constexpr int kSymFWarps = 4, kSymFTile = 4;

struct SymArgs {
    const double *pred;
    double *rows, *cols;   // j-sums [group][active chunk][F][32]; i-sums [group][smax][GC chunks][F][32]
    double *force;         // [nact][F]
    int nchunk, ca;        // chunks of all slots; chunks with active ones
    int nact;
    int g0, ng, smax, lc;  // band: first group, groups, slices per group at most, chunks per slice
    double eps2;
    int *err;
    unsigned spin;
};

// Slices of group g: its own chunks and those after them.
__host__ __device__ __forceinline__ int sym_slices(int nchunk, int g, int gc, int lc)
{
    return (nchunk - g * gc + lc - 1) / lc;
}

// One pair for both: f gets i's share (J.m), fj the negated share of j (I.m).
template <int ORDER>
__device__ __forceinline__ void interact64_both(const Body64 &I, const Body64 &J, double eps2,
                                                double *f, double *fj)
{
    double dr[3], dv[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        dr[k] = J.x[k] - I.x[k];
        dv[k] = J.v[k] - I.v[k];
    }
    const double r2 = fma(dr[2], dr[2], fma(dr[1], dr[1], fma(dr[0], dr[0], eps2)));
    const double rv = fma(dr[2], dv[2], fma(dr[1], dv[1], dr[0] * dv[0]));
    const double ri = rsqrt_fp64(r2);
    const double ri2 = ri * ri, ri3 = ri * ri2;
    const double mj = J.m * ri3, mi = I.m * ri3;
    const double al = rv * ri2;              // alpha = (r.v)/r^2
    double t[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        f[k] = fma(mj, dr[k], f[k]);
        fj[k] = fma(-mi, dr[k], fj[k]);
        t[k] = fma(-3.0 * al, dr[k], dv[k]);   // v - 3 alpha r
        f[3 + k] = fma(mj, t[k], f[3 + k]);
        fj[3 + k] = fma(-mi, t[k], fj[3 + k]);
    }
    if constexpr (ORDER >= 6) {
        double da[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) da[k] = J.a[k] - I.a[k];
        const double vvra = fma(dr[2], da[2], fma(dr[1], da[1], fma(dr[0], da[0],
                            fma(dv[2], dv[2], fma(dv[1], dv[1], dv[0] * dv[0])))));
        const double be = fma(al, al, vvra * ri2);       // beta
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const double u = fma(-3.0 * be, dr[k], fma(-6.0 * al, t[k], da[k]));
            f[6 + k] = fma(mj, u, f[6 + k]);
            fj[6 + k] = fma(-mi, u, fj[6 + k]);
        }
    }
}

template <int ORDER>
struct SymShape {
    static constexpr int NI = ORDER == 4 ? 4 : 3;   // i-chunks per warp
    static constexpr int MINB = 2;                 // CTAs per SM
    static constexpr int unroll = ORDER == 4 ? 2 : 8;   // steps; all of 1, 2, 4, 8 within 2 %
    static constexpr int GC = kSymFWarps * NI;            // chunks of a group
    static constexpr int F = Frc<ORDER>::words, CB = Pred64<ORDER>::chunk_bytes;
    static constexpr int tile_bytes = kSymFTile * CB;
    static constexpr int acc_off = 2 * tile_bytes;                     // [warp][tile chunk][F][32]
    static constexpr int bar_off = acc_off + kSymFWarps * kSymFTile * F * 32 * 8;
    static constexpr int bytes = bar_off + 16;
};

template <int ORDER>
__global__ void __launch_bounds__(kSymFWarps * 32, SymShape<ORDER>::MINB)
force_sym_kernel(const SymArgs a)
{
    pdl_enter();
    using Sh = SymShape<ORDER>;
    constexpr int F = Sh::F, NC = Pred64<ORDER>::ncomp, NI = Sh::NI, GC = Sh::GC, T = kSymFWarps * 32;
    constexpr int UNROLL = Sh::unroll;
    extern __shared__ __align__(128) unsigned char smem[];
    double *accj = reinterpret_cast<double *>(smem + Sh::acc_off);
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem + Sh::bar_off);
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    int g = a.g0, s = blockIdx.x;
    while (s >= sym_slices(a.nchunk, g, GC, a.lc)) s -= sym_slices(a.nchunk, g++, GC, a.lc);
    const int own0 = g * GC, own1 = own0 + GC;
    const int c0 = own0 + s * a.lc, c1 = min(c0 + a.lc, a.nchunk);
    const int ntile = (c1 - c0 + kSymFTile - 1) / kSymFTile;

    if (tid == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        fence_mbar_init();
    }
    __syncthreads();
    auto issue = [&](int t) {
        const int cnt = min(kSymFTile, c1 - c0 - t * kSymFTile);
        mbar_arrive_expect_tx(&bar[t & 1], (uint32_t)(cnt * Sh::CB));
        bulk_load(smem + (t & 1) * Sh::tile_bytes, a.pred + (size_t)(c0 + t * kSymFTile) * NC * 32,
                  (uint32_t)(cnt * Sh::CB), &bar[t & 1]);
    };
    if (tid == 0) {
        issue(0);
        if (ntile > 1) issue(1);
    }
    // this lane's i-particles; one that is not active adds nothing to the j-sums
    Body64 I[NI];
    double f[NI][F];
#pragma unroll
    for (int n = 0; n < NI; ++n) {
        const int ci = own0 + w * NI + n;
        load_i64<ORDER>(a.pred, min(ci, a.nchunk - 1), lane, I[n]);
        if (ci * 32 + lane >= a.nact) I[n].m = 0.0;
#pragma unroll
        for (int c = 0; c < F; ++c) f[n][c] = 0.0;
    }
    for (int t = 0; t < ntile; ++t) {
        const bool got = mbar_wait_bounded(&bar[t & 1], (uint32_t)((t >> 1) & 1), a.spin);
        if (!__syncthreads_and(got)) {
            if (tid == 0) {
                raise_error(a.err, kErrWaitTimeout);
                for (int u = t; u < ntile && u < t + 2; ++u)
                    mbar_wait_bounded(&bar[u & 1], (uint32_t)((u >> 1) & 1));
            }
            return;
        }
        const int ct = c0 + t * kSymFTile, cnt = min(kSymFTile, c1 - ct);
        const double *tile = reinterpret_cast<const double *>(smem + (t & 1) * Sh::tile_bytes);
        // the tile's chunks past the group that hold active particles
        const int q0 = min(max(own1 - ct, 0), cnt), q1 = max(q0, min(a.ca - ct, cnt));
#pragma unroll 1
        for (int q = 0; q < cnt; ++q) {
            const double *cp = tile + q * NC * 32;
            if (q < q0 || q >= q1) {
                chunk64<ORDER, NI>(cp, I, a.eps2, f);
                continue;
            }
            double fj[F];
#pragma unroll
            for (int c = 0; c < F; ++c) fj[c] = 0.0;
            const int next = (lane + 1) & 31;
            int jl = lane;
#pragma unroll UNROLL
            for (int st = 0; st < 32; ++st) {
                Body64 J;
                load_i64<ORDER>(cp, 0, jl, J);
#pragma unroll
                for (int n = 0; n < NI; ++n) interact64_both<ORDER>(I[n], J, a.eps2, f[n], fj);
                jl = (jl + 1) & 31;
#pragma unroll
                for (int c = 0; c < F; ++c) fj[c] = __shfl_sync(0xffffffffu, fj[c], next);
            }
            double *o = accj + (size_t)(w * kSymFTile + q) * F * 32 + lane;
#pragma unroll
            for (int c = 0; c < F; ++c) o[c * 32] = fj[c];
        }
        __syncthreads();
        if (tid == 0 && t + 2 < ntile) issue(t + 2);
        if (q1 > q0) {
            double *row = a.rows + ((size_t)(g - a.g0) * a.ca + ct) * F * 32;
            for (int e = q0 * F * 32 + tid; e < q1 * F * 32; e += T) {
                double v = accj[e];
#pragma unroll
                for (int ww = 1; ww < kSymFWarps; ++ww) v += accj[ww * kSymFTile * F * 32 + e];
                row[e] = v;
            }
            __syncthreads();
        }
    }
    double *col = a.cols + (((size_t)(g - a.g0) * a.smax + s) * GC + w * NI) * F * 32 + lane;
#pragma unroll
    for (int n = 0; n < NI; ++n)
#pragma unroll
        for (int c = 0; c < F; ++c) col[(n * F + c) * 32] = f[n][c];
}

// Adds a band's sums to the forces of the chunks from its first group on.
template <int ORDER>
__global__ void __launch_bounds__(256)
sym_band_kernel(const SymArgs a)
{
    pdl_enter();
    constexpr int F = SymShape<ORDER>::F, GC = SymShape<ORDER>::GC;
    const int first = a.g0 * GC;
    const long long e = (long long)blockIdx.x * 256 + threadIdx.x;     // [chunk][F][32]
    const int c = first + (int)(e / (F * 32)), comp = (int)(e / 32) % F, j = c * 32 + (int)(e & 31);
    if (c >= a.ca || j >= a.nact) return;
    const int gj = c / GC;
    double *out = a.force + (size_t)j * F + comp;
    double acc[8] = {a.g0 > 0 ? *out : 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    auto add = [&](const double *p, size_t stride, int cnt) {
        int k = 0;
        for (; k + 8 <= cnt; k += 8)
#pragma unroll
            for (int u = 0; u < 8; ++u) acc[u] += __ldcg(p + (size_t)(k + u) * stride);
#pragma unroll
        for (int u = 0; u < 7; ++u)
            if (k + u < cnt) acc[u] += __ldcg(p + (size_t)(k + u) * stride);
    };
    // rows of the band's groups below j's own, then j's own slices
    const size_t in_row = (size_t)c * F * 32 + comp * 32 + (j & 31);
    add(a.rows + in_row, (size_t)a.ca * F * 32, min(gj - a.g0, a.ng));
    if (gj - a.g0 < a.ng)
        add(a.cols + ((size_t)(gj - a.g0) * a.smax * GC + (c - gj * GC)) * F * 32 + comp * 32 + (j & 31),
            (size_t)GC * F * 32, sym_slices(a.nchunk, gj, GC, a.lc));
    *out = ((acc[0] + acc[1]) + (acc[2] + acc[3])) + ((acc[4] + acc[5]) + (acc[6] + acc[7]));
}

}  // namespace hb
