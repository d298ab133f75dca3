// hb_force_lanes.cu -- FP64 force on a handful of active particles.
//
// The tiled force kernel (hb_force.cuh) gives every lane of a warp its own
// i-particle, so a block step with nact < 32 active particles leaves
// 32 - nact lanes idle: at nact = 1 the j sum runs at 1/32 of the FP64 pipe
// (about 24 us of arithmetic at N = 262144, 6th order, where the j records
// take 6.5 us to stream from HBM).
//
// Here a warp's 32 lanes form P groups of G = 32/P lanes, P = nact rounded
// up to a power of two (nact <= 16, so G >= 2; from 17 on, one lane per i,
// the tiled kernel measured faster at N >= 2^18).  The G lanes of group p share
// i-particle p and take every G-th j of each 32-slot chunk; their partial
// sums meet in a fixed xor-shuffle tree.  The warps of a CTA take the chunks
// of its j-slice in turn; each warp brings its chunks' raw records into shared
// memory by bulk copies, two in flight (every wait bounded), and predicts them
// there (one lane per slot), so a launch reads every j record once.  The CTAs of
// the grid are j-slices, added by a chained reduce launch.  Every sum has a fixed
// association for a given (nact, N), so results are deterministic.
//
// Measured at 6th order, N = 262144, back to back: nact = 1 / 4 / 16 take 11.1 /
// 14.5 / 25.5 us.  With the slices added by the last CTA (up to 37 rounds of
// loads in turn) and records read word by word (4-way bank conflicts) they
// took 14.5 / 18.5 / 37.6.  8th order, N = 2^20, nact = 1: 37.9 us, of which the
// records take 33.8 at the measured HBM copy rate.
//
// The same job as the reference's force_kernel with its j-blocks
// (SRC/hermite4-titan.cu:189-238, SRC/hermite6-titan.cu:245-299,
// SRC/hermite8-titan.cu:304-364) for the small blocks of the block-step
// scheme; the pair algebra is interact64 (hb_math.cuh).
#include <algorithm>
#include <mutex>

#include "hb_force.cuh"

namespace hb {
namespace {

constexpr int kLanesWarps = 8;
constexpr int kLanesStages = 2;     // raw chunks in flight per warp

// Dynamic shared memory of one CTA: per warp, kLanesStages raw chunks (32
// records each, AoS, filled by bulk copies) and one predicted chunk; then
// the warps' mbarriers.  After the j loop the front of it holds the warps'
// group sums.
template <int ORDER>
struct LanesSmem {
    static constexpr int raw = 32 * Rec<ORDER>::bytes;        // 3584 / 5120 / 6656
    static constexpr int pred = Pred64<ORDER>::ncomp * 32 * 8;
    static constexpr int warp = kLanesStages * raw + pred;
    static constexpr int bar_off = kLanesWarps * warp;
    static constexpr int bytes = bar_off + kLanesWarps * kLanesStages * 8;
    static_assert(raw % 16 == 0 && pred % 16 == 0, "bulk copies need 16-byte offsets");
    static_assert(bar_off >= kLanesWarps * kLanesMaxAct * Frc<ORDER>::words * 8, "reduction space");
};

// A lane's raw record from a chunk in shared memory, 16 bytes a load (records
// are 14, 20 or 26 words).  20-word records lie 160 bytes apart, so lanes l and
// l + 4 of a quarter warp meet in the same banks: lanes 4..7 take every two
// loads in the other order.  Loading word by word cost 160 shared-memory cycles a
// 6th-order chunk; this costs 40.
template <int ORDER>
__device__ __forceinline__ void load_record(const double *raw, int lane, double *r)
{
    constexpr int R = Rec<ORDER>::words;
    static_assert(R % 2 == 0, "16-byte records");
    const double2 *p = reinterpret_cast<const double2 *>(raw + lane * R);
    if constexpr (R % 4 == 0) {
        const int swap = (lane >> 2) & 1;
#pragma unroll
        for (int k = 0; k < R / 2; k += 2) {
            const double2 a = p[k + swap], b = p[k + 1 - swap];
            r[2 * k] = swap ? b.x : a.x;
            r[2 * k + 1] = swap ? b.y : a.y;
            r[2 * k + 2] = swap ? a.x : b.x;
            r[2 * k + 3] = swap ? a.y : b.y;
        }
    } else {
#pragma unroll
        for (int k = 0; k < R / 2; ++k) {
            const double2 a = p[k];
            r[2 * k] = a.x;
            r[2 * k + 1] = a.y;
        }
    }
}

template <int ORDER>
__device__ __forceinline__ void predict_lane(const double *raw, int chunk, int nbody, double tsys,
                                             Body64 &b)
{
    const int lane = threadIdx.x & 31, slot = chunk * 32 + lane;
    if (slot < nbody) {
        double r[Rec<ORDER>::words];
        load_record<ORDER>(raw, lane, r);
        predict_slot<ORDER>(r, tsys, b.x, b.v, b.a, b.jk);
        b.m = r[3];
    } else {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            b.x[k] = pad_position(slot, k);
            b.v[k] = b.a[k] = b.jk[k] = 0.0;
        }
        b.m = 0.0;
    }
}

// Predicts the 32 slots of chunk `chunk` (one per lane) from their raw
// records in shared memory into the predicted FP64 chunk layout at dst.  Out
// of line: the i-particles come from the same code, so a particle's i- and
// j-states are bit-identical and its self term is exactly zero.
template <int ORDER>
__device__ __noinline__ void predict_raw_chunk(const double *raw, int chunk, int nbody,
                                               double tsys, double *dst)
{
    const int lane = threadIdx.x & 31;
    Body64 b;
    predict_lane<ORDER>(raw, chunk, nbody, tsys, b);
    double *c = dst + lane;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        c[(P64_X + k) * 32] = b.x[k];
        c[(P64_V + k) * 32] = b.v[k];
        if constexpr (ORDER >= 6) c[(P64_A + k) * 32] = b.a[k];
        if constexpr (ORDER >= 8) c[(P64_J + k) * 32] = b.jk[k];
    }
    c[P64_M * 32] = b.m;
}

__device__ __forceinline__ double from_lane0(double v) { return __shfl_sync(0xffffffffu, v, 0); }

template <int ORDER, int LOG2G>
__global__ void __launch_bounds__(kLanesWarps * 32)
force_lanes_kernel(ForceArgs a)
{
    using L = LanesSmem<ORDER>;
    constexpr int G = 1 << LOG2G, STG = kLanesStages;
    constexpr int F = Frc<ORDER>::words, R = Rec<ORDER>::words;
    pdl_enter();
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int s_fail;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int p = lane >> LOG2G, g = lane & (G - 1);
    const int S = gridDim.x, sl = blockIdx.x, nact = a.nact;
    unsigned char *wraw = smem + w * L::warp;                            // this warp's raw stages
    double *my = reinterpret_cast<double *>(wraw + STG * L::raw);        // its predicted chunk
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem + L::bar_off) + w * STG;

    if (tid == 0) s_fail = 0;
    if (lane == 0) {
#pragma unroll
        for (int st = 0; st < STG; ++st) mbar_init(&bar[st], 1);
        fence_mbar_init();
    }
    __syncthreads();

    // This warp's loads: chunk 0 (the i-particles are its first nact slots),
    // then chunks c0 + w, c0 + w + kLanesWarps, ... of the CTA's j-slice.
    const int c0 = (int)((long long)sl * a.nchunk / S);
    const int c1 = (int)((long long)(sl + 1) * a.nchunk / S);
    const int nload = 1 + (c0 + w < c1 ? (c1 - c0 - w + kLanesWarps - 1) / kLanesWarps : 0);
    auto chunk_of = [&](int q) { return q == 0 ? 0 : c0 + w + (q - 1) * kLanesWarps; };
    auto issue = [&](int q) {   // lane 0 only
        const int st = q % STG;
        mbar_arrive_expect_tx(&bar[st], (uint32_t)L::raw);
        bulk_load(wraw + st * L::raw, a.jp + (size_t)chunk_of(q) * 32 * R, (uint32_t)L::raw, &bar[st]);
    };
    if (lane == 0)
        for (int q = 0; q < STG && q < nload; ++q) issue(q);

    Body64 I;
    double f[F];
#pragma unroll
    for (int q = 0; q < F; ++q) f[q] = 0.0;
    int failed_at = -1;
    for (int q = 0; q < nload; ++q) {
        const int st = q % STG;
        const bool got = mbar_wait_bounded(&bar[st], (uint32_t)((q / STG) & 1), a.spin);
        if (!__all_sync(0xffffffffu, got)) { failed_at = q; break; }
        if constexpr (LOG2G == 5) {
            // one i-particle: every lane keeps the j it predicts in registers;
            // this one copy of the code serves i (chunk 0, lane 0) and j
            Body64 J;
            predict_lane<ORDER>(reinterpret_cast<const double *>(wraw + st * L::raw), chunk_of(q),
                                a.nbody, a.tsys, J);
            __syncwarp();                // the raw stage is read: refill it
            if (lane == 0 && q + STG < nload) issue(q + STG);
            if (q == 0) {
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    I.x[k] = from_lane0(J.x[k]);
                    I.v[k] = from_lane0(J.v[k]);
                    if constexpr (ORDER >= 6) I.a[k] = from_lane0(J.a[k]);
                    if constexpr (ORDER >= 8) I.jk[k] = from_lane0(J.jk[k]);
                }
            } else {
                interact64<ORDER>(I, J, a.eps2, f);
            }
            continue;
        }
        predict_raw_chunk<ORDER>(reinterpret_cast<const double *>(wraw + st * L::raw), chunk_of(q),
                                 a.nbody, a.tsys, my);
        __syncwarp();                    // the raw stage is read: refill it
        if (lane == 0 && q + STG < nload) issue(q + STG);
        if (q == 0)
            load_i64<ORDER>(my, 0, min(p, nact - 1), I);   // lanes of groups p >= nact: a copy
        else
            chunk64_lanes<ORDER, LOG2G>(my, I, a.eps2, f);
        __syncwarp();                    // `my` is read: the next prediction may overwrite it
    }
    if (failed_at >= 0) {
        // leave no bulk copy writing into shared memory after this CTA ends
        if (lane == 0) {
            for (int q = failed_at; q < nload && q < failed_at + STG; ++q)
                mbar_wait_bounded(&bar[q % STG], (uint32_t)((q / STG) & 1));
            atomicOr(&s_fail, 1);
        }
    }
    __syncthreads();
    if (s_fail) {
        if (tid == 0) raise_error(a.err, kErrWaitTimeout);
        return;
    }
    // the G lanes of a group: a fixed butterfly
#pragma unroll
    for (int o = G >> 1; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q < F; ++q) f[q] += __shfl_xor_sync(0xffffffffu, f[q], o);
    double *red = reinterpret_cast<double *>(smem);          // [warp][i][F]
    if (g == 0 && p < nact)
#pragma unroll
        for (int q = 0; q < F; ++q) red[(w * kLanesMaxAct + p) * F + q] = f[q];
    __syncthreads();

    const int V = nact * F;
    for (int e = tid; e < V; e += blockDim.x) {
        double v = red[e];
#pragma unroll
        for (int ww = 1; ww < kLanesWarps; ++ww) v += red[ww * kLanesMaxAct * F + e];
        if (S == 1) a.force[e] = v;
        else a.partial[(size_t)sl * kLanesMaxAct * F + e] = v;
    }
}

}  // namespace

namespace {

using LanesKernel = void (*)(ForceArgs);
const LanesKernel kLanesTable[3][5] = {   // groups of G = 2..32 lanes
    {force_lanes_kernel<4, 1>, force_lanes_kernel<4, 2>, force_lanes_kernel<4, 3>,
     force_lanes_kernel<4, 4>, force_lanes_kernel<4, 5>},
    {force_lanes_kernel<6, 1>, force_lanes_kernel<6, 2>, force_lanes_kernel<6, 3>,
     force_lanes_kernel<6, 4>, force_lanes_kernel<6, 5>},
    {force_lanes_kernel<8, 1>, force_lanes_kernel<8, 2>, force_lanes_kernel<8, 3>,
     force_lanes_kernel<8, 4>, force_lanes_kernel<8, 5>}};
constexpr int kLanesBytes[3] = {LanesSmem<4>::bytes, LanesSmem<6>::bytes, LanesSmem<8>::bytes};

// Per device (up to 64): the kernels' shared-memory attribute set once, and
// the resident CTAs per SM of each order.
std::mutex g_lanes_mu;
unsigned long long g_lanes_ready = 0;
int g_lanes_per_sm[64][3];

cudaError_t lanes_setup(int oi, int *per_sm)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lk(g_lanes_mu);
    if (!(g_lanes_ready >> dev & 1ull)) {
        for (int o = 0; o < 3; ++o) {
            for (int v = 0; v < 5; ++v) {
                e = cudaFuncSetAttribute(kLanesTable[o][v], cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         kLanesBytes[o]);
                if (e != cudaSuccess) return e;
            }
            int nb = 0;
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kLanesTable[o][4], kLanesWarps * 32,
                                                              kLanesBytes[o]);
            if (e != cudaSuccess) return e;
            g_lanes_per_sm[dev][o] = std::max(1, nb);
        }
        g_lanes_ready |= 1ull << dev;
    }
    *per_sm = g_lanes_per_sm[dev][oi];
    return cudaSuccess;
}

}  // namespace

cudaError_t launch_force_lanes(int order, const ForceArgs &a, int nsm, cudaStream_t s, int *launches)
{
    static_assert(kLanesMaxAct <= 16, "one lane per i-particle is the tiled kernel's job");
    if (a.nact < 1 || a.nact > kLanesMaxAct || a.nchunk < 1) return cudaErrorInvalidValue;
    const int oi = order == 4 ? 0 : order == 6 ? 1 : order == 8 ? 2 : -1;
    if (oi < 0) return cudaErrorInvalidValue;
    int per_sm = 1;
    cudaError_t e = lanes_setup(oi, &per_sm);
    if (e != cudaSuccess) return e;
    const int log2g = lanes_log2g(a.nact);                // P = 2^(5 - log2g) >= nact, G >= 2
    // j-slices of at least two chunks a warp, all CTAs resident at once
    const int S = std::max(1, std::min(std::min(2, per_sm) * nsm, a.nchunk / (2 * kLanesWarps)));
    const int F = 3 * (order / 2);
    e = launch_pdl(kLanesTable[oi][log2g - 1], dim3(S), kLanesWarps * 32, kLanesBytes[oi], s, a);
    if (e != cudaSuccess) return e;
    ++*launches;
    if (S == 1) return cudaSuccess;
    ++*launches;
    return launch_reduce(a.partial, (size_t)kLanesMaxAct * F, S, a.nact * F, a.force, s);
}

}  // namespace hb
