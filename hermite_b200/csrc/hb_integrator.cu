// hb_integrator.cu -- block-timestep Hermite integration resident on the GPU.
//
// The reference integrates on the host: per block step NbodySystem finds the
// next block time and the active set (calc_dtlim / count_nact over a
// dt-sorted array, SRC/nbodysystem.h:652-690), calls the force calculator,
// corrects the active particles and re-sorts them (:693-765).  Here the whole
// step stays on the device, three phases per step, replayed from a captured
// CUDA graph (no host round trip per step):
//   1. active set       = slots with tlast + dt == the next block time
//                         (compaction), dtlim from it (calc_dtlim), and every
//                         slot predicted to it
//   2. force            = active set against the predicted slots, work items
//                         (i-tile, j-slice) sized on the device from nact
//   3. corrector        = sum of the slices, Particle::correct + quantised
//                         Aarseth dt, and the minimum of tlast + dt over all
//                         slots: the next block time
// Slots are never re-sorted; the j summation order is the slot order.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>

#include "hermite_b200.h"
#include "hb_common.cuh"
#include "hb_corrector.cuh"
#include "hb_force.cuh"
#include "hb_internal.h"

namespace hb {

constexpr unsigned long long kInfBits = 0x7ff0000000000000ull;   // +inf
constexpr int kStepThreads = 128;       // CTAs of the first two phases
constexpr int kCorrectThreads = 256;    // and of the third (graph engine)

struct StepArgs {
    double *jp, *dt, *tn, *aux;   // records; per slot dt, tlast + dt, dump derivatives
    void *pred;                   // predicted slots, AoSoA32
    int *ilist;
    Sched *s;
    double *force;                // [nact][F], indexed by position in ilist (one slice)
    double *partial;              // [S][gx*ti][F]
    int *err;
    int n, nchunk;
    size_t partial_cap;
    int resident;                 // nominal CTAs of the force phase at once
};

// The work split of a step with nact active slots: wj warps of a CTA's four
// share an i-group of 32 (ti = 128 / wj particles per i-tile), S j-slices.
// Thin tiles and slices where the pairs are few, so that a step of a few
// particles still fills the GPU; slices of about 8 waves of CTAs for large
// steps, which evens out CTAs that do not end together.  A slice of the thin
// shape has 4 to 16 chunks, one to four per warp in turn (0.7 us each); with
// more slices the sum in the corrector grows.  The bounds are flat: halving or
// doubling any of them moves the mean step by at most 3 % (N = 2500 ... 131072,
// 4th to 8th order); slices of one chunk, a quarter of it per warp, measured 1 us
// slower at N = 512 ... 8192 (the sum grows by more than the chain shrinks).
//
// Per block step, 4th order, N = 4096 / 16384 / 65536: 12.6 / 25.6 / 112 us, from
// 18.4 / 34.0 / 125 us with five kernels, raw records predicted by every item and
// the last CTA of an i-tile adding its slices.
struct StepSplit {
    int wj, ti, gx, S;
};
template <int F>
__device__ __forceinline__ StepSplit step_split(int nact, const StepArgs &a)
{
    StepSplit r;
    const long long units = (long long)((nact + 63) / 64) * a.nchunk;
    r.wj = nact <= 64 || units <= 32768 ? 4 : nact < 4096 ? 2 : 1;
    r.ti = 128 / r.wj;
    r.gx = (nact + r.ti - 1) / r.ti;
    const float x = (float)r.gx * (float)a.nchunk / (float)a.resident;    // chunks per resident CTA
    int c = r.wj == 4 ? 4 * max(1, min(4, (int)fmaxf(sqrtf(x), a.nchunk / 1024.0f))) : 8;
    c = max(c, (int)(x * 0.125f));
    r.S = max(1, a.nchunk / c);
    const size_t row = (size_t)r.gx * r.ti * F;
    if (r.S * row > a.partial_cap) r.S = (int)max((size_t)1, a.partial_cap / row);
    return r;
}

// Before a run's first step: tlast + dt per slot, their minimum, counters.
__global__ void step_reset_kernel(Sched *s)
{
    s->next_bits = kInfBits;
    s->nact[0] = s->nact[1] = 0;
}

template <int ORDER>
__global__ void step_start_kernel(StepArgs a)
{
    constexpr int R = Rec<ORDER>::words;
    double m = __longlong_as_double((long long)kInfBits);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += gridDim.x * blockDim.x) {
        const double t = a.dt[i] + a.jp[(size_t)i * R + 7];
        a.tn[i] = t;
        m = fmin(m, t);
    }
    for (int o = 16; o; o >>= 1) m = fmin(m, __shfl_xor_sync(0xffffffffu, m, o));
    // positive doubles order like their bit patterns
    if ((threadIdx.x & 31) == 0) atomicMin(&a.s->next_bits, (unsigned long long)__double_as_longlong(m));
}

// Phase 1: active set, dtlim and prediction.  Returns whether the step is live
// (its time within tend and no error): the same answer in every thread of the
// grid.  Steps alternate between two active counters (par), so that the
// counter of the next step is cleared while nobody reads it.
template <int ORDER, bool MIXED>
__device__ __forceinline__ bool active_phase(const StepArgs &a, int par)
{
    constexpr int R = Rec<ORDER>::words;
    Sched *s = a.s;
    const double tnext = __longlong_as_double((long long)s->next_bits);
    const bool live = tnext <= s->tend && s->error == 0;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        s->tnext = tnext;
        s->dtlim = calc_dtlim(tnext, s->dtmax);
        s->work = 0;
        if (!live) s->nact[0] = s->nact[1] = 0;   // the later phases do nothing
    }
    if (!live) return false;
    for (int base = blockIdx.x * kStepThreads; base < a.nchunk * 32; base += gridDim.x * kStepThreads) {
        const int i = base + threadIdx.x;
        double x[3], v[3], ac[3] = {0, 0, 0}, jk[3] = {0, 0, 0}, xl[3] = {0, 0, 0}, m;
        bool act = false;
        if (i < a.n) {
            const double *r = a.jp + (size_t)i * R;
            double q[R];
            if constexpr (R % 2 == 0) {
#pragma unroll
                for (int k = 0; k < R; k += 2) {
                    const double2 d = *reinterpret_cast<const double2 *>(r + k);
                    q[k] = d.x;
                    q[k + 1] = d.y;
                }
            } else {
#pragma unroll
                for (int k = 0; k < R; ++k) q[k] = r[k];
            }
            act = a.tn[i] == tnext;
            predict_slot<ORDER>(q, tnext, x, v, ac, jk, xl);
            m = q[3];
        } else {
#pragma unroll
            for (int k = 0; k < 3; ++k) { x[k] = pad_position(i, k); v[k] = 0.0; }
            m = 0.0;
        }
        unsigned char *chunk = static_cast<unsigned char *>(a.pred) +
                               (size_t)(i >> 5) * Layout<ORDER, MIXED>::chunk_bytes;
        put_predicted<ORDER, MIXED>(chunk + (i & 31) * (MIXED ? 4 : 8), x, v, ac, jk, xl, m);
        const unsigned ballot = __ballot_sync(0xffffffffu, act);
        int off = 0;
        if ((threadIdx.x & 31) == 0 && ballot) off = atomicAdd(&s->nact[par], __popc(ballot));
        off = __shfl_sync(0xffffffffu, off, 0);
        if (act) a.ilist[off + __popc(ballot & ((1u << (threadIdx.x & 31)) - 1u))] = i;
    }
    return true;
}

template <int ORDER, bool MIXED>
__global__ void __launch_bounds__(kStepThreads) step_active_kernel(StepArgs a, int par)
{
    pdl_enter();
    active_phase<ORDER, MIXED>(a, par);
}

// Phase 2: the pair sums of the step's work items, taken by this CTA until
// none are left (the first by block index, the rest from a device counter).
template <int ORDER, bool MIXED>
struct StepShape {
    static constexpr int NW = kStepThreads / 32, TCH = 4, STG = 2;
    static constexpr int F = Frc<ORDER>::words, CB = Layout<ORDER, MIXED>::chunk_bytes;
    static constexpr int tile_bytes = TCH * CB, ring_bytes = STG * tile_bytes;
    static constexpr int red_bytes = (NW - 1) * F * 32 * 8;
    static constexpr int body_bytes = ring_bytes > red_bytes ? ring_bytes : red_bytes;
    static constexpr int smem_bytes = body_bytes + 64;   // + mbarriers
};

// bar: two initialised mbarriers whose phases continue from g (tiles issued by
// this CTA before).  Returns false when a wait gave up (the error is raised, the
// CTA's copies drained).
template <int ORDER, bool MIXED>
__device__ __forceinline__ bool force_phase(const StepArgs &a, int par, unsigned char *smem,
                                            uint64_t *bar, unsigned &g)
{
    using Sh = StepShape<ORDER, MIXED>;
    constexpr int TCH = Sh::TCH, STG = Sh::STG, F = Sh::F, CB = Sh::CB;
    constexpr int NCOMP = Layout<ORDER, MIXED>::ncomp;
    __shared__ int s_item;
    Sched *s = a.s;
    const int nact = s->nact[par];
    if (nact == 0) return true;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        s->nact[1 - par] = 0;
        s->next_bits = kInfBits;
    }
    const StepSplit sp = step_split<F>(nact, a);
    const double eps2 = s->eps2;
    const float2 eps2f = f2((float)eps2);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ig = warp / sp.wj, jg = warp % sp.wj;
    const int items = sp.gx * sp.S;
    const int len = a.nchunk / sp.S, rem = a.nchunk % sp.S;     // chunks of a slice, one more in the first rem
    const size_t ispan = (size_t)sp.gx * sp.ti;
    double *out = sp.S == 1 ? a.force : a.partial;
    // FP64 steps of at most kLanesMaxAct active slots: lanes share an
    // i-particle and split each chunk's j (lanes_log2g, hb_force.cuh)
    constexpr bool kLaneSplit = !MIXED && ORDER != 9;
    const int lg = kLaneSplit && nact <= kLanesMaxAct ? lanes_log2g(nact) : 0;

    for (int item = blockIdx.x; item < items;) {
        const int itile = item / sp.S, sl = item % sp.S;
        const int c0 = sl * len + min(sl, rem), c1 = c0 + len + (sl < rem ? 1 : 0);
        const int ntile = (c1 - c0 + TCH - 1) / TCH;
        auto issue = [&](int t) {   // thread 0 only
            const unsigned gt = g + t;
            const int st = gt % STG;
            const int cs = c0 + t * TCH, cnt = min(TCH, c1 - cs);
            const uint32_t bytes = (uint32_t)(cnt * CB);
            mbar_arrive_expect_tx(&bar[st], bytes);
            bulk_load(smem + st * Sh::tile_bytes, static_cast<const unsigned char *>(a.pred) + (size_t)cs * CB,
                      bytes, &bar[st]);
        };
        if (tid == 0)
            for (int t = 0; t < STG && t < ntile; ++t) issue(t);

        // this lane's i-particle, from the predicted slots
        const int row = ig * 32 + (lg ? min(lane >> lg, nact - 1) : lane);
        const int slot = a.ilist[min(itile * sp.ti + row, nact - 1)];
        using IBody = typename std::conditional<MIXED, NegI32, Body64>::type;
        IBody I[1];
        if constexpr (MIXED)
            load_i_mixed<ORDER>(static_cast<const float *>(a.pred) + (size_t)(slot >> 5) * NCOMP * 32, 0, slot & 31, I[0]);
        else
            load_i64<ORDER>(static_cast<const double *>(a.pred) + (size_t)(slot >> 5) * NCOMP * 32, 0, slot & 31, I[0]);

        double f[1][F], tot[1][F], cmp[1][F];   // 8th order FP64: per-tile sums, Kahan-folded
#pragma unroll
        for (int c = 0; c < F; ++c) f[0][c] = tot[0][c] = cmp[0][c] = 0.0;
        int failed_at = -1;
        for (int t = 0; t < ntile; ++t) {
            const unsigned gt = g + t;
            const int st = gt % STG;
            const bool got = mbar_wait_bounded(&bar[st], (gt / STG) & 1u);
            if (!__syncthreads_and(got)) { failed_at = t; break; }
            const int cnt = min(TCH, c1 - (c0 + t * TCH));
            const unsigned char *tile = smem + st * Sh::tile_bytes;
            for (int q = jg; q < cnt; q += sp.wj) {
                if constexpr (MIXED) {
                    chunk_mixed<ORDER, 1, (HB_MIXED_REFINE != 0)>(reinterpret_cast<const float *>(tile + q * CB), I, eps2f, f);
                } else {
                    if (kLaneSplit && lg)
                        chunk64_lanes<ORDER>(lg, reinterpret_cast<const double *>(tile + q * CB), I[0], eps2, f[0]);
                    else
                        chunk64<ORDER, 1>(reinterpret_cast<const double *>(tile + q * CB), I, eps2, f);
                }
            }
            if constexpr (kKahan<ORDER, MIXED>) kahan_fold<1, F>(tot, cmp, f);
            __syncthreads();
            if (tid == 0 && t + STG < ntile) issue(t + STG);
        }
        if (failed_at >= 0) {
            if (tid == 0) {
                raise_error(a.err, kErrWaitTimeout);
                for (int t = failed_at; t < ntile && t < failed_at + STG; ++t)
                    mbar_wait_bounded(&bar[(g + t) % STG], ((g + t) / STG) & 1u);
            }
            s->error = 2;
            return false;
        }
        g += ntile;
        if constexpr (kKahan<ORDER, MIXED>) {
#pragma unroll
            for (int c = 0; c < F; ++c) f[0][c] = __dsub_rn(tot[0][c], cmp[0][c]);
        }
        if (kLaneSplit && lg) lanes_gather<F>(lg, f[0]);

        // the wj warps of an i-group, in warp order
        double *red = reinterpret_cast<double *>(smem);
        if (jg > 0)
#pragma unroll
            for (int c = 0; c < F; ++c) red[((warp - ig - 1) * F + c) * 32 + lane] = f[0][c];
        if (tid == 0) s_item = gridDim.x + atomicAdd(&s->work, 1);
        __syncthreads();
        item = s_item;
        if (jg == 0) {
            // warps ig * wj + 1 ... of the group hold rows ig * (wj - 1) ... of red
            for (int w = 0; w < sp.wj - 1; ++w)
#pragma unroll
                for (int c = 0; c < F; ++c) f[0][c] += red[((ig * (sp.wj - 1) + w) * F + c) * 32 + lane];
            double *o = out + (size_t)sl * ispan * F + (size_t)(itile * sp.ti + ig * 32 + lane) * F;
            if (sp.S > 1 || itile * sp.ti + ig * 32 + lane < nact)
#pragma unroll
                for (int c = 0; c < F; ++c) o[c] = f[0][c];
        }
        __syncthreads();
    }
    return true;
}

template <int ORDER, bool MIXED>
__global__ void __launch_bounds__(kStepThreads, 4) step_force_kernel(StepArgs a, int par)
{
    pdl_wait();
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem + StepShape<ORDER, MIXED>::body_bytes);
    if (threadIdx.x == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        fence_mbar_init();
    }
    __syncthreads();
    unsigned g = 0;   // tiles issued by this CTA so far (mbarrier phases)
    force_phase<ORDER, MIXED>(a, par, smem, bar, g);
    // not before the items are taken: the corrector's waiting CTAs would hold
    // registers that this kernel's need (2-3 % of the mean step at N = 65536)
    pdl_launch_next();
}

// What the host reads between replays.  A step's end would wait for the writes
// to cross the host link, so only the last step of a replay reports.
__device__ __forceinline__ void report_status(const Sched *s)
{
    IntStatus *st = s->status;
    st->tsys = s->tsys;
    st->particle_steps = s->particle_steps;
    st->block_steps = s->block_steps;
    st->error = s->error;
}

// Phase 3: slices summed, corrector, and the next block time.  L lanes (a
// power of two covering S, at most 32) add a particle's slices, lane l taking
// l, l + L, ..., and meet in a fixed butterfly: the association depends on S
// alone, not on the particle's place in the active list, which the compaction
// does not fix.
template <int ORDER>
__device__ __forceinline__ void correct_phase(const StepArgs &a, int par, bool report)
{
    constexpr int R = Rec<ORDER>::words, F = Frc<ORDER>::words;
    Sched *s = a.s;
    const int nact = s->nact[par], nt = blockDim.x, lane = threadIdx.x & 31;
    if (nact > 0) {
        const double tnext = s->tnext, dtlim = s->dtlim, etapow = s->etapow;
        const StepSplit sp = step_split<F>(nact, a);
        const size_t stride = (size_t)sp.gx * sp.ti * F;
        // every slot's time: those not corrected here as they stand (one
        // corrected meanwhile by another CTA counts with its new time, twice)
        double m = __longlong_as_double((long long)kInfBits);
        for (int i = blockIdx.x * nt + threadIdx.x; i < a.n; i += gridDim.x * nt) {
            const double t = a.tn[i];
            if (t != tnext) m = fmin(m, t);
        }
        int lb = 0;
        while ((1 << lb) < sp.S && lb < 5) ++lb;
        const int L = 1 << lb, l = lane & (L - 1), per = nt >> lb;
        // with 8 lanes and more, they also fetch the record (beside the slices,
        // not after them) and write it back
        constexpr int kRecs = kCorrectThreads / 8;
        __shared__ double rec[kRecs * R];
        const bool staged = L >= 8;
        for (int k0 = blockIdx.x * per; k0 < nact; k0 += gridDim.x * per) {
            const int k = k0 + (threadIdx.x >> lb);
            double *mine = rec + (staged ? (threadIdx.x >> lb) * R : 0);
            double f[F], dt = 0.0;
            int i = 0;
#pragma unroll
            for (int c = 0; c < F; ++c) f[c] = 0.0;
            if (k < nact) {
                i = a.ilist[k];
                dt = a.dt[i];
                if (staged)
                    for (int w = l; w < R; w += L) mine[w] = a.jp[(size_t)i * R + w];
                if (sp.S == 1) {
#pragma unroll
                    for (int c = 0; c < F; ++c) f[c] = a.force[(size_t)k * F + c];
                } else {
                    const double *p = a.partial + (size_t)k * F;
#pragma unroll 4
                    for (int sl = l; sl < sp.S; sl += L)
#pragma unroll
                        for (int c = 0; c < F; ++c) f[c] += __ldcg(p + (size_t)sl * stride + c);
                }
            }
            for (int o = L >> 1; o; o >>= 1)
#pragma unroll
                for (int c = 0; c < F; ++c) f[c] += __shfl_xor_sync(0xffffffffu, f[c], o);
            __syncwarp();
            if (k < nact && l == 0) {
                double *r = staged ? mine : a.jp + (size_t)i * R;
                const double dtn = correct_particle<ORDER>(r, f, dt, etapow, dtlim,
                                                           a.aux + (size_t)i * kAuxWords);
                if (!(dtn >= 0x1p-48)) s->error = 1;   // timestep underflow (or NaN)
                const double t = dtn + r[7];
                a.dt[i] = dtn;
                a.tn[i] = t;
                m = fmin(m, t);
            }
            __syncwarp();
            if (staged && k < nact)
                for (int w = l; w < R; w += L) a.jp[(size_t)i * R + w] = mine[w];
            __syncwarp();
        }
        for (int o = 16; o; o >>= 1) m = fmin(m, __shfl_xor_sync(0xffffffffu, m, o));
        __shared__ double wm[kCorrectThreads / 32];
        if (lane == 0) wm[threadIdx.x >> 5] = m;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 1; w < nt / 32; ++w) m = fmin(m, wm[w]);
            atomicMin(&s->next_bits, (unsigned long long)__double_as_longlong(m));
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (nact > 0) {
            s->tsys = s->tnext;
            s->particle_steps += nact;
            s->block_steps += 1;
        }
        if (report) report_status(s);
    }
}

template <int ORDER>
__global__ void __launch_bounds__(kCorrectThreads) step_correct_kernel(StepArgs a, int par, int report)
{
    pdl_enter();
    correct_phase<ORDER>(a, par, report != 0);
}

// ---------------------------------------------------------------------------
// Persistent engine: the three phases of a block step in one cooperative
// kernel, its CTAs all resident, separated by grid barriers in place of kernel
// boundaries; up to max_steps steps per launch.  The phases are the graph
// engine's own code, and the force phase takes the same work items (the same
// nominal grid), so both engines give the same block steps and records bit for bit.
struct PersistArgs {
    StepArgs a;
    unsigned *gbar;          // grid barrier: [0] arrivals, [1] generation
    long long max_steps;
    unsigned spin;           // poll limit of one barrier wait
};

// Barrier over a co-resident grid.  Thread 0 of each CTA reads the generation
// word, then arrives on the counter (acquire-release); the last CTA to arrive
// resets the counter and advances the generation (release), which the others
// poll (acquire).  The CTA barriers on both sides carry the ordering to the
// CTA's other threads, so every write made before the barrier anywhere in the
// grid is visible to every read after it, the bulk copies that thread 0
// issues included (proxy fences).  A wait is bounded: after `spin` polls the CTA reports false (the
// caller raises the error and returns; the other CTAs then give up at their
// next barrier).
__device__ __forceinline__ unsigned ld_relaxed_gpu(const unsigned *p)
{
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned ld_acquire_gpu(const unsigned *p)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void fence_proxy_async_global()
{
    asm volatile("fence.proxy.async.global;" ::: "memory");
}

__device__ __forceinline__ bool grid_barrier(unsigned *gbar, unsigned spin)
{
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        // The phases read records with bulk copies (async proxy) that other
        // CTAs wrote with ordinary stores (generic proxy): proxy fences on
        // both sides of the barrier order the two.
        fence_proxy_async_global();
        const unsigned my = ld_relaxed_gpu(gbar + 1);
        unsigned old;
        asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;"
                     : "=r"(old) : "l"(gbar) : "memory");
        int ok = 1;
        if (old == gridDim.x - 1) {
            asm volatile("st.relaxed.gpu.global.u32 [%0], 0;" :: "l"(gbar) : "memory");
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" :: "l"(gbar + 1) : "memory");
        } else {
            ok = 0;
            for (unsigned it = 0; it < spin; ++it) {
                if (ld_acquire_gpu(gbar + 1) != my) {
                    ok = 1;
                    break;
                }
                __nanosleep(64);
            }
        }
        fence_proxy_async_global();
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

template <int ORDER, bool MIXED>
__global__ void __launch_bounds__(kStepThreads, 4)
persistent_kernel(PersistArgs p)
{
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem + StepShape<ORDER, MIXED>::body_bytes);
    const StepArgs &a = p.a;
    Sched *s = a.s;
    if (threadIdx.x == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        fence_mbar_init();
    }
    __syncthreads();
    unsigned g = 0;   // tiles issued by this CTA so far (mbarrier phases)
    bool gave_up = false;
    for (long long k = 0; k < p.max_steps && !gave_up; ++k) {
        // an even number of steps per launch: the counters' turn starts over
        const int par = (int)(k & 1);
        const bool live = active_phase<ORDER, MIXED>(a, par);
        if (!grid_barrier(p.gbar, p.spin)) { gave_up = true; break; }
        if (!live) break;                // every CTA reads the same state
        if (!force_phase<ORDER, MIXED>(a, par, smem, bar, g))
            return;                      // raised; the others give up at the next barrier
        if (!grid_barrier(p.gbar, p.spin)) { gave_up = true; break; }
        correct_phase<ORDER>(a, par, false);
        if (!grid_barrier(p.gbar, p.spin)) { gave_up = true; break; }
    }
    if (!gave_up && blockIdx.x == 0 && threadIdx.x == 0) report_status(s);
    if (gave_up && threadIdx.x == 0) {   // a barrier wait gave up
        s->error = 2;
        raise_error(a.err, kErrWaitTimeout);
    }
}

// Initialisation: write the force of all slots into the records (assign_force)
// and, on the last pass, the initial dt (init_dt).
template <int ORDER>
__global__ void assign_kernel(double *__restrict__ jp, double *__restrict__ dt,
                              const double *__restrict__ force, int n, int set_dt, double eta_s,
                              double dtmax)
{
    constexpr int R = Rec<ORDER>::words, F = Frc<ORDER>::words;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double *r = jp + (size_t)i * R;
    const double *f = force + (size_t)i * F;
    for (int c = 0; c < F; ++c) r[8 + c] = f[c];
    if (set_dt) dt[i] = initial_dt<ORDER>(f, eta_s, dtmax);
}

// 0.5*sum m v^2 and 0.5*sum m phi, per-block partials then one block, in a
// fixed order.
template <int ORDER>
__global__ void energy_partial_kernel(const double *__restrict__ jp, const double *__restrict__ pot,
                                      int n, double *__restrict__ part)
{
    constexpr int R = Rec<ORDER>::words;
    double ke = 0.0, pe = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double *r = jp + (size_t)i * R;
        ke += r[3] * (r[4] * r[4] + r[5] * r[5] + r[6] * r[6]);
        pe += r[3] * pot[i];
    }
    __shared__ double sk[256], sp[256];
    sk[threadIdx.x] = ke;
    sp[threadIdx.x] = pe;
    __syncthreads();
    for (int o = blockDim.x / 2; o; o >>= 1) {
        if (threadIdx.x < o) {
            sk[threadIdx.x] += sk[threadIdx.x + o];
            sp[threadIdx.x] += sp[threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = sk[0];
        part[2 * blockIdx.x + 1] = sp[0];
    }
}

__global__ void energy_final_kernel(const double *part, int nblk, double *out)
{
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        double ke = 0.0, pe = 0.0;
        for (int b = 0; b < nblk; ++b) {
            ke += part[2 * b];
            pe += part[2 * b + 1];
        }
        out[0] = 0.5 * ke;
        out[1] = 0.5 * pe;
    }
}

constexpr int kEnergyBlocks = 256;

static StepArgs step_args(const IntegratorLaunch &L)
{
    return StepArgs{L.jp, L.dt, L.tn, L.aux, L.pred, L.ilist, L.sched, L.force, L.partial, L.err,
                    L.n, L.nchunk, L.partial_cap, L.nsm * 4};
}

// One (order, precision) instance of the step's kernels.
template <int ORDER, bool MIXED>
struct StepKernels {
    static cudaError_t launch(const IntegratorLaunch &L, int par, bool report, cudaStream_t s)
    {
        const StepArgs a = step_args(L);
        const int nb = std::min(L.nchunk / 4, L.nsm * 16);       // 128 slots per CTA
        cudaError_t e = launch_pdl(step_active_kernel<ORDER, MIXED>, dim3(nb), kStepThreads, 0, s, a, par);
        if (e == cudaSuccess)
            e = launch_pdl(step_force_kernel<ORDER, MIXED>, dim3(L.nsm * 4), kStepThreads,
                           StepShape<ORDER, MIXED>::smem_bytes, s, a, par);
        if (e == cudaSuccess)
            e = launch_pdl(step_correct_kernel<ORDER>, dim3(std::max(1, std::min(L.nchunk / 4, L.nsm * 2))),
                           kCorrectThreads, 0, s, a, par, report ? 1 : 0);
        return e;
    }
    static cudaError_t start(const IntegratorLaunch &L, cudaStream_t s)
    {
        step_reset_kernel<<<1, 1, 0, s>>>(L.sched);
        step_start_kernel<ORDER><<<std::min((L.n + 255) / 256, L.nsm * 8), 256, 0, s>>>(step_args(L));
        return cudaGetLastError();
    }
    static cudaError_t setup()
    {
        return cudaFuncSetAttribute(step_force_kernel<ORDER, MIXED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    StepShape<ORDER, MIXED>::smem_bytes);
    }
    static cudaError_t persistent_setup(int *per_sm)
    {
        const void *k = (const void *)&persistent_kernel<ORDER, MIXED>;
        const int smem = StepShape<ORDER, MIXED>::smem_bytes;
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, k, kStepThreads, smem);
        return e;
    }
    static cudaError_t persistent(const PersistArgs &p, int grid, cudaStream_t s)
    {
        PersistArgs arg = p;
        void *args[] = {&arg};
        return cudaLaunchCooperativeKernel((const void *)&persistent_kernel<ORDER, MIXED>, dim3(grid),
                                           dim3(kStepThreads), args,
                                           (size_t)StepShape<ORDER, MIXED>::smem_bytes, s);
    }
};

// Calls fn with the StepKernels of (order, precision); double-double positions
// (order 9) are FP64 only.
template <typename Fn>
static cudaError_t with_step(int order, bool mixed, Fn fn)
{
    switch (order * 2 + (mixed && order != 9 ? 1 : 0)) {
    case 8: return fn(StepKernels<4, false>());
    case 9: return fn(StepKernels<4, true>());
    case 12: return fn(StepKernels<6, false>());
    case 13: return fn(StepKernels<6, true>());
    case 16: return fn(StepKernels<8, false>());
    case 17: return fn(StepKernels<8, true>());
    case 18: return fn(StepKernels<9, false>());
    }
    return cudaErrorInvalidValue;
}

cudaError_t integrator_step_launch(int order, const IntegratorLaunch &L, int par, bool report, cudaStream_t s)
{
    return with_step(order, L.mixed, [&](auto k) { return decltype(k)::launch(L, par, report, s); });
}

cudaError_t integrator_start(int order, const IntegratorLaunch &L, cudaStream_t s)
{
    return with_step(order, L.mixed, [&](auto k) { return decltype(k)::start(L, s); });
}

cudaError_t integrator_kernel_setup(int order, bool mixed)
{
    return with_step(order, mixed, [&](auto k) { return decltype(k)::setup(); });
}

cudaError_t persistent_setup(int order, bool mixed, int *per_sm)
{
    return with_step(order, mixed, [&](auto k) { return decltype(k)::persistent_setup(per_sm); });
}

cudaError_t persistent_launch(int order, const IntegratorLaunch &L, unsigned *gbar,
                              long long max_steps, unsigned spin, int grid, cudaStream_t s)
{
    const PersistArgs p{step_args(L), gbar, max_steps, spin};
    return with_step(order, L.mixed, [&](auto k) { return decltype(k)::persistent(p, grid, s); });
}

cudaError_t integrator_assign(int order, double *jp, double *dt, const double *force, int n,
                              int set_dt, double eta_s, double dtmax, cudaStream_t s)
{
    const int g = (n + 127) / 128;
    switch (order) {
    case 4: assign_kernel<4><<<g, 128, 0, s>>>(jp, dt, force, n, set_dt, eta_s, dtmax); break;
    case 6: assign_kernel<6><<<g, 128, 0, s>>>(jp, dt, force, n, set_dt, eta_s, dtmax); break;
    case 8: assign_kernel<8><<<g, 128, 0, s>>>(jp, dt, force, n, set_dt, eta_s, dtmax); break;
    case 9: assign_kernel<9><<<g, 128, 0, s>>>(jp, dt, force, n, set_dt, eta_s, dtmax); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t integrator_energy(int order, const double *jp, const double *pot, int n, double *part,
                              double *out, cudaStream_t s)
{
    switch (order) {
    case 4: energy_partial_kernel<4><<<kEnergyBlocks, 256, 0, s>>>(jp, pot, n, part); break;
    case 6: energy_partial_kernel<6><<<kEnergyBlocks, 256, 0, s>>>(jp, pot, n, part); break;
    case 8: energy_partial_kernel<8><<<kEnergyBlocks, 256, 0, s>>>(jp, pot, n, part); break;
    case 9: energy_partial_kernel<9><<<kEnergyBlocks, 256, 0, s>>>(jp, pot, n, part); break;
    default: return cudaErrorInvalidValue;
    }
    energy_final_kernel<<<1, 32, 0, s>>>(part, kEnergyBlocks, out);
    return cudaGetLastError();
}

}  // namespace hb
