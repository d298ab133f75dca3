// hb_force_sym.cu -- launches of the each-pair-once FP64 force.
#include <algorithm>

#include "hb_force_sym.cuh"

namespace hb {
namespace {

template <int ORDER>
cudaError_t launch_t(const ForceArgs &f, size_t cap, int nsm, cudaStream_t s, int *launches)
{
    constexpr int F = Frc<ORDER>::words, GC = SymShape<ORDER>::GC;
    cudaError_t e = cudaFuncSetAttribute(force_sym_kernel<ORDER>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         SymShape<ORDER>::bytes);
    if (e != cudaSuccess) return e;
    SymArgs a{};
    a.pred = static_cast<const double *>(f.pred);
    a.force = f.force;
    a.nchunk = f.nchunk;
    a.nact = f.nact;
    a.ca = (f.nact + 31) / 32;
    a.eps2 = f.eps2;
    a.err = f.err;
    a.spin = f.spin;
    const int groups = (a.ca + GC - 1) / GC;
    const long long chunk = F * 32, room = (long long)(cap / chunk);   // scratch in [F][32] blocks
    for (int g0 = 0; g0 < groups; g0 += a.ng) {
        // as many groups as the scratch has rows and slice sums for, in slices
        // that make 10 to 20 waves of CTAs, in whole tiles: 20 as long as the slice
        // sums take no more than 0.4 of the rows' room (with 32 rows, 6th order, N =
        // 131072: 4 waves 41.7 ms, 6 40.5, 10 40.0; with 64, 10 39.7, 20 39.3; N =
        // 50000 5.92, 5.98)
        a.g0 = g0;
        a.ng = (int)std::min((long long)(groups - g0), room / a.ca);
        for (int pass = 0; pass < 3; ++pass) {
            if (a.ng < 1) return cudaErrorInvalidValue;
            const long long units = (long long)a.ng * (a.nchunk - (long long)g0 * GC) - (long long)GC * a.ng * (a.ng - 1) / 2;
            const long long wave = SymShape<ORDER>::MINB * nsm;
            const long long lc = std::min(units / (10 * wave),
                                          std::max(units / (20 * wave), 5LL * GC * a.nchunk / (2 * a.ca)));
            a.lc = (int)std::max(1LL, (lc + kSymFTile - 1) / kSymFTile) * kSymFTile;
            a.smax = sym_slices(a.nchunk, g0, GC, a.lc);
            a.ng = (int)std::min((long long)a.ng, room / (a.ca + (long long)a.smax * GC));
        }
        if (a.ng < 1) return cudaErrorInvalidValue;
        a.rows = f.partial;
        a.cols = f.partial + (size_t)a.ng * a.ca * chunk;
        int ctas = 0;
        for (int g = g0; g < g0 + a.ng; ++g) ctas += sym_slices(a.nchunk, g, GC, a.lc);
        e = launch_pdl(force_sym_kernel<ORDER>, dim3(ctas), kSymFWarps * 32, SymShape<ORDER>::bytes, s, a);
        const long long values = (long long)(a.ca - g0 * GC) * chunk;
        if (e == cudaSuccess)
            e = launch_pdl(sym_band_kernel<ORDER>, dim3((unsigned)((values + 255) / 256)), 256, 0, s, a);
        if (e != cudaSuccess) return e;
        *launches += 2;
    }
    return cudaSuccess;
}

}  // namespace

// The share of the pairs that is one-sided grows as fewer particles are active, and
// small calls do not fill the waves.  Both sides measured (ms, ordered pairs /
// pairs once): all of N = 4096 0.060 / 0.049 at 4th order and 0.088 / 0.090 at
// 6th, 131072 59.9 / 39.0 (6th); a fifth of N = 40000 0.656 / 0.640 (4th) and
// 1.122 / 1.090 (6th), of 262144 47.1 / 44.0 (6th), 0.15 of 65536 1.291 / 1.302
// (4th); 4096 of 16384 0.155 / 0.157 (4th) and 0.252 / 0.259 (6th).  The 8th-order
// sums are compensated; they keep ordered pairs.
bool force_sym_takes(int order, bool mixed, int nact, int npad, size_t cap)
{
    if (mixed || (order != 4 && order != 6)) return false;
    const size_t blocks = cap / (size_t)(3 * (order / 2) * 32);
    const bool most = nact >= 4096 && nact >= npad * 4LL / 10, many = nact >= 8192 && nact >= npad / 5;
    return (most || many) && blocks >= (size_t)npad / 32 * 2;
}

cudaError_t launch_force_sym(int order, const ForceArgs &f, size_t cap, int nsm, cudaStream_t s, int *launches)
{
    switch (order) {
    case 4: return launch_t<4>(f, cap, nsm, s, launches);
    case 6: return launch_t<6>(f, cap, nsm, s, launches);
    }
    return cudaErrorInvalidValue;
}

}  // namespace hb
