// hb_force_sym.cu -- launches of the each-pair-once FP64 force.
#include <algorithm>

#include "hb_force_sym.cuh"

namespace hb {
namespace {

struct Band {
    int ng, lc, smax;      // groups, chunks per slice, slices per group at most
};

// The band from group g0 on, for scratch of `room` [F][32] blocks: as many groups as
// it has rows and slice sums for, in slices that make 10 to 20 waves of CTAs, in
// whole tiles: 20 as long as the slice sums take no more than 0.4 of the rows' room
// (with 32 rows, 6th order, N = 131072: 4 waves 41.7 ms, 6 40.5, 10 40.0; with 64,
// 10 39.7, 20 39.3; N = 50000 5.92, 5.98).  Little scratch makes the slices longer:
// a group's row and its slice sums fit wherever two rows do.
template <int ORDER>
Band band_from(int g0, int ca, int nchunk, long long room, int nsm)
{
    constexpr int GC = SymShape<ORDER>::GC;
    const int groups = (ca + GC - 1) / GC;
    const long long wave = SymShape<ORDER>::MINB * nsm, most = (room - ca) / GC;
    Band b{(int)std::min((long long)(groups - g0), room / ca), 0, 0};
    if (most < 1) return Band{};
    for (int pass = 0; pass < 3 && b.ng > 0; ++pass) {
        const long long units = (long long)b.ng * (nchunk - (long long)g0 * GC) - (long long)GC * b.ng * (b.ng - 1) / 2;
        long long lc = std::min(units / (10 * wave), std::max(units / (20 * wave), 5LL * GC * nchunk / (2 * ca)));
        lc = std::max({lc, (nchunk - (long long)g0 * GC + most - 1) / most, 1LL});
        b.lc = (int)((lc + kSymFTile - 1) / kSymFTile) * kSymFTile;
        b.smax = sym_slices(nchunk, g0, GC, b.lc);
        b.ng = (int)std::min((long long)b.ng, room / (ca + (long long)b.smax * GC));
    }
    return b;
}

template <int ORDER>
int bands_t(int ca, int nchunk, size_t cap, int nsm)
{
    const long long room = (long long)(cap / (Frc<ORDER>::words * 32));
    int bands = 0;
    for (int g0 = 0; g0 * SymShape<ORDER>::GC < ca; ++bands) {
        const Band b = band_from<ORDER>(g0, ca, nchunk, room, nsm);
        // its rows and slice sums have to fit
        if (b.ng < 1 || b.ng * (ca + (long long)b.smax * SymShape<ORDER>::GC) > room) return -1;
        g0 += b.ng;
    }
    return bands;
}

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
        const Band b = band_from<ORDER>(g0, a.ca, a.nchunk, room, nsm);
        a.g0 = g0;
        a.ng = b.ng;
        a.lc = b.lc;
        a.smax = b.smax;
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
// pairs once): all of N = 4096 0.088 / 0.090 at 6th order, 131072 59.9 / 39.0
// (6th); a fifth of N = 40000 0.656 / 0.640 (4th) and 1.122 / 1.090 (6th), of
// 262144 47.1 / 44.0 (6th), 0.15 of 65536 1.291 / 1.302 (4th); 4096 of 16384 0.252 /
// 0.259 (6th).  At 4th order it starts where the results are too large to be
// written straight to the host (kZeroCopyBytes, hb_capi.cu: 5461 records): below,
// whole calls through the host take longer with it and the copy that the bands'
// device sums then need (4096 of 4500 106 / 121 us, of 8000 133 / 141, 4800 of 8000 158 /
// 161), and one rule has to serve every entry point, or their bits would differ.
// The 8th-order sums are compensated; they keep ordered pairs.
bool force_sym_takes(int order, bool mixed, int nact, int npad, size_t cap)
{
    if (mixed || (order != 4 && order != 6)) return false;
    const size_t blocks = cap / (size_t)(3 * (order / 2) * 32);
    const bool most = nact >= (order == 4 ? 5462 : 4096) && nact >= npad * 4LL / 10;
    const bool many = nact >= 8192 && nact >= npad / 5;
    return (most || many) && blocks >= (size_t)npad / 32 * 2;
}

int force_sym_bands(int order, int nact, int npad, size_t cap, int nsm)
{
    if (!force_sym_takes(order, false, nact, npad, cap)) return 0;
    const int ca = (nact + 31) / 32;
    return order == 4 ? bands_t<4>(ca, npad / 32, cap, nsm) : bands_t<6>(ca, npad / 32, cap, nsm);
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
