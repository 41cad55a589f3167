// Dimension-3 lines of field_36864 ([2, 3, 8, 64], 3072 residues): one line per CTA.
#include "ntt_run.cuh"

namespace {

/// Specialised dimension-3 NTT: one line (i, j, k) per CTA.
template <int MODE, bool FIX, int THREADS, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) ntt_line_kernel(KView t, PlanPtrs plans, KView mul, KMods mods) {
    grid_wait();
    extern __shared__ __align__(16) int64_t smem[];
    const int64_t tile = blockIdx.x;
    const int64_t k = tile % t.n2, r = tile / t.n2;
    const int64_t j = r % t.n1, i = r / t.n1;
    const DevPlanHeader* P = plans.p[j];
    int64_t* g = reinterpret_cast<int64_t*>(t.p) + i * t.s0 + j * t.s1 + k * t.s2;
    const int64_t* mulp = nullptr;
    int64_t me = 0, mn = 0, mi = 0;
    if (MODE & 2) {
        mulp = multiplier<MODE>(mul, i, j, k, 0);
        me = mul.b3 ? 0 : 1;
        mn = mods.n[j], mi = mods.ninv[j];
    }
    run_line3072<MODE, FIX>(fast::CtaTeam{}, P, smem, g, mulp, me, mn, mi);
}

template <int MODE, bool FIX, int THREADS, int MINB>
hc_status launch_as(hc_context ctx, const KView& t, const PlanPtrs& pp, const KView& mul, const KMods& mods, int64_t tiles) {
    constexpr size_t smem = (size_t)LINE3072_WORDS * 8;
    auto kern = ntt_line_kernel<MODE, FIX, THREADS, MINB>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return hc::cuda_check(e, "ntt smem attribute");
    hc::launch_kernel(kern, (unsigned)tiles, THREADS, smem, hc::stream_of(ctx), t, pp, mul, mods);
    hc::count_launch(ctx);
    return hc::cuda_check(cudaGetLastError(), "ntt kernel launch");
}
/// 128 threads per line: the fewest idle slots in the last wave, and seven (forward, 72 registers: ntt_mul
/// of [24, 20, 12, 3072] 124 us, with eight 130) or eight (inverse: intt 105 us, with seven 107) independent
/// CTAs per SM to cover each other's barriers. Up to three lines per SM (one
/// element of 38 factors) a line's own latency is the launch's, and 384 threads shorten it: one element at
/// r = 16 41.5 -> 36.7 us per transform; with the line at two per SM instead a ct-mult at r = 16 (384 lines beside
/// another stream's launches) 407 us, at three 400, at six 404, and one per SM costs the one element 5 us.
template <int MODE, bool FIX>
hc_status launch(hc_context ctx, const KView& t, const PlanPtrs& pp, const KView& mul, const KMods& mods, int64_t tiles) {
    if (tiles <= 3 * (int64_t)hc::num_sms(ctx)) return launch_as<MODE, FIX, 384, 2>(ctx, t, pp, mul, mods, tiles);
    return launch_as<MODE, FIX, 128, (MODE & 1) ? 8 : 7>(ctx, t, pp, mul, mods, tiles);
}

template <bool FIX>
hc_status launch_mode(hc_context ctx, int mode, const KView& t, const PlanPtrs& pp, const KView& mul, const KMods& mods, int64_t tiles) {
    if (mode == 0) return launch<0, FIX>(ctx, t, pp, mul, mods, tiles);
    if (mode == 1) return launch<1, FIX>(ctx, t, pp, mul, mods, tiles);
    if (mode == 2) return launch<2, FIX>(ctx, t, pp, mul, mods, tiles);
    if (FIX && mode == 6) return launch<6, true>(ctx, t, pp, mul, mods, tiles);
    return launch<3, FIX>(ctx, t, pp, mul, mods, tiles);
}

}  // namespace

namespace hc {

hc_status launch_ntt_line3072(hc_context ctx, int mode, bool fix, const KView& t, const PlanPtrs& pp, const KView& mul, const KMods& mods, int64_t tiles) {
    return fix ? launch_mode<true>(ctx, mode, t, pp, mul, mods, tiles) : launch_mode<false>(ctx, mode, t, pp, mul, mods, tiles);
}

}  // namespace hc
