// Dimension-3 lines of field_49152 ([3, 64, 64], 12288 residues): one line per 3-CTA cluster.
#include <cooperative_groups.h>

#include "ntt_run.cuh"

namespace {

/// [3, 64, 64] lines along dimension 3 as 3-CTA clusters: CTA `blk` of a cluster computes block
/// blk (4096 residues) of one line.
template <int MODE, bool FIX, int THREADS>
__global__ void __cluster_dims__(3, 1, 1) __launch_bounds__(THREADS, 768 / THREADS)
    ntt_line3_kernel(KView t, PlanPtrs plans, KView mul, KMods mods) {
    grid_wait();
    extern __shared__ __align__(16) int64_t smem[];
    const int64_t tile = blockIdx.x / 3;
    const int blk = (int)(blockIdx.x % 3);
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
    auto csync = [] { cooperative_groups::this_cluster().sync(); };
    const auto c = make_ctx<PassCtx<FIX>>(P);
    int4* tws = reinterpret_cast<int4*>(smem + 4096);
    with_sched<HC_SHAPE_L12288, (MODE & 1) != 0, FIX>(P, [&](const auto& sch) {
        if constexpr (FIX) fast::stage_tail_twiddles<(MODE & 1) != 0>(fast::CtaTeam{}, c, sch, tws, 1, 63, 7);
        fast::line12288_block<MODE>(sch, c, smem, tws, g, blk, mulp, me, mn, mi, csync);
    });
}

template <int MODE, bool FIX, int THREADS>
hc_status launch_as(hc_context ctx, const KView& t, const PlanPtrs& pp, const KView& mul, const KMods& mods, int64_t tiles) {
    // one 3-CTA cluster per line: a 4096-residue block per CTA
    constexpr size_t smem = (size_t)BLOCK4096_WORDS * 8;
    auto kern = ntt_line3_kernel<MODE, FIX, THREADS>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return hc::cuda_check(e, "ntt smem attribute");
    if (tiles * 3 > 0x7fffffff) return hc::fail(HC_ERR_UNSUPPORTED, "too many NTT lines in one call");
    hc::launch_kernel(kern, (unsigned)(tiles * 3), THREADS, smem, hc::stream_of(ctx), t, pp, mul, mods);
    hc::count_launch(ctx);
    return hc::cuda_check(cudaGetLastError(), "ntt kernel launch");
}
/// 128 threads per CTA, or 256 for lines that all fit the device at once (three CTAs per SM, one line
/// per SM), where a line's own latency is the launch's, and for the general products ([8, 4, 12, 12288] at a 45-bit
/// prime 77 us forward and 79 inverse, 92 and 94 with 128).
template <int MODE, bool FIX>
hc_status launch(hc_context ctx, const KView& t, const PlanPtrs& pp, const KView& mul, const KMods& mods, int64_t tiles) {
    if constexpr (FIX) {
        if (tiles > hc::num_sms(ctx)) return launch_as<MODE, FIX, 128>(ctx, t, pp, mul, mods, tiles);
    }
    return launch_as<MODE, FIX, 256>(ctx, t, pp, mul, mods, tiles);
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

hc_status launch_ntt_line12288(hc_context ctx, int mode, bool fix, const KView& t, const PlanPtrs& pp, const KView& mul, const KMods& mods, int64_t tiles) {
    return fix ? launch_mode<true>(ctx, mode, t, pp, mul, mods, tiles) : launch_mode<false>(ctx, mode, t, pp, mul, mods, tiles);
}

}  // namespace hc
