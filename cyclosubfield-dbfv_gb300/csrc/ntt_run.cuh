// One specialised line or column of a plan, as the single-call kernels and the batched-transform kernel
// run them.
#pragma once
#include "ntt_plan.cuh"

namespace {

/// The arithmetic of a specialised kernel: limb products for the fixed plans (FIX), the general ones
/// otherwise.
template <bool FIX>
using PassCtx = std::conditional_t<FIX, fast::CtxL, fast::Ctx>;

/// The multiplier of tile element (i, j, k, l): Montgomery words, or a table of limbs (mode bit 2).
template <int MODE>
__device__ __forceinline__ const int64_t* multiplier(const KView& mul, int64_t i, int64_t j, int64_t k, int64_t l) {
    if constexpr ((MODE & 4) != 0) return reinterpret_cast<const int64_t*>(kat<BarrettLimbs>(mul, i, j, k, l));
    else return kat<int64_t>(mul, i, j, k, l);
}

/// One [2, 3, 8, 64] line g of plan P through the CTA's shared-memory line buffer s; FIX: the plan is
/// fixed.
template <int MODE, bool FIX>
__device__ __forceinline__ void run_line3072(const DevPlanHeader* P, int64_t* s, int64_t* g, const int64_t* mulp,
                                             int64_t me, int64_t mn, int64_t mi) {
    const auto c = make_ctx<PassCtx<FIX>>(P);
    with_sched<HC_SHAPE_L3072, (MODE & 1) != 0, FIX>(
        P, [&](const auto& sch) { fast::line3072<MODE>(sch, c, s, g, mulp, me, mn, mi); });
}

/// One specialised column g[0], g[ge], ... of shape SHAPE transformed in registers; it is read
/// from gs[0], gs[gse], ... (g itself for an in-place call).
template <int SHAPE, int MODE, bool FIX>
__device__ __forceinline__ void run_column(const DevPlanHeader* P, int64_t* g, int64_t ge,
                                           const int64_t* gs, int64_t gse, const int64_t* mulp, int64_t mstride,
                                           int64_t mn, int64_t mi) {
    constexpr bool inv = MODE & 1;
    typedef PassCtx<FIX> CTX;
    const CTX c = make_ctx<CTX>(P);
    const auto mont = fast::make_mont<CTX, MODE>(mn, mi);
    constexpr int NST = SHAPE == HC_SHAPE_C12 ? 3 : 2;
    with_sched<SHAPE, inv, FIX>(P, [&](const auto& sch) {
        fast::SF f[NST];
#pragma unroll
        for (int q = 0; q < NST; q++) f[q] = fast::sflags(sch, q);
        if constexpr (SHAPE == HC_SHAPE_C12) {
            int64_t x[4][3];
#pragma unroll
            for (int a = 0; a < 4; a++)
#pragma unroll
                for (int b = 0; b < 3; b++) x[a][b] = gs[(3 * a + b) * gse];
            fast::col12(c, f, inv, MODE == 0, x);
#pragma unroll
            for (int a = 0; a < 4; a++)
#pragma unroll
                for (int b = 0; b < 3; b++) {
                    int64_t v = x[a][b];
                    if (MODE & 2) v = mont.mul(v, mont.load(mulp, (3 * a + b) * mstride));
                    g[(3 * a + b) * ge] = v;
                }
        } else {
            int64_t x[4];
#pragma unroll
            for (int a = 0; a < 4; a++) x[a] = gs[a * gse];
            fast::col4(c, f, inv, MODE == 0, x);
#pragma unroll
            for (int a = 0; a < 4; a++) {
                int64_t v = x[a];
                if (MODE & 2) v = mont.mul(v, mont.load(mulp, a * mstride));
                g[a * ge] = v;
            }
        }
    });
}

}  // namespace
