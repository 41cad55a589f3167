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

/// One [2, 3, 8, 64] line g of plan P through the team's shared-memory buffer s (LINE3072_WORDS); FIX: the
/// plan is fixed; stage: its twiddles are not there yet (from the same plan and direction).
template <int MODE, bool FIX, class TEAM>
__device__ __forceinline__ void run_line3072(const TEAM& tm, const DevPlanHeader* P, int64_t* s, int64_t* g, const int64_t* mulp,
                                             int64_t me, int64_t mn, int64_t mi, bool stage = true) {
    const auto c = make_ctx<PassCtx<FIX>>(P);
    int4* tws = reinterpret_cast<int4*>(s + 3072);
    with_sched<HC_SHAPE_L3072, (MODE & 1) != 0, FIX>(P, [&](const auto& sch) {
        if constexpr (FIX) {
            if (stage) fast::stage_tail_twiddles<(MODE & 1) != 0>(tm, c, sch, tws, 2, 7, 5);
        }
        fast::line3072<MODE>(tm, sch, c, s, tws, g, mulp, me, mn, mi);
    });
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
    auto store = [&](auto& x) {
        constexpr int A = sizeof(x) / sizeof(x[0]), B = sizeof(x[0]) / 8;
        uint32_t seen = 0;
#pragma unroll
        for (int a = 0; a < A; a++)
#pragma unroll
            for (int b = 0; b < B; b++) {
                int64_t v = x[a][b];
                if constexpr ((MODE & 2) != 0) {
                    const auto w = mont.load(mulp, (B * a + b) * mstride);
                    if constexpr (MODE == 2 && FIX) mont.see(seen, w);
                    v = mont.mul(v, w);
                }
                g[(B * a + b) * ge] = v;
            }
        if constexpr (MODE == 2 && FIX) {
            if (mont.out(seen)) {
                int64_t u[A * B];  // in memory, unlike x
#pragma unroll
                for (int a = 0; a < A; a++)
#pragma unroll
                    for (int b = 0; b < B; b++) u[B * a + b] = x[a][b];
                fast::mul_mont_column<A * B>(u, g, ge, mulp, mstride, mont.n(), mont.ninv());
            }
        }
    };
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
            store(x);
        } else {
            int64_t x[1][4];
#pragma unroll
            for (int a = 0; a < 4; a++) x[0][a] = gs[a * gse];
            fast::col4(c, f, inv, MODE == 0, x[0]);
            store(x);
        }
    });
}

/// The lead pass of a field_49152 slab at one position p of its blocks (see crt_slab.cu): the four-point
/// columns, with DIR 0 their products with the dimension-2 kernel m2 [4], and the radix-3 stage of the
/// four rows, from gs[k ss2 + 4096 b] to g[k s2 + 4096 b].
template <int DIR, int LG>
__device__ __forceinline__ void lead12288(const fast::CtxL& c2, const fast::CtxL& c3, const int64_t* gs, int64_t ss2,
                                          int64_t* g, int64_t s2, const BarrettLimbs* m2, int64_t n) {
    constexpr bool inv = DIR == 1;
    const FixedSched<HC_SHAPE_C4, LG, inv> sch2{};
    const FixedSched<HC_SHAPE_L12288, LG, inv> sch3{};
    const fast::SF f2[2] = {fast::sflags(sch2, 0), fast::sflags(sch2, 1)};
    const fast::SF f3 = fast::sflags(sch3, 0);
    int64_t x[3][4];
#pragma unroll
    for (int b = 0; b < 3; b++)
#pragma unroll
        for (int k = 0; k < 4; k++) x[b][k] = gs[k * ss2 + 4096 * b];
#pragma unroll
    for (int b = 0; b < 3; b++) fast::col4(c2, f2, inv, false, x[b]);
    const fast::MontC mont{mont_const_mod(n)};
#pragma unroll
    for (int k = 0; k < 4; k++) {
        if (DIR == 0) {
            const BarrettLimbs w = load_limbs(m2 + k);
#pragma unroll
            for (int b = 0; b < 3; b++) x[b][k] = mont.mul(x[b][k], w);
        }
        if (f3.red) {
#pragma unroll
            for (int b = 0; b < 3; b++) x[b][k] = fast::red1(c3, x[b][k]);
        }
        if (inv) fast::inv3(c3, f3, x[0][k], x[1][k], x[2][k]);
        else fast::fwd3<true>(c3, f3, false, 0, x[0][k], x[1][k], x[2][k]);
#pragma unroll
        for (int b = 0; b < 3; b++) g[k * s2 + 4096 * b] = x[b][k];
    }
}

}  // namespace
