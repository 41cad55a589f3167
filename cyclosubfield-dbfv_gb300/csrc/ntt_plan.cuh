// Device-side NTT plan layout shared by the translation units that run NTT kernels: the stage
// program and twiddle table a plan uploads (built by csrc/ntt.cu:build_plan), the specialised
// shapes of the two large field descriptors with their compiled-in schedules, and the register /
// shared-memory building blocks of ntt_fast.cuh.
#pragma once
#include <type_traits>

#include "common.cuh"

/// Division by an invariant divisor d (1 <= d < 2^32) with a multiply-high and shifts
/// (Granlund & Montgomery, "Division by invariant integers using multiplication", 1994, fig. 4.1).
struct FastDiv {
    uint32_t d, m, s1, s2;
};

struct DevStage {
    int32_t radix;      // 2 or 3
    int32_t stride;     // element stride of the factor's digit within the axis (suffix product)
    int32_t flen;       // factor length
    int32_t stage_len;  // length of one block in this stage
    int32_t tw_off;     // twiddle offset (pairs z,u): fwd r2: 1/block, fwd r3: 6/block, inv r2: 1, inv r3: 2
    int32_t zeta_off;   // inverse radix-3: offset of (zeta, zeta2)
    int32_t reduce_before;
    int32_t skip_ok;    // forward only
    int32_t last;       // last stage of the last factor (fwd: fusable reduction, inv: fused len^-1)
    int32_t span;       // (stage_len / radix) * stride: butterflies per group, distance of the legs
    FastDiv div_span;   // butterfly index -> (group, offset in group)
    FastDiv div_nblocks;  // group -> twiddle block (group mod flen / stage_len)
};

inline FastDiv make_fastdiv(uint32_t d) {
    FastDiv f;
    f.d = d;
    uint32_t l = 0;
    while (l < 32 && ((uint64_t)1 << l) < d) l++;
    f.m = (uint32_t)((((uint64_t)1 << 32) * ((((uint64_t)1) << l) - d)) / d + 1);
    f.s1 = l < 1 ? l : 1;
    f.s2 = l > 1 ? l - 1 : 0;
    return f;
}

/// A pass of the kernel: either one stage through shared memory (kind 0, any radix), or k <= 3
/// consecutive radix-2 stages of one factor executed in registers (kind 1): each thread loads a
/// group of 2^k elements `span` apart, applies the k stages' butterflies to it in the
/// reference's order, and stores it back.
struct DevPass {
    int32_t kind;
    int32_t k;
    int32_t first;  // index of the pass's first stage in the (forward or inverse) program
    int32_t span;   // distance of consecutive group elements
    int32_t glen;   // extent of the block a group lies in (stage_len * stride)
    int32_t nb;     // blocks of that stage within the factor (twiddle block of a group)
    FastDiv div_span;
    FastDiv div_nb;
};

struct DevPlanHeader {
    int64_t n;
    int32_t len;
    int32_t nfwd;
    int32_t ninv;
    int32_t ntw;
    int32_t nfpass;
    int32_t nipass;
    int32_t cls;  // fixed plans: 56 or 57 (the schedule's fixed_masks), else 0
    int32_t pad;
    int64_t one_z, one_u, invlen_z, invlen_u;
    BarrettMod mod;  // limb forms, used by the plans whose products fit them (hc_ntt_plan_s::fixed)
    BarrettLimbs invlen;
    DevStage fwd[HC_MAX_STAGES];
    DevStage inv[HC_MAX_STAGES];
    DevPass fpass[HC_MAX_STAGES];
    DevPass ipass[HC_MAX_STAGES];
    // followed by the twiddle table as ntw pairs (z, u), then as ntw BarrettLimbs
};

struct PlanPtrs {
    const DevPlanHeader* p[HC_MAX_MODS];
};
static_assert(sizeof(DevPlanHeader) % 16 == 0, "plan twiddle tables must be 16-byte aligned");

namespace {
#include "ntt_fast.cuh"

#define HC_SHAPE_GENERIC 0
#define HC_SHAPE_L3072 1   // dimension-3 line [2, 3, 8, 64]
#define HC_SHAPE_L12288 2  // dimension-3 line [3, 64, 64]
#define HC_SHAPE_C12 3     // dimension-2 column [4, 3]
#define HC_SHAPE_C4 4      // dimension-2 column [4]

#define HC_COL_THREADS 256  // of the column kernel

/// Shared-memory words of a 3072-residue line, and of a 4096-residue block of a 12288-residue one: the
/// tile, then its staged twiddles.
constexpr int LINE3072_WORDS = 3072 + fast::staged_words(7), BLOCK4096_WORDS = 4096 + fast::staged_words(63);
static_assert(LINE3072_WORDS % 2 == 0 && BLOCK4096_WORDS % 2 == 0, "staged twiddles are read 16 bytes at a time");

/// Contexts of a plan: its twiddles are read from global memory (L1-cached).
template <class CTX>
__device__ __forceinline__ CTX make_ctx(const DevPlanHeader* P) {
    CTX c;
    const int64_t* tw = reinterpret_cast<const int64_t*>(P + 1);
    if constexpr (CTX::LIMBS) {
        c.m = P->mod, c.il = P->invlen;
        c.tw = reinterpret_cast<const int4*>(tw + 2 * P->ntw);
    } else {
        c.n = P->n, c.one_u = P->one_u, c.il_z = P->invlen_z, c.il_u = P->invlen_u;
        c.tw = tw;
    }
    return c;
}

/// The reduction / skip / fused-final schedule (bit s = the flag of stage s) of a specialised shape's
/// plan for a prime just below 2^lg, by the bound tracking of build_plan in units of the prime (k
/// primes fit a signed word exactly when k <= 2^(63 - lg)). The rings sample their primes below 2^57
/// and 2^56, often both in one base, so a kernel carries these two schedules and each CTA takes its
/// row's (`cls` of the plan): compiled in, the flags fold into straight-line code (intt along dimension
/// 3 of a [24, 20, 12, 3072] tensor 111 us, 146 us with the flags read from the plan). A plan
/// counts as fixed when it has one of the two and its products fit the limb forms (BarrettLimbs).
struct SchedMasks {
    uint32_t fred, fskip, flast, ired, ilast;
};
__host__ __device__ constexpr SchedMasks fixed_masks(int shape, int lg) {
    // radices of the stages, forward and inverse (a factor's stages are alike in both directions)
    const int nst = shape == HC_SHAPE_L3072 ? 11 : shape == HC_SHAPE_L12288 ? 13 : shape == HC_SHAPE_C12 ? 3 : shape == HC_SHAPE_C4 ? 2 : 0;
    const int r3 = shape == HC_SHAPE_L3072 ? 1 : shape == HC_SHAPE_L12288 ? 0 : shape == HC_SHAPE_C12 ? 2 : -1;
    const int64_t max = (int64_t)1 << (63 - lg);
    SchedMasks m{0u, 0u, 0u, 0u, 0u};
    int64_t f = 2, v = 2;
    for (int s = 0; s < nst; s++) {
        const int64_t radix = s == r3 ? 3 : 2;
        if (f + radix - 1 > max) m.fred |= 1u << s, f = 1;
        if (radix * f <= max) m.fskip |= 1u << s, f *= radix;
        else f += radix - 1;
        if (radix * v > max) m.ired |= 1u << s, v = 1;
        v *= radix;
    }
    if (nst) m.flast = m.ilast = 1u << (nst - 1);
    return m;
}
/// Offsets of a specialised shape's twiddle table as build_plan lays it out: per factor the two cube roots
/// of a factor 3, then its forward stages (2^s or 6 3^s entries), then its inverse stages.
struct TableLayout {
    int fwd[16], inv[16], zeta[16];  // by stage; zeta: of the inverse stage's factor
    int words;
};
__host__ __device__ constexpr TableLayout table_layout(int shape) {
    TableLayout t{};
    const int factors[4][4] = {{2, 3, 8, 64}, {3, 64, 64, 1}, {4, 3, 1, 1}, {4, 1, 1, 1}};
    int at = 0, st = 0;
    for (int i = 0; i < 4; i++) {
        const int f = factors[shape - HC_SHAPE_L3072][i], radix = f == 3 ? 3 : 2;
        int nst = 0, zeta = 0;
        for (int l = 1; l < f; l *= radix) nst++;
        if (f == 3) zeta = at, at += 2;
        for (int q = 0, n = 1; q < nst; q++, n *= radix) t.fwd[st + q] = at, at += radix == 3 ? 6 * n : n;
        for (int q = 0; q < nst; q++) {  // the inverse runs the stages in reverse order
            int n = 1;
            for (int e = 0; e < nst - 1 - q; e++) n *= radix;
            t.inv[st + q] = at, t.zeta[st + q] = zeta, at += radix == 3 ? 2 * n : n;
        }
        st += nst;
    }
    t.words = at;
    return t;
}
template <int SHAPE, bool INV>
struct Table {
    __host__ __device__ static constexpr int offset(int s) { return INV ? table_layout(SHAPE).inv[s] : table_layout(SHAPE).fwd[s]; }
    __host__ __device__ static constexpr int zeta(int s) { return table_layout(SHAPE).zeta[s]; }
};

template <int SHAPE, int LG, bool INV>
using FixedSched = fast::FixSched<INV ? fixed_masks(SHAPE, LG).ired : fixed_masks(SHAPE, LG).fred,
                                  INV ? 0u : fixed_masks(SHAPE, LG).fskip,
                                  INV ? fixed_masks(SHAPE, LG).ilast : fixed_masks(SHAPE, LG).flast, Table<SHAPE, INV>>;

/// Calls f with the compiled-in schedule of a fixed plan (SHAPE, direction INV), or with the
/// schedule read from any plan (FIX = false). Uniform over a CTA that works for one plan.
template <int SHAPE, bool INV, bool FIX, class F>
__device__ __forceinline__ void with_sched(const DevPlanHeader* P, F f) {
    if constexpr (!FIX) f(fast::DynSched{INV ? P->inv : P->fwd});
    else if constexpr (std::is_same_v<FixedSched<SHAPE, 56, INV>, FixedSched<SHAPE, 57, INV>>) f(FixedSched<SHAPE, 57, INV>{});
    else if (P->cls == 57) f(FixedSched<SHAPE, 57, INV>{});
    else f(FixedSched<SHAPE, 56, INV>{});
}

}  // namespace
