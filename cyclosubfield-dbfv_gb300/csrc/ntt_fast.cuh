// Specialised NTT kernels for the factorisations of the two large field descriptors:
//   dimension 3 lines   [2, 3, 8, 64] (field_36864, deg_K = 3072)  and [3, 64, 64] (field_49152, 12288)
//   dimension 2 columns [4, 3]        (field_36864, deg_L' = 12)    and [4]         (field_49152, 4)
// They execute the same stage programs as the generic kernel (same butterflies, same order, the
// same reduction/skip/fused-final decisions read from the plan), so results are bit-identical; what
// differs is the schedule:
//  * every stage geometry is a compile-time constant, so index arithmetic is shifts and
//    immediate offsets;
//  * lines: the first register pass reads its elements straight from global memory and runs the
//    leading radix-2/radix-3 factors together; the remaining radix-2 stages run three at a time on
//    eight elements per thread; the tile lives in shared memory, its columns swizzled so that
//    every pass's 64-bit accesses are free of bank conflicts (sw), with the twiddles of the passes
//    behind the first beside it;
//  * columns: one thread transforms a whole column (12 or 4 residues) in registers, loading and
//    storing it coalesced across neighbouring columns - no shared memory at all;
//  * a twiddle-1 butterfly skips its multiplication only where the skip is uniform across the
//    warp (a stage with a single twiddle block); elsewhere the product is computed and the
//    unmultiplied value selected, exactly as the reference's result requires.
#pragma once

namespace fast {

/// Slot of tile element i: its low four bits XOR-ed with bits 4..6, bit 6 entering twice (bits 2 and 3).
/// Sixteen 8-byte words span the banks, and every access of a half-warp here is one of: sixteen
/// neighbours, eight words apart (neighbours' groups), or two runs of eight 64 apart; each of these
/// falls into sixteen distinct columns. (One word of padding per eight, the layout before, made the
/// sixteen neighbours collide: a third of the shared-memory cycles.) The map is linear over XOR.
__host__ __device__ constexpr int sw(int i) { return i ^ ((i >> 4) & 7) ^ ((i >> 3) & 8); }
/// Element base + part of a tile, for a constant part whose bits are clear in base; swb = sw(base).
__device__ __forceinline__ int64_t& el(int64_t* s, int swb, int part) {
    return s[(swb ^ (sw(part) & 127)) + (sw(part) & ~127)];
}

/// Products of a plan with any schedule and modulus: (z, u) pairs.
struct Ctx {
    static constexpr bool LIMBS = false;
    int64_t n, one_u, il_z, il_u;
    const int64_t* tw;  // twiddle pairs
    typedef longlong2 Tw;
    __device__ __forceinline__ Tw get(int idx) const { return reinterpret_cast<const longlong2*>(tw)[idx]; }
    __device__ __forceinline__ int64_t mul(const Tw& w, int64_t x) const { return bmul(w.x, w.y, x, n); }
    __device__ __forceinline__ int64_t scale(int64_t x) const { return bmul(il_z, il_u, x, n); }
    __device__ __forceinline__ int64_t red(int64_t x) const { return bmul1(one_u, x, n); }
};

/// The same products in limbs (barrett_mul), for the plans with the compiled-in schedules.
struct CtxL {
    static constexpr bool LIMBS = true;
    BarrettMod m;
    BarrettLimbs il;
    const int4* tw;  // twiddles (BarrettLimbs)
    typedef BarrettLimbs Tw;
    __device__ __forceinline__ Tw get(int idx) const {
        const int4 a = __ldg(tw + idx);
        return BarrettLimbs{a.x, a.y, a.z, a.w};
    }
    __device__ __forceinline__ int64_t mul(const Tw& w, int64_t x) const { return barrett_mul(w, x, m); }
    __device__ __forceinline__ int64_t scale(int64_t x) const { return barrett_mul(il, x, m); }
    __device__ __forceinline__ int64_t red(int64_t x) const { return barrett_red(x, m); }
};

/// CtxL with a pass's twiddles in shared memory (stage_tail_twiddles).
struct CtxS {
    static constexpr bool LIMBS = true;
    BarrettMod m;
    BarrettLimbs il;
    const int4* tw;
    typedef BarrettLimbs Tw;
    __device__ __forceinline__ Tw get(int idx) const {
        const int4 a = tw[idx];
        return BarrettLimbs{a.x, a.y, a.z, a.w};
    }
    __device__ __forceinline__ int64_t mul(const Tw& w, int64_t x) const { return barrett_mul(w, x, m); }
    __device__ __forceinline__ int64_t scale(int64_t x) const { return barrett_mul(il, x, m); }
    __device__ __forceinline__ int64_t red(int64_t x) const { return barrett_red(x, m); }
};

/// Stage flags of the program, read once per pass (uniform).
struct SF {
    int tw_off, zeta_off;
    bool red, skip_ok, last;
};

/// The plan's reduction / skip / fused-final schedule and table offsets read at run time (any prime).
struct DynSched {
    const DevStage* st;
    __device__ __forceinline__ bool red(int s) const { return st[s].reduce_before; }
    __device__ __forceinline__ bool skip(int s) const { return st[s].skip_ok; }
    __device__ __forceinline__ bool last(int s) const { return st[s].last; }
    __device__ __forceinline__ int tw(int s) const { return st[s].tw_off; }
    __device__ __forceinline__ int zeta(int s) const { return st[s].zeta_off; }
};
/// A schedule known at compile time (bit s = the flag of stage s) with the table offsets T of its
/// shape and direction, for primes whose plan has exactly this schedule: flags fold into
/// straight-line code and offsets into addresses, with no load of the stage program in front of the
/// loads of its twiddles.
template <uint32_t RED, uint32_t SKIP, uint32_t LAST, class T>
struct FixSched {
    __device__ __forceinline__ bool red(int s) const { return (RED >> s) & 1; }
    __device__ __forceinline__ bool skip(int s) const { return (SKIP >> s) & 1; }
    __device__ __forceinline__ bool last(int s) const { return (LAST >> s) & 1; }
    __device__ __forceinline__ int tw(int s) const { return T::offset(s); }
    __device__ __forceinline__ int zeta(int s) const { return T::zeta(s); }
};

template <class SCH>
__device__ __forceinline__ SF sflags(const SCH& sch, int s) {
    SF f;
    f.tw_off = sch.tw(s), f.zeta_off = sch.zeta(s);
    f.red = sch.red(s), f.skip_ok = sch.skip(s), f.last = sch.last(s);
    return f;
}

template <class CTX>
__device__ __forceinline__ int64_t red1(const CTX& c, int64_t x) { return c.red(x); }

/// The threads that run one line or block together: a whole CTA, or a part of it with a barrier of its
/// own (named barrier `bar`).
struct CtaTeam {
    __device__ __forceinline__ int tid() const { return threadIdx.x; }
    __device__ __forceinline__ int size() const { return blockDim.x; }
    __device__ __forceinline__ void sync() const { __syncthreads(); }
};
struct PartTeam {
    int rank, threads, bar;
    __device__ __forceinline__ int tid() const { return rank; }
    __device__ __forceinline__ int size() const { return threads; }
    __device__ __forceinline__ void sync() const { asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(threads) : "memory"); }
};

// ---------------------------------------------------------------- butterflies

/// Forward radix-2 butterfly of block `tb` (src/hal/ntt.rs:338-349), whose twiddle is entry `at` of its
/// stage's. UNIFORM0: the block is 0 for the whole warp, so a permitted skip avoids the product.
template <bool UNIFORM0, class CTX>
__device__ __forceinline__ void fwd2(const CTX& c, const SF& f, bool fuse, int tb, int at, int64_t& x, int64_t& y) {
    int64_t t;
    if (UNIFORM0) {
        if (f.skip_ok) {
            t = y;
        } else {
            t = c.mul(c.get(f.tw_off), y);
        }
    } else {
        t = c.mul(c.get(f.tw_off + at), y);
        if (f.skip_ok && tb == 0) t = y;
    }
    int64_t o0 = wadd(x, t), o1 = wsub(x, t);
    if (fuse) {
        o0 = red1(c, o0);
        o1 = red1(c, o1);
    }
    x = o0;
    y = o1;
}

/// Forward radix-3 butterfly of block `blk` (src/hal/ntt.rs:386-406).
template <bool UNIFORM0, class CTX>
__device__ __forceinline__ void fwd3(const CTX& c, const SF& f, bool fuse, int blk, int64_t& a, int64_t& b,
                                     int64_t& d) {
    const int base = f.tw_off + 6 * blk;
    int64_t t_b, t_c;
    if (f.skip_ok && blk == 0) {  // block 0's twiddle is 1
        t_b = b;
        t_c = d;
    } else {
        t_b = c.mul(c.get(base), b);
        t_c = c.mul(c.get(base + 3), d);
    }
    const int64_t t_bz = c.mul(c.get(base + 1), b), t_bzz = c.mul(c.get(base + 2), b);
    const int64_t t_cz = c.mul(c.get(base + 4), d), t_czz = c.mul(c.get(base + 5), d);
    int64_t o0 = wadd(wadd(a, t_b), t_c), o1 = wadd(wadd(a, t_bz), t_czz), o2 = wadd(wadd(a, t_bzz), t_cz);
    if (fuse) {
        o0 = red1(c, o0);
        o1 = red1(c, o1);
        o2 = red1(c, o2);
    }
    a = o0;
    b = o1;
    d = o2;
}

/// Inverse radix-3 butterfly of a factor-3 stage (src/hal/ntt.rs:511-530). Every radix-3 stage
/// of the specialised shapes is the single stage of a factor of length 3: it has one block, whose
/// twiddles are v^0 = 1, so the reference's twiddle-1 skip always applies and the outputs take
/// no block-twiddle product (only the fused len^-1 scaling when the stage is the last one).
template <class CTX>
__device__ __forceinline__ void inv3(const CTX& c, const SF& f, int64_t& a, int64_t& b, int64_t& d) {
    const auto w1 = c.get(f.zeta_off), w2 = c.get(f.zeta_off + 1);
    const int64_t y1z = c.mul(w1, b), y1zz = c.mul(w2, b), y2z = c.mul(w1, d), y2zz = c.mul(w2, d);
    const int64_t s0 = wadd(wadd(a, b), d);
    const int64_t sy = wadd(wadd(a, y1zz), y2z), sz = wadd(wadd(a, y1z), y2zz);
    if (f.last) {
        a = c.scale(s0);
        b = c.scale(sy);
        d = c.scale(sz);
        return;
    }
    a = s0;
    b = sy;
    d = sz;
}

// ---------------------------------------------------------------- register groups of radix-2 stages

/// K forward radix-2 stages on the group x[0..2^K) (element m at distance m * span). block0:
/// the group's twiddle block at the first stage (0 for the whole warp when NB0 == 1). BY_PART: the
/// stages' tables are ordered by the block's compile-time part (stage_tail_twiddles).
template <int K, bool NB1, bool BY_PART = false, class CTX>
__device__ __forceinline__ void fwd_group(const CTX& c, const SF* f, const bool* fuse, int block0, int64_t* x) {
    constexpr int M = 1 << K;
#pragma unroll
    for (int q = 0; q < K; q++) {
        if (f[q].red) {
#pragma unroll
            for (int m = 0; m < M; m++) x[m] = red1(c, x[m]);
        }
        const int half = M >> (q + 1);
#pragma unroll
        for (int j = 0; j < M / 2; j++) {
            const int m1 = ((j / half) * 2 * half) + (j % half), m2 = m1 + half;
            const int tbc = m1 >> (K - q);  // compile-time part of the block
            const int tb = (block0 << q) + tbc;
            if (NB1 && tbc == 0) fwd2<true>(c, f[q], fuse[q], 0, 0, x[m1], x[m2]);
            else fwd2<false>(c, f[q], fuse[q], tb, BY_PART ? 8 * tbc + block0 : tb, x[m1], x[m2]);
        }
    }
}

/// K inverse radix-2 stages (distances growing) on the group x[0..2^K); blockK: the group's block
/// at the pass's last stage (NBK1: 0 for the whole warp).
template <int K, bool NBK1, bool BY_PART = false, class CTX>
__device__ __forceinline__ void inv_group(const CTX& c, const SF* f, int blockK, int64_t* x) {
    constexpr int M = 1 << K;
#pragma unroll
    for (int q = 0; q < K; q++) {
        if (f[q].red) {
#pragma unroll
            for (int m = 0; m < M; m++) x[m] = red1(c, x[m]);
        }
        const int dist = 1 << q;
#pragma unroll
        for (int j = 0; j < M / 2; j++) {
            const int m1 = ((j >> q) << (q + 1)) | (j & (dist - 1)), m2 = m1 + dist;
            const int tbc = m1 >> (q + 1);
            const int64_t sum = wadd(x[m1], x[m2]), dif = wsub(x[m1], x[m2]);
            if (f[q].last) {
                x[m1] = c.scale(sum);
                x[m2] = c.scale(dif);
            } else if (NBK1 && tbc == 0) {
                // block 0 for the whole warp: twiddle 1, product skipped
                x[m1] = sum;
                x[m2] = dif;
            } else {
                const int tb = (blockK << (K - 1 - q)) + tbc;
                int64_t t = c.mul(c.get(f[q].tw_off + (BY_PART ? 8 * tbc + blockK : tb)), dif);
                if (tbc == 0 && tb == 0) t = dif;  // block 0's twiddle is 1, no other block's is
                x[m1] = sum;
                x[m2] = t;
            }
        }
    }
}

/// One pass of K radix-2 stages of a factor over a shared-memory tile: groups of 2^K
/// elements at distance SPAN (= 2^LOG_SPAN) inside blocks of 2^LOG_GLEN elements, 2^LOG_NB twiddle
/// blocks per factor at the pass's reference stage (first stage forward, last stage inverse).
template <bool INV, int K, int LOG_SPAN, int LOG_GLEN, int LOG_NB, class SCH, class CTX, class TEAM>
__device__ __forceinline__ void r2_pass(const TEAM& tm, const CTX& c, int64_t* s, int ngroups, const SCH& sch, int s0,
                                        bool reduce_output) {
    constexpr int M = 1 << K, SPAN = 1 << LOG_SPAN;
    SF f[K];
    bool fuse[K];
#pragma unroll
    for (int q = 0; q < K; q++) {
        f[q] = sflags(sch, s0 + q);
        fuse[q] = f[q].last && reduce_output;
    }
    for (int gg = tm.tid(); gg < ngroups; gg += tm.size()) {
        const int g = gg >> LOG_SPAN, o = gg & (SPAN - 1);
        const int blk = g & ((1 << LOG_NB) - 1);
        const int swb = sw((g << LOG_GLEN) + o);
        int64_t x[M];
#pragma unroll
        for (int m = 0; m < M; m++) x[m] = el(s, swb, m * SPAN);
        if (INV) inv_group<K, LOG_NB == 0>(c, f, blk, x);
        else fwd_group<K, LOG_NB == 0>(c, f, fuse, blk, x);
#pragma unroll
        for (int m = 0; m < M; m++) el(s, swb, m * SPAN) = x[m];
    }
}

// ---------------------------------------------------------------- lines

/// The Montgomery product of modes 2 and 3: mul_mont for any modulus, its limb form beside the limb
/// Barrett products, and for a mode with bit 2 (6: forward, multipliers in a table of limbs) the
/// product by a constant (mont_const_limbs: 8 multiplications instead of 12). Modes 2 and 11 (3 with bit 3)
/// multiply by the caller's words, which may be any (MontAny).
struct Mont {
    int64_t n, ninv;
    typedef int64_t W;
    __device__ __forceinline__ W load(const int64_t* p, int64_t i) const { return p[i]; }
    __device__ __forceinline__ int64_t mul(int64_t a, W b) const { return mul_mont(a, b, n, ninv); }
};
struct MontL {
    MontLimbs m;
    typedef int64_t W;
    __device__ __forceinline__ W load(const int64_t* p, int64_t i) const { return p[i]; }
    __device__ __forceinline__ int64_t mul(int64_t a, W b) const { return mont_mul(a, b, m); }
};
/// The general product in functions of their own, so that the kernels' registers stay those of the limb product:
/// eight tile elements, STEP apart, and a column x, into global memory.
template <int STEP>
__device__ __noinline__ void mul_mont_tile(int64_t* s, int swb, int64_t* g, const int64_t* mulp, int64_t me, int64_t n, int64_t ninv) {
#pragma unroll 1
    for (int m = 0; m < 8; m++) g[STEP * m] = mul_mont(el(s, swb, STEP * m), mulp[STEP * m * me], n, ninv);
}
template <int N>
__device__ __noinline__ void mul_mont_column(const int64_t* x, int64_t* g, int64_t ge, const int64_t* mulp, int64_t me, int64_t n,
                                             int64_t ninv) {
#pragma unroll 1
    for (int i = 0; i < N; i++) g[i * ge] = mul_mont(x[i], mulp[i * me], n, ninv);
}
/// mont_mul of the caller's words (modes 2 and 11). Its middle limbs hold the product for |a1| + |b1| < 2^31 - 2^27
/// and n < 2^57, and the transforms' results have |a| <= 0.9 x 2^63 in mode 2, |a| <= n in mode 11: a thread that
/// sees other words (out) takes mul_mont for what it holds, the same integer. In mode 2 after the products, so
/// that no product waits for the others' words: the test before them, hal_ntt_mul along dimension 3 of a
/// [24, 34, 12, 3072] tensor 195 -> 207 us, along dimension 2 91 -> 101.
template <int MODE>
struct MontAny {
    MontLimbs m;
    typedef int64_t W;
    __device__ __forceinline__ W load(const int64_t* p, int64_t i) const { return p[i]; }
    __device__ __forceinline__ int64_t mul(int64_t a, W b) const { return mont_mul(a, b, m); }
    /// Of the words seen: mode 2 |b| <= 2^58, mode 11 |b| <= 2^62.
    static constexpr uint32_t HALF = MODE == 2 ? 1u << 26 : 1u << 30;
    __device__ __forceinline__ void see(uint32_t& seen, W b) const { seen |= hi32(b) + HALF; }
    __device__ __forceinline__ bool out(uint32_t seen) const { return seen >= 2 * HALF; }
    __device__ __forceinline__ int64_t n() const { return (int64_t)(((uint64_t)(uint32_t)m.n1 << 32) + (uint64_t)(int64_t)m.n0); }
    __device__ __forceinline__ int64_t ninv() const { return pack64(m.i0, m.i1); }
};
struct MontC {
    BarrettMod m;
    typedef BarrettLimbs W;
    __device__ __forceinline__ W load(const int64_t* p, int64_t i) const {
        return load_limbs(reinterpret_cast<const BarrettLimbs*>(p) + i);
    }
    __device__ __forceinline__ int64_t mul(int64_t a, const W& b) const { return barrett_mul(b, a, m); }
};
template <class CTX, int MODE>
__device__ __forceinline__ auto make_mont(int64_t n, int64_t ninv) {
    if constexpr ((MODE & 4) != 0) return MontC{mont_const_mod(n)};
    else if constexpr (CTX::LIMBS && (MODE == 2 || MODE == 11)) return MontAny<MODE>{mont_limbs(n, ninv)};
    else if constexpr (CTX::LIMBS) return MontL{mont_limbs(n, ninv)};
    else return Mont{n, ninv};
}

/// The multipliers of 4096-residue block blk of a line (words, or limbs of 16 bytes; me = 0: one for all).
template <int MODE>
__device__ __forceinline__ const int64_t* block_multiplier(const int64_t* mulp, int64_t me, int blk) {
    return mulp + me * 4096 * blk * ((MODE & 4) ? 2 : 1);
}

/// Words of the staged twiddles behind a tile: NA entries of the pass before a tail, 63 of the tail.
__host__ __device__ constexpr int staged_words(int na) { return 2 * (na + 63); }
/// Copies the limb twiddles of a line's passes behind its first to shared memory: the `na` entries from
/// stage sa on (a factor's stages, contiguous), and the 63 of the tail's factor 64 (stages sb ..),
/// with the three stages whose blocks differ between lanes ordered by the compile-time part of the
/// block, so that eight lanes' twiddles are neighbours. A 16-byte load through L1 takes the load path
/// eight cycles however few addresses a warp has, a quarter of the line kernels' load cycles in all.
/// Visible after the next barrier.
template <bool INV, class SCH, class TEAM>
__device__ __forceinline__ void stage_tail_twiddles(const TEAM& tm, const CtxL& c, const SCH& sch, int4* dst, int sa, int na,
                                                    int sb) {
    for (int t = tm.tid(); t < na + 63; t += tm.size()) {
        const int e = t - na;
        int at = t;
        if (e >= 0) {
            // stages of 8 2^k entries, block << k | part
            const int k = INV ? (e < 32 ? 2 : e < 48 ? 1 : e < 56 ? 0 : -1) : (e >= 31 ? 2 : e >= 15 ? 1 : e >= 7 ? 0 : -1);
            if (k >= 0) {
                const int base = INV ? (k == 2 ? 0 : k == 1 ? 32 : 48) : (8 << k) - 1, r = e - base;
                at = na + base + 8 * (r & ((1 << k) - 1)) + (r >> k);
            }
        }
        dst[at] = __ldg(c.tw + (e < 0 ? sch.tw(sa) + t : sch.tw(sb) + e));
    }
}
/// A pass's context with its staged twiddles (from stage s0 on, at `at`); general plans keep theirs.
template <class SCH>
__device__ __forceinline__ CtxS staged_ctx(const CtxL& c, const SCH& sch, const int4* at, int s0) {
    return CtxS{c.m, c.il, at - sch.tw(s0)};
}
template <class SCH>
__device__ __forceinline__ const Ctx& staged_ctx(const Ctx& c, const SCH&, const int4*, int) { return c; }

/// The last six stages of a line (a factor 64: distances 32 .. 1 forward, 1 .. 32 inverse; first stage s0)
/// and its way to global memory, multiplying (modes 2 and 3) by mulp[e * me] in Montgomery form.
/// They act within 64 consecutive elements, so each warp takes 256 of them (32 register groups of
/// eight per pass) through both passes and the store with warp barriers only: no block barrier, and
/// no warp waits for another's loads of the multiplier, which are all in flight before the warp turns
/// the forward pass's eight neighbours per lane into coalesced rows through its part of the tile
/// (the inverse pass's lanes hold runs of eight already and store from registers). Against block
/// barriers around each pass and a store loop that loaded its multipliers as it went: pb_to_crt of
/// [24, 23, 4, 12288] 611 -> 561 us, of [24, 34, 12, 3072] 574 -> 557 us.
template <int MODE, class SCH, class CTX, class MONT, class TEAM>
__device__ __forceinline__ void tail64(const TEAM& tm, const CTX& c, int64_t* s, int len, const SCH& sch, int s0, bool reduce_output,
                                       int64_t* g, const int64_t* mulp, int64_t me, const MONT& mont) {
    constexpr bool inv = MODE & 1, mul = MODE & 2;
    SF f[6];
    bool fuse[6];
#pragma unroll
    for (int q = 0; q < 6; q++) {
        f[q] = sflags(sch, s0 + q);
        fuse[q] = f[q].last && reduce_output;
    }
    const int lane = tm.tid() & 31;
    uint32_t seen = 0;  // of the multipliers (MontAny)
    for (int e0 = (tm.tid() >> 5) << 8; e0 < len; e0 += tm.size() << 3) {
        // groups of eight at distance 8 (lane = 8 block + offset), and of eight neighbours
        const int ea = e0 + ((lane >> 3) << 6) + (lane & 7), wa = sw(ea), wb = sw(e0 + (lane << 3));
        int64_t x[8];
        if constexpr (!inv) {
#pragma unroll
            for (int m = 0; m < 8; m++) x[m] = el(s, wa, 8 * m);
            fwd_group<3, true>(c, f, fuse, 0, x);
#pragma unroll
            for (int m = 0; m < 8; m++) el(s, wa, 8 * m) = x[m];
            __syncwarp();
#pragma unroll
            for (int m = 0; m < 8; m++) x[m] = el(s, wb, m);
            fwd_group<3, false, CTX::LIMBS>(c, f + 3, fuse + 3, lane & 7, x);
            constexpr int AHEAD = sizeof(typename MONT::W) == 8 ? 8 : 2;  // multipliers in registers
            typename MONT::W w[AHEAD];
            if (mul) {
#pragma unroll
                for (int m = 0; m < AHEAD; m++) w[m] = mont.load(mulp, (e0 + 32 * m + lane) * me);
            }
#pragma unroll
            for (int m = 0; m < 8; m++) el(s, wb, m) = x[m];
            __syncwarp();
            const int wc = sw(e0 + lane);
#pragma unroll
            for (int m = 0; m < 8; m++) {
                int64_t v = el(s, wc, 32 * m);
                if (mul) {
                    if constexpr (MODE == 2 && CTX::LIMBS) mont.see(seen, w[m]);
                    v = mont.mul(v, w[m % AHEAD]);
                    if (m + AHEAD < 8) w[m % AHEAD] = mont.load(mulp, (e0 + 32 * (m + AHEAD) + lane) * me);
                }
                g[e0 + 32 * m + lane] = v;
            }
        } else {
#pragma unroll
            for (int m = 0; m < 8; m++) x[m] = el(s, wb, m);
            inv_group<3, false, CTX::LIMBS>(c, f, lane & 7, x);
#pragma unroll
            for (int m = 0; m < 8; m++) el(s, wb, m) = x[m];
            __syncwarp();
#pragma unroll
            for (int m = 0; m < 8; m++) x[m] = el(s, wa, 8 * m);
            inv_group<3, true>(c, f + 3, 0, x);
            typename MONT::W w[MODE == 11 ? 8 : 1];
            if constexpr (MODE == 11) {
#pragma unroll
                for (int m = 0; m < 8; m++) w[m] = mont.load(mulp, (ea + 8 * m) * me);
                seen = 0;
#pragma unroll
                for (int m = 0; m < 8; m++) mont.see(seen, w[m]);
                if (mont.out(seen)) {
#pragma unroll
                    for (int m = 0; m < 8; m++) el(s, wa, 8 * m) = x[m];  // the lane's own elements
                    mul_mont_tile<8>(s, wa, g + ea, mulp + ea * me, me, mont.n(), mont.ninv());
                    continue;
                }
            }
#pragma unroll
            for (int m = 0; m < 8; m++) {
                if constexpr (MODE == 11) x[m] = mont.mul(x[m], w[m]);
                else if constexpr (mul) x[m] = mont.mul(x[m], mont.load(mulp, (ea + 8 * m) * me));
                g[ea + 8 * m] = x[m];
            }
        }
    }
    if constexpr (MODE == 2 && CTX::LIMBS) {
        if (mont.out(seen))  // the tile still holds the transform
            for (int e0 = (tm.tid() >> 5) << 8; e0 < len; e0 += tm.size() << 3)
                mul_mont_tile<32>(s, sw(e0 + lane), g + e0 + lane, mulp + (e0 + lane) * me, me, mont.n(), mont.ninv());
    }
}

/// Reduces every element of a register group when the stage asks for it (src/hal/ntt.rs: the
/// reduction pass before a stage whose growth could overflow).
template <int N, class CTX>
__device__ __forceinline__ void red_all(const CTX& c, bool red, int64_t* x) {
    if (red) {
#pragma unroll
        for (int m = 0; m < N; m++) x[m] = red1(c, x[m]);
    }
}

/// [2, 3, 8, 64] line (3072 residues): g -> g, via the tile s (3072 words); tws: the staged twiddles of
/// factors 8 and 64 (limb plans; complete at the first barrier here). MODE as the
/// tile kernel (0 forward, 1 inverse, 2 forward + product, 3 inverse + product); the schedule
/// SCH is that of the programme of MODE's direction. Stages: 0 = factor 2, 1 = factor 3,
/// 2..4 = factor 8, 5..10 = factor 64.
template <int MODE, class SCH, class CTX, class TEAM>
__device__ __forceinline__ void line3072(const TEAM& tm, const SCH& sch, const CTX& c, int64_t* s, const int4* tws, int64_t* g,
                                         const int64_t* mulp, int64_t me, int64_t mn, int64_t mi) {
    constexpr bool inv = MODE & 1, reduce_output = MODE == 0;
    // pass 1: factors 2 (distance 1536) and 3 (distance 512), straight from global memory
    {
        const SF f0 = sflags(sch, 0), f1 = sflags(sch, 1);
        const bool fz0 = f0.last && reduce_output, fz1 = f1.last && reduce_output;
        for (int o = tm.tid(); o < 512; o += tm.size()) {
            const int swb = sw(o);
            int64_t x[2][3];
#pragma unroll
            for (int b = 0; b < 2; b++)
#pragma unroll
                for (int a = 0; a < 3; a++) x[b][a] = g[o + 512 * a + 1536 * b];
            red_all<6>(c, f0.red, &x[0][0]);
            if (!inv) {
#pragma unroll
                for (int a = 0; a < 3; a++) fwd2<true>(c, f0, fz0, 0, 0, x[0][a], x[1][a]);
                red_all<6>(c, f1.red, &x[0][0]);
#pragma unroll
                for (int b = 0; b < 2; b++) fwd3<true>(c, f1, fz1, 0, x[b][0], x[b][1], x[b][2]);
            } else {
#pragma unroll
                for (int a = 0; a < 3; a++) {
                    // factor 2: one block, twiddle 1 unless fused
                    const int64_t sum = wadd(x[0][a], x[1][a]), dif = wsub(x[0][a], x[1][a]);
                    if (f0.last) {
                        x[0][a] = c.scale(sum);
                        x[1][a] = c.scale(dif);
                    } else {
                        x[0][a] = sum;
                        x[1][a] = dif;
                    }
                }
                red_all<6>(c, f1.red, &x[0][0]);
#pragma unroll
                for (int b = 0; b < 2; b++) inv3(c, f1, x[b][0], x[b][1], x[b][2]);
            }
#pragma unroll
            for (int b = 0; b < 2; b++)
#pragma unroll
                for (int a = 0; a < 3; a++) el(s, swb, 512 * a + 1536 * b) = x[b][a];
        }
    }
    tm.sync();
    if (!inv) {
        r2_pass<false, 3, 6, 9, 0>(tm, staged_ctx(c, sch, tws, 2), s, 384, sch, 2, reduce_output);  // factor 8: distances 256, 128, 64
    } else {
        r2_pass<true, 3, 6, 9, 0>(tm, staged_ctx(c, sch, tws, 2), s, 384, sch, 2, false);  // factor 8: distances 64, 128, 256
    }
    tm.sync();
    tail64<MODE>(tm, staged_ctx(c, sch, tws + 7, 5), s, 3072, sch, 5, reduce_output, g, mulp, me,
                 make_mont<CTX, MODE>(mn, mi));  // factor 64
}

/// One of the three 4096-residue blocks of a [3, 64, 64] line, computed by one CTA of a 3-CTA
/// cluster: the factor-3 stage couples the blocks, but each output of a radix-3 butterfly needs
/// only its own two twiddle products, so the CTA of block `blk` reads all three inputs of its
/// positions and computes just its output; the remaining 12 stages act within the block. The
/// line is transformed in place, so no CTA may store before all three have read their inputs:
/// `cluster_sync` (a cluster-wide barrier) separates the first pass from the stores.
template <int MODE, class SCH, class CTX, class SYNC>
__device__ __forceinline__ void line12288_block(const SCH& sch, const CTX& c, int64_t* s, const int4* tws, int64_t* g, int blk,
                                                const int64_t* mulp, int64_t me, int64_t mn, int64_t mi,
                                                SYNC cluster_sync) {
    constexpr bool inv = MODE & 1, reduce_output = MODE == 0;
    {
        SF f[4];
        bool fz[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            f[q] = sflags(sch, q);
            fz[q] = f[q].last && reduce_output;
        }
        // twiddles of the factor-3 stage (one block, whose block twiddles are 1: the inverse
        // outputs take no block-twiddle product, as inv3 explains)
        // forward: the two products of output blk; inverse: zeta, zeta^2
        const int i0 = blk == 0 ? 0 : (blk == 1 ? 1 : 2), i1 = blk == 0 ? 3 : (blk == 1 ? 5 : 4);
        const auto w0 = c.get(inv ? f[0].zeta_off : f[0].tw_off + i0), w1 = c.get(inv ? f[0].zeta_off + 1 : f[0].tw_off + i1);
        constexpr int span = inv ? 64 : 512;
        for (int gg = threadIdx.x; gg < 512; gg += blockDim.x) {
            const int base = inv ? ((gg >> 6) << 9) + (gg & 63) : gg;
            int64_t x[8];
#pragma unroll
            for (int m = 0; m < 8; m++) {
                const int p = base + span * m;
                int64_t a = g[p], b = g[p + 4096], d = g[p + 8192];
                if (f[0].red) {
                    a = red1(c, a);
                    b = red1(c, b);
                    d = red1(c, d);
                }
                int64_t o;
                if (!inv) {
                    // src/hal/ntt.rs:386-406, output blk of the butterfly
                    int64_t tb, tc;
                    if (blk == 0 && f[0].skip_ok) {
                        tb = b;
                        tc = d;
                    } else {
                        tb = c.mul(w0, b);
                        tc = c.mul(w1, d);
                    }
                    o = wadd(wadd(a, tb), tc);
                    if (fz[0]) o = red1(c, o);
                } else {
                    // src/hal/ntt.rs:511-530, output blk of the butterfly
                    if (blk == 0) {
                        o = wadd(wadd(a, b), d);
                    } else if (blk == 1) {
                        o = wadd(wadd(a, c.mul(w1, b)), c.mul(w0, d));
                    } else {
                        o = wadd(wadd(a, c.mul(w0, b)), c.mul(w1, d));
                    }
                    if (f[0].last) o = c.scale(o);
                }
                x[m] = o;
            }
            if (!inv) fwd_group<3, true>(c, f + 1, fz + 1, 0, x);
            else inv_group<3, false>(c, f + 1, gg >> 6, x);
#pragma unroll
            for (int m = 0; m < 8; m++) el(s, sw(base), span * m) = x[m];
        }
    }
    cluster_sync();  // also a barrier of this CTA
    if (!inv) {
        r2_pass<false, 3, 6, 9, 3>(CtaTeam{}, staged_ctx(c, sch, tws, 1), s, 512, sch, 4, reduce_output);  // factor 64 (a): 256, 128, 64
    } else {
        r2_pass<true, 3, 9, 12, 0>(CtaTeam{}, staged_ctx(c, sch, tws, 1), s, 512, sch, 4, false);  // factor 64 (a): 512, 1024, 2048
    }
    __syncthreads();
    tail64<MODE>(CtaTeam{}, staged_ctx(c, sch, tws + 63, 7), s, 4096, sch, 7, reduce_output, g + 4096 * blk, block_multiplier<MODE>(mulp, me, blk), me,
                 make_mont<CTX, MODE>(mn, mi));  // factor 64 (b)
}

/// Stages 1..12 of one 4096-residue block of a [3, 64, 64] line (the two factors 64, which act within the
/// block): g -> g via the tile s; tws: the staged twiddles of both (complete at the first barrier here);
/// mulp: the block's multipliers.
template <int MODE, class SCH, class CTX, class MONT, class TEAM>
__device__ __forceinline__ void block4096(const TEAM& tm, const SCH& sch, const CTX& c, int64_t* s, const int4* tws,
                                          int64_t* g, const int64_t* mulp,
                                          int64_t me, const MONT& mont) {
    constexpr bool inv = MODE & 1, reduce_output = MODE == 0;
    {
        SF f[3];
        bool fz[3];
#pragma unroll
        for (int q = 0; q < 3; q++) {
            f[q] = sflags(sch, 1 + q);
            fz[q] = f[q].last && reduce_output;
        }
        // factor 64 (a): distances 2048, 1024, 512 forward, 64, 128, 256 inverse, straight from global memory
        constexpr int span = inv ? 64 : 512;
        for (int gg = tm.tid(); gg < 512; gg += tm.size()) {
            const int base = inv ? ((gg >> 6) << 9) + (gg & 63) : gg;
            int64_t x[8];
#pragma unroll
            for (int m = 0; m < 8; m++) x[m] = g[base + span * m];
            if (!inv) fwd_group<3, true>(c, f, fz, 0, x);
            else inv_group<3, false>(c, f, gg >> 6, x);
#pragma unroll
            for (int m = 0; m < 8; m++) el(s, sw(base), span * m) = x[m];
        }
    }
    tm.sync();
    if (!inv) {
        r2_pass<false, 3, 6, 9, 3>(tm, staged_ctx(c, sch, tws, 1), s, 512, sch, 4, reduce_output);  // factor 64 (a): 256, 128, 64
    } else {
        r2_pass<true, 3, 9, 12, 0>(tm, staged_ctx(c, sch, tws, 1), s, 512, sch, 4, false);  // factor 64 (a): 512, 1024, 2048
    }
    tm.sync();
    tail64<MODE>(tm, staged_ctx(c, sch, tws + 63, 7), s, 4096, sch, 7, reduce_output, g, mulp, me, mont);  // factor 64 (b)
}

// ---------------------------------------------------------------- columns

/// [4, 3] column (12 residues at element stride ge): factor 4 (distance 3) then factor 3
/// (distance 1). Forward stages: 0 = factor 4 length 4, 1 = factor 4 length 2, 2 = factor 3;
/// inverse stages: 0 = factor 4 length 2, 1 = factor 4 length 4, 2 = factor 3.
template <class CTX>
__device__ __forceinline__ void col12(const CTX& c, const SF* f, bool inv, bool reduce_output, int64_t (&x)[4][3]) {
    if (!inv) {
        if (f[0].red)
#pragma unroll
            for (int a = 0; a < 4; a++)
#pragma unroll
                for (int b = 0; b < 3; b++) x[a][b] = red1(c, x[a][b]);
        const bool z0 = f[0].last && reduce_output, z1 = f[1].last && reduce_output, z2 = f[2].last && reduce_output;
#pragma unroll
        for (int a = 0; a < 2; a++)
#pragma unroll
            for (int b = 0; b < 3; b++) fwd2<true>(c, f[0], z0, 0, 0, x[a][b], x[a + 2][b]);
        if (f[1].red)
#pragma unroll
            for (int a = 0; a < 4; a++)
#pragma unroll
                for (int b = 0; b < 3; b++) x[a][b] = red1(c, x[a][b]);
#pragma unroll
        for (int b = 0; b < 3; b++) {
            fwd2<true>(c, f[1], z1, 0, 0, x[0][b], x[1][b]);
            // block 1: an ordinary twiddle (not 1), product always taken
            const int64_t t = c.mul(c.get(f[1].tw_off + 1), x[3][b]);
            int64_t o0 = wadd(x[2][b], t), o1 = wsub(x[2][b], t);
            if (z1) {
                o0 = red1(c, o0);
                o1 = red1(c, o1);
            }
            x[2][b] = o0;
            x[3][b] = o1;
        }
        if (f[2].red)
#pragma unroll
            for (int a = 0; a < 4; a++)
#pragma unroll
                for (int b = 0; b < 3; b++) x[a][b] = red1(c, x[a][b]);
#pragma unroll
        for (int a = 0; a < 4; a++) fwd3<true>(c, f[2], z2, 0, x[a][0], x[a][1], x[a][2]);
    } else {
        if (f[0].red)
#pragma unroll
            for (int a = 0; a < 4; a++)
#pragma unroll
                for (int b = 0; b < 3; b++) x[a][b] = red1(c, x[a][b]);
#pragma unroll
        for (int b = 0; b < 3; b++) {
            // factor 4, length-2 stage: block 0 (pair 0, 1) and block 1 (pair 2, 3)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int64_t sum = wadd(x[2 * h][b], x[2 * h + 1][b]), dif = wsub(x[2 * h][b], x[2 * h + 1][b]);
                if (f[0].last) {
                    x[2 * h][b] = c.scale(sum);
                    x[2 * h + 1][b] = c.scale(dif);
                } else if (h == 0) {
                    x[0][b] = sum;
                    x[1][b] = dif;
                } else {
                    x[2][b] = sum;
                    x[3][b] = c.mul(c.get(f[0].tw_off + 1), dif);  // block 1's twiddle, never 1
                }
            }
        }
        if (f[1].red)
#pragma unroll
            for (int a = 0; a < 4; a++)
#pragma unroll
                for (int b = 0; b < 3; b++) x[a][b] = red1(c, x[a][b]);
#pragma unroll
        for (int a = 0; a < 2; a++)
#pragma unroll
            for (int b = 0; b < 3; b++) {
                const int64_t sum = wadd(x[a][b], x[a + 2][b]), dif = wsub(x[a][b], x[a + 2][b]);
                if (f[1].last) {
                    x[a][b] = c.scale(sum);
                    x[a + 2][b] = c.scale(dif);
                } else {
                    x[a][b] = sum;
                    x[a + 2][b] = dif;
                }
            }
        if (f[2].red)
#pragma unroll
            for (int a = 0; a < 4; a++)
#pragma unroll
                for (int b = 0; b < 3; b++) x[a][b] = red1(c, x[a][b]);
#pragma unroll
        for (int a = 0; a < 4; a++) inv3(c, f[2], x[a][0], x[a][1], x[a][2]);
    }
}

/// [4] column (4 residues): forward stages 0 = length 4, 1 = length 2; inverse the reverse.
template <class CTX>
__device__ __forceinline__ void col4(const CTX& c, const SF* f, bool inv, bool reduce_output, int64_t (&x)[4]) {
    if (!inv) {
        if (f[0].red)
#pragma unroll
            for (int a = 0; a < 4; a++) x[a] = red1(c, x[a]);
        const bool z0 = f[0].last && reduce_output, z1 = f[1].last && reduce_output;
        fwd2<true>(c, f[0], z0, 0, 0, x[0], x[2]);
        fwd2<true>(c, f[0], z0, 0, 0, x[1], x[3]);
        if (f[1].red)
#pragma unroll
            for (int a = 0; a < 4; a++) x[a] = red1(c, x[a]);
        fwd2<true>(c, f[1], z1, 0, 0, x[0], x[1]);
        const int64_t t = c.mul(c.get(f[1].tw_off + 1), x[3]);
        int64_t o0 = wadd(x[2], t), o1 = wsub(x[2], t);
        if (z1) {
            o0 = red1(c, o0);
            o1 = red1(c, o1);
        }
        x[2] = o0;
        x[3] = o1;
    } else {
        if (f[0].red)
#pragma unroll
            for (int a = 0; a < 4; a++) x[a] = red1(c, x[a]);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int64_t sum = wadd(x[2 * h], x[2 * h + 1]), dif = wsub(x[2 * h], x[2 * h + 1]);
            if (f[0].last) {
                x[2 * h] = c.scale(sum);
                x[2 * h + 1] = c.scale(dif);
            } else if (h == 0) {
                x[0] = sum;
                x[1] = dif;
            } else {
                x[2] = sum;
                x[3] = c.mul(c.get(f[0].tw_off + 1), dif);
            }
        }
        if (f[1].red)
#pragma unroll
            for (int a = 0; a < 4; a++) x[a] = red1(c, x[a]);
#pragma unroll
        for (int a = 0; a < 2; a++) {
            const int64_t sum = wadd(x[a], x[a + 2]), dif = wsub(x[a], x[a + 2]);
            if (f[1].last) {
                x[a] = c.scale(sum);
                x[a + 2] = c.scale(dif);
            } else {
                x[a] = sum;
                x[a + 2] = dif;
            }
        }
    }
}

}  // namespace fast
