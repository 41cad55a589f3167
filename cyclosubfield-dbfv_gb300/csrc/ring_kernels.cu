// Fused ring-level kernels. Each replaces a sequence of Backend calls of the reference's ring /
// BFV layer with one pass over the data, computing exactly the same integers:
//  - bconv_fused_kernel: BEHZ base conversion, plain (BConvCache::bconv,
//    cyclosubfield-dbfv/src/ring.rs:1663-1701) and gadget-batched (GadgetBConvCache::bconv,
//    src/ring.rs:1809-1851): mul_mont64 by (q/p)^-1, the small-K matmul (exact, in 29-bit limbs),
//    the double reduction, the q~-scaled correction and the conversion to Montgomery form, without
//    the i128 `tmp` / `correction` tensors ever reaching HBM.
//  - galois_kernel: both permutation passes of apply_galois (src/ring.rs:1212-1222) as one gather.
//  - keyswitch_async_kernel (keyswitch1_kernel for odd or unaligned views): the key-switch inner
//    product, the addition of c0 / c1 through mont(1) and reduce_wide (src/bfv.rs:498-556,
//    src/ring.rs:460-485, :503-509, :846-865).
//  - tensor_kernel: hom_mul_raw_acc + reduce_wide (src/bfv.rs:667-683).
//  - giant_kernel: one giant step of the homomorphic CRT transform for up to four output digits:
//    the baby-step inner product over the digit convolution (dbfv_acc_inner_product_element_lprime,
//    src/dbfv.rs:291-399), the addition of the carried result (dbfv_acc_add, :153-163) and the
//    reduction (dbfv_finish_accumulator, :401-404), without the wide accumulator in HBM.
#include <algorithm>
#include <cstring>

#include "limb_sum.cuh"

namespace {

constexpr int BCONV_THREADS = 128;

struct BconvArgs {
    KView src;  // [ns, r, dl, dk]
    KView dst;  // [ns * nb, rd, dl, dk]
    BconvConsts c;
    int r, rd, nb;
    int ochunk;  // outputs per CTA (even): blockIdx.z selects the outputs [z ochunk, (z + 1) ochunk)
    int64_t npos;
    const BarrettLimbs* sub_mul;  // optional [rd]: store mul_mont(dst - v, b_j) instead of v
};

/// The conversion matrix as a kernel parameter (BconvConsts::hmat), read as uniform constants that never
/// pass the load path: up to 1152 entries (9 KB: bases of 33 factors; field_49152 r = 23 has 552); one
/// entry: the matrix is read from memory (mat2).
template <int N>
struct BconvMatrix {
    static constexpr int ENTRIES = N;
    int2 m[N];
};
typedef BconvMatrix<1152> BconvParam;
typedef BconvMatrix<96> BconvSmall;  // a launch copies its parameters: two field_18 rows 7.9 us with these, 8.2 with all
typedef BconvMatrix<1> BconvMemory;

constexpr int LIMB_UNROLL = 16;  // terms unrolled together

/// Multiply-accumulate of O output rows (r limb pairs each, consecutive from m) over the lifts u in
/// [lo, hi): the exact sums sum_u m_u x_u (|x| < 2^57, |m| < 2^56) as 128-bit words h:l.
/// N terms (n of them valid) into the column sums.
template <int O, int N, bool PARAM>
__device__ __forceinline__ void limb_terms(const int2* __restrict__ xp, const int2* __restrict__ m, int r, int n,
                                           LimbSum (&s)[O]) {
#pragma unroll
    for (int t = 0; t < N; t++) {
        if (N == LIMB_UNROLL || t < n) {
            const int2 x = xp[t * BCONV_THREADS];
            const int xs = x.x + x.y;
#pragma unroll
            for (int o = 0; o < O; o++) {
                const int2 w = PARAM ? m[o * r + t] : __ldg(m + o * r + t);
                s[o].mac(x, xs, w, w.x + w.y);
            }
        }
    }
}
template <int O, bool PARAM>
__device__ __forceinline__ void limb_mac(const int2* __restrict__ xcol, const int2* __restrict__ m, int r, int lo, int hi,
                                         uint64_t (&l)[O], int64_t (&h)[O]) {
#pragma unroll
    for (int o = 0; o < O; o++) l[o] = 0, h[o] = 0;
    for (int g0 = lo; g0 < hi; g0 += LIMB_TERMS) {
        const int n = min(LIMB_TERMS, hi - g0);
        LimbSum s[O];
#pragma unroll
        for (int o = 0; o < O; o++) s[o].zero();
        const int2* xp = xcol + g0 * BCONV_THREADS;
        // sixteen terms fully unrolled (every address an immediate offset), the rest in steps of four
        int t = 0;
        if (n >= LIMB_UNROLL) limb_terms<O, LIMB_UNROLL, PARAM>(xp, m + g0, r, n, s), t = LIMB_UNROLL;
        for (; t < n; t += 4) limb_terms<O, 4, PARAM>(xp + t * BCONV_THREADS, m + g0 + t, r, n - t, s);
#pragma unroll
        for (int o = 0; o < O; o++) s[o].fold(l[o], h[o]);
    }
}

/// The conversion's epilogue for output j of block b: v (the double-reduced sums) plus the
/// correction mul_mont(q, qmodp), to Montgomery form, optionally dst <- mul_mont(dst - y, b_j).
template <bool SUB>
__device__ __forceinline__ void bconv_store(const BconvArgs& a, const KMods& dm, int b, int j, int64_t q, int64_t v,
                                            int64_t* p, int64_t old) {
    const int64_t n = dm.n[j], ninv = dm.ninv[j];
    const int64_t* qt = a.c.qtab + (b * a.rd + j) * (2 * a.c.qhalf + 1) + a.c.qhalf;
    const int64_t qm = (q >= -a.c.qhalf && q <= a.c.qhalf) ? __ldg(qt + q)
                                                            : mul_mont(q, a.c.qmodp[b * a.rd + j], n, ninv);
    const BarrettMod mm = mont_const_mod(n);
    const int64_t y = barrett_mul(load_limbs(a.c.r2 + j), wadd(v, qm), mm);  // to_mont64
    if constexpr (SUB)
        *p = barrett_mul(load_limbs(a.sub_mul + j), wsub(old, y), mm);
    else
        *p = y;
}

/// Outputs j .. j + O - 1 of the conversion (dst row j at d + j * s1).
template <bool ONE_CHUNK, bool SUB, int O, class MAT>
__device__ __forceinline__ void bconv_outputs(const BconvArgs& a, const KMods& dm, int b, int j, int u0, int u1,
                                              const int2* xcol, int64_t q, int64_t* d, const MAT& mx) {
    constexpr bool PARAM = MAT::ENTRIES > 1;
    const int stride = PARAM ? u1 - u0 : a.r;
    const int2* m = PARAM ? mx.m + u0 * a.rd + j * stride - u0 : a.c.mat2 + ((int64_t)b * a.rd + j) * a.r;
    // the subtract-and-multiply store's operands, loaded before the sums so that their latency hides
    // behind the multiply-accumulate
    int64_t old[O] = {}, v[O] = {};
    if constexpr (SUB) {
#pragma unroll
        for (int o = 0; o < O; o++) old[o] = d[(j + o) * a.dst.s1];
    }
    // the reference's chunked matmul (src/ring.rs:1678-1691) splits the columns into chunks of `chunk` (one
    // chunk whenever r <= chunk, which holds for all 57-bit bases up to 8192 factors) and
    // double-reduces each chunk's sum
    uint64_t l[O];
    int64_t h[O];
    bool first = true;
    for (int c0 = 0; ONE_CHUNK ? first : c0 < a.r; c0 += a.c.chunk) {
        const int lo = ONE_CHUNK ? u0 : max(c0, u0), hi = ONE_CHUNK ? u1 : min(min(c0 + a.c.chunk, a.r), u1);
        limb_mac<O, PARAM>(xcol, m, stride, lo, hi, l, h);
#pragma unroll
        for (int o = 0; o < O; o++) {
            const int64_t r = mont_red_double(l[o], h[o], mont_limbs(dm.n[j + o], dm.ninv[j + o]));
            v[o] = first ? r : wadd(v[o], r);
        }
        first = false;
    }
#pragma unroll
    for (int o = 0; o < O; o++) bconv_store<SUB>(a, dm, b, j + o, q, v[o], d + (j + o) * a.dst.s1, old[o]);
}

/// BEHZ base conversion of one position per thread (BConvCache::bconv, src/ring.rs:1660-1702, and the
/// gadget form of :1800-1852). CTA (x, y, z): 128 positions of source row y / nb, output block y % nb
/// (a gadget digit), outputs [z ochunk, (z + 1) ochunk) of the block; only the block's own source
/// columns are lifted. The products with the conversion matrix use its limb form: the shared array
/// holds each lift as its limb pair (x mod 2^29, x >> 29).
/// What bounds it: the multiply pipe, near 0.9 of its products' time ([24, 16 -> 18] of field_36864 134 us, 119 for
/// 441 cycles of lifts and 18 times 277 of sums and reductions per warp). Each lane's copy of a matrix
/// entry from memory takes the load path as long as a lift does, so a thread holds four output rows (one
/// lift and four 8-byte entries for twelve wide products, the entries' limb sums formed, not read), and
/// matrices that fit come as kernel parameters (BconvMatrix). Two rows and 16-byte entries: 75 % of the load path
/// busy beside 67 % of the multiply pipe, [2, 16 -> 18] 32 us against 24, [6, 23 -> 24] of field_49152 160 against
/// 130; the parameters on top: a field_49152 r = 23 ct-mult 813 -> 788 us, batched r = 16 of field_36864 2769 -> 2744. Two
/// positions per thread take 128 registers and gain nothing.
/// ONE_CHUNK: the block's columns form one chunk of the reference's chunked matmul (always for 57-bit
/// primes); SUB: rescale's subtract-and-multiply store (BconvArgs::sub_mul).
template <bool ONE_CHUNK, bool SUB, class MAT>
__global__ void __launch_bounds__(BCONV_THREADS, 5) bconv_fused_kernel(BconvArgs a, KMods sm, KMods dm, const __grid_constant__ MAT mx) {
    grid_wait();
    extern __shared__ int2 xs[];  // [r][BCONV_THREADS]
    const int b = (int)(blockIdx.y % (unsigned)a.nb);
    const int64_t i = blockIdx.y / (unsigned)a.nb;
    const int jbeg = (int)blockIdx.z * a.ochunk, jend = min(a.rd, jbeg + a.ochunk);
    const int u0 = a.c.ucol[2 * b], u1 = a.c.ucol[2 * b + 1];
    const int64_t pos = (int64_t)blockIdx.x * BCONV_THREADS + threadIdx.x;
    if (pos >= a.npos) return;
    const int64_t k = pos / a.src.n3, l = pos - k * a.src.n3;
    const int64_t* srcp = kat<int64_t>(a.src, i, 0, k, l);  // row u at u * src.s1
    int64_t* dstp = kat<int64_t>(a.dst, i * a.nb + b, 0, k, l);          // row j at j * dst.s1
    // the source is multiplied by (Q/p)^-1 in Montgomery form, giving plain lifts in (-p, p); the source's words are
    // the caller's, and those beyond the limb product's range (64 p of a prime just below 2^57 is the whole
    // word) are lifted by the general product, in a second pass over the columns of a thread that met one
    bool beyond = false;
    for (int u = u0; u < u1; u++) {
        const int64_t w = srcp[u * a.src.s1];
        beyond = beyond || !limb_range(w);
        xs[u * BCONV_THREADS + threadIdx.x] = limb_split(barrett_mul(load_limbs(a.c.qinv + u), w, mont_const_mod(sm.n[u])));
    }
    if (beyond)
        for (int u = u0; u < u1; u++) {
            const int64_t w = srcp[u * a.src.s1], n = sm.n[u];
            if (!limb_range(w))
                xs[u * BCONV_THREADS + threadIdx.x] = limb_split(mul_mont(w, mont_const_value(load_limbs(a.c.qinv + u), n), n, sm.ninv[u]));
        }
    const i128 half = (i128)1 << (a.c.shift - 1);
    const int2* xcol = xs + threadIdx.x;  // this thread's lifts, stride BCONV_THREADS
    const int64_t* __restrict__ mq = a.c.mat + ((int64_t)b * (a.rd + 1) + a.rd) * a.r;
    // the correction q = round(sum_u x_u round(2^shift / p_u) / 2^shift)
    i128 corr;
    if (a.c.corr_limb) {
        int64_t c0 = 0, c1 = 0;
#pragma unroll 4
        for (int u = u0; u < u1; u++) {
            const int2 x = xcol[u * BCONV_THREADS];
            const int m = (int)__ldg(mq + u);
            c0 = mad_wide(x.x, m, c0);
            c1 = mad_wide(x.y, m, c1);
        }
        corr = (i128)c0 + (i128)((u128)(i128)c1 << LIMB_BITS);
    } else {
        corr = 0;
        for (int u = u0; u < u1; u++) {
            const int2 x = xcol[u * BCONV_THREADS];
            const int64_t lift = (int64_t)x.y * ((int64_t)1 << LIMB_BITS) + x.x;
            corr = (i128)((u128)corr + (u128)((i128)__ldg(mq + u) * (i128)lift));
        }
    }
    const int64_t q = (int64_t)((i128)((u128)corr + (u128)half) >> a.c.shift);
    int j = jbeg;
    for (; j + 4 <= jend; j += 4) bconv_outputs<ONE_CHUNK, SUB, 4>(a, dm, b, j, u0, u1, xcol, q, dstp, mx);
    if (j + 2 <= jend) bconv_outputs<ONE_CHUNK, SUB, 2>(a, dm, b, j, u0, u1, xcol, q, dstp, mx), j += 2;
    if (j < jend) bconv_outputs<ONE_CHUNK, SUB, 1>(a, dm, b, j, u0, u1, xcol, q, dstp, mx);
}

/// A sum of at most HC_MAX_TERMS + 1 products of words within 2p: reduced once, or twice and back to
/// Montgomery form.
__device__ __forceinline__ int64_t finish_wide(uint64_t lo, int64_t hi, bool full, const MontLimbs& m, int64_t r2) {
    return full ? mont_mul(mont_red_double(lo, hi, m), r2, m) : mont_red(lo, hi, m);
}

/// Whether words went beyond the range of the limb sums, |y| <= 2^58 (LIMB_TERMS2): the caller's keys and
/// ciphertexts may be unreduced. Three instructions for two words; a thread that met such a word forms its
/// sums again in 128 bits.
struct WordRange {
    uint32_t seen = 0;
    __device__ __forceinline__ void see(int64_t y0, int64_t y1) {
        seen |= (hi32(y0) + (1u << 26)) | (hi32(y1) + (1u << 26));
    }
    __device__ __forceinline__ bool beyond() const { return (seen >> 27) != 0; }
};

/// finish_wide of any sum, also where lo and hi wrapped.
__device__ __noinline__ int64_t finish_any(uint64_t lo, int64_t hi, bool full, int64_t n, int64_t ninv, int64_t r2) {
    const i128 v = (i128)(((u128)(uint64_t)hi << 64) | lo);
    return full ? to_mont64(double_red128(v, n, ninv), n, ninv, r2) : red128(v, n, ninv);
}

/// One digit of the dBFV reduction at one position per thread (dbfv_reduce, src/dbfv.rs:968-1032, with
/// split_overflow, :891-950): rows x <- reduce(x mont(1) + sum_k carry_k Delta_k) when a carry comes in,
/// then the overflow of x modulo Q as limbs (lifts, the matrix sums, the power-of-two correction of
/// src/hal/cpu.rs:983-1057), then x <- reduce(x mont(1) + sum_k overflow_k (-b Delta)_k). The position's
/// words stay in shared memory between the three, and the overflow replaces the carry.
/// What bounds it: the multiply pipe, about 100 wide products per word. As the calls of the tensor HAL a digit took
/// 10 to 17 launches and wrote its lifts, 128-bit sums and accumulators to memory: a product of two
/// three-digit ciphertexts at field_49152 r = 16 took 2617 us and takes 2117 (26 to 37 us per digit here).
/// src [c, r, dl, dk] (p null: zeros) to x, carry [c, limbs, dl, dk] in place; CTAs over (128 positions, row).
__global__ void __launch_bounds__(BCONV_THREADS) dbfv_split_kernel(KView x, KView src, KView carry, DbfvSplit d, int r,
                                                                   KMods m, int64_t npos) {
    grid_wait();
    extern __shared__ __align__(16) int64_t sx[];  // [r][BCONV_THREADS]
    const int64_t pos = (int64_t)blockIdx.x * BCONV_THREADS + threadIdx.x;
    if (pos >= npos) return;
    const int64_t i = blockIdx.y, k = pos / x.n3, l = pos - k * x.n3;
    int64_t* xp = kat<int64_t>(x, i, 0, k, l);
    const int64_t* sp = src.p ? kat<int64_t>(src, i, 0, k, l) : nullptr;
    int64_t* cp = kat<int64_t>(carry, i, 0, k, l);
    auto fma = [](i128 acc, int64_t a, int64_t b) { return (i128)((u128)acc + (u128)((i128)a * (i128)b)); };
    auto finish = [&](i128 acc, int j, bool full) {
        return finish_wide((uint64_t)acc, (int64_t)(acc >> 64), full, mont_limbs(m.n[j], m.ninv[j]), m.r2[j]);
    };
    int64_t c[2] = {0, 0};
    if (d.have_carry)
        for (int q = 0; q < d.limbs; q++) c[q] = cp[q * carry.s1];
    // the sums modulo 2^128; one limb only needs them modulo 2^64 (log2m <= 62)
    i128 v = 0, corr = 0;
    uint64_t v64 = 0;
    int64_t c0 = 0, c1 = 0;
    const int64_t* mq = d.mat + d.limbs * r;
    for (int u = 0; u < r; u++) {
        int64_t w = sp ? sp[u * src.s1] : 0;
        if (d.have_carry) {
            i128 acc = (i128)w * (i128)__ldg(d.one + u);
            for (int q = 0; q < d.limbs; q++) acc = fma(acc, c[q], __ldg(d.delta[q] + u));
            w = finish(acc, u, d.full_in);
        }
        sx[u * BCONV_THREADS + threadIdx.x] = w;
        const int64_t lift = mul_mont(w, __ldg(d.rqinv + u), m.n[u], m.ninv[u]);  // w: any word the bound allows
        if (d.limbs == 1) v64 += (uint64_t)__ldg(d.mat + u) * (uint64_t)lift;
        else v = (i128)((u128)fma(v, __ldg(d.mat + u), lift) + ((u128)((uint64_t)__ldg(d.mat + r + u) * (uint64_t)lift) << 64));
        if (d.corr_limb) {
            const int2 y = limb_split(lift);
            const int g = (int)__ldg(mq + u);
            c0 = mad_wide(y.x, g, c0);
            c1 = mad_wide(y.y, g, c1);
        } else {
            corr = fma(corr, __ldg(mq + u), lift);
        }
    }
    if (d.corr_limb) corr = (i128)c0 + (i128)((u128)(i128)c1 << LIMB_BITS);
    const i128 quot = (i128)((u128)corr + ((u128)1 << (d.shift - 1))) >> d.shift;
    int64_t o[2] = {0, 0};
    if (d.limbs == 1) {
        const uint64_t y = (v64 - (uint64_t)quot * (uint64_t)d.f0) * (uint64_t)d.f1;
        const int64_t mod = (int64_t)1 << d.log2m, red = (int64_t)(y & (uint64_t)(mod - 1));
        o[0] = red > mod / 2 ? red - mod : red;
    } else {
        const u128 y = ((u128)v - (u128)quot * (u128)d.f0) * (u128)d.f1;
        const i128 mod = (i128)1 << d.log2m, red = (i128)(y & ((u128)mod - 1));
        const i128 e = red > mod / 2 ? red - mod : red;
        o[0] = (int64_t)(uint64_t)e;
        o[1] = (int64_t)((e - (i128)o[0]) >> 64);
    }
    for (int q = 0; q < d.limbs; q++) cp[q * carry.s1] = o[q];
    for (int u = 0; u < r; u++) {
        i128 acc = (i128)sx[u * BCONV_THREADS + threadIdx.x] * (i128)__ldg(d.one + u);
        for (int q = 0; q < d.limbs; q++) acc = fma(acc, o[q], __ldg(d.nbd[q] + u));
        xp[u * x.s1] = finish(acc, u, d.full_out);
    }
}

/// dst[i,j,k,l] = src[i,j,p2[k],p3[l]]
__global__ void __launch_bounds__(256) galois_kernel(KView d, KView s, const uint32_t* p2, const uint32_t* p3,
                                                     int64_t lines, int chunks) {
    grid_wait();
    const int64_t tiles = lines * chunks;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        int64_t line = tile / chunks;
        int64_t l = (tile - line * chunks) * blockDim.x + threadIdx.x;
        if (l >= d.n3) continue;
        int64_t k = line % d.n2, r = line / d.n2;
        int64_t j = r % d.n1, i = r / d.n1;
        *kat<int64_t>(d, i, j, k, l) = *kat<int64_t>(s, i, j, p2[k], p3[l]);
    }
}

// Asynchronous global -> shared copies (cp.async): a thread's copies complete in the order of its
// commit groups, and wait_group N returns once at most N of its groups are still in flight. All clobber memory: a
// slot's reads stay behind its wait and in front of the next copy into it.
__device__ __forceinline__ void cp_async8(int64_t* smem, const int64_t* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

struct KsArgs {
    KView parts[HC_MAX_TERMS];  // [B, r, dl, dk] digit t of each of the B ciphertexts (row stride: s0)
    KView keys[HC_MAX_TERMS];   // [2, r, dl, dk] key t restricted to the ciphertext base
    int nterms;
    int64_t batch;              // B; output rows 2i, 2i+1 and summand rows i belong to ciphertext i
    KView add0, add1;  // optional (has_add*) CRT-basis summands of rows 0 / 1, multiplied by mont(1)
    int has_add0, has_add1;
    int full0, full1;  // rows needing the full double reduction
    KView dst;         // [2B, r, dl, dk], its pointer group.dst
    KsGroup group;
    // tiles in reverse order: a launch that follows one over the same parts and summands starts
    // on the tiles that launch read last, which are still in L2
    int reverse;
};

/// R accumulators of one position: one digit word times R key words per step.
template <int R>
struct KsAcc {
    LimbSum s[R];
    uint64_t lo[R];
    int64_t hi[R];
    __device__ __forceinline__ void start() {
#pragma unroll
        for (int q = 0; q < R; q++) s[q].zero(), lo[q] = 0, hi[q] = 0;
    }
    __device__ __forceinline__ void add(int64_t x, const int64_t (&y)[R]) {
        const int2 v = limb_split(x);
#pragma unroll
        for (int q = 0; q < R; q++) {
            const int2 w = limb_split(y[q]);
            s[q].mac(v, v.x + v.y, w, w.x + w.y);
        }
    }
    /// A summand's product, after the fold: in 128 bits, as c0 and c1 are the caller's and may be lazy sums of any
    /// size, while the limbs hold words up to 2^60 only. Once per output word; it costs what the limb product did.
    __device__ __forceinline__ void add_wide(int q, int64_t x, int64_t y) {
        const u128 v = (((u128)(uint64_t)hi[q] << 64) | lo[q]) + (u128)((i128)x * (i128)y);
        lo[q] = (uint64_t)v, hi[q] = (int64_t)(v >> 64);
    }
    __device__ __forceinline__ void fold() {
#pragma unroll
        for (int q = 0; q < R; q++) s[q].fold(lo[q], hi[q]), s[q].zero();
    }
};

__global__ void __launch_bounds__(256) keyswitch1_kernel(KsArgs a, KMods m, const int64_t* one, int64_t lines,
                                                        int chunks) {
    grid_wait();
    const int64_t tiles = lines * chunks;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        int64_t line = tile / chunks;  // (j, k)
        int64_t l = (tile - line * chunks) * blockDim.x + threadIdx.x;
        if (l >= a.dst.n3) continue;
        int64_t k = line % a.dst.n2, r = line / a.dst.n2;
        int64_t j = r % a.dst.n1, i = r / a.dst.n1;
        const int64_t sk = a.group.p2[0] ? (int64_t)a.group.p2[0][k] : k, sl = a.group.p3[0] ? (int64_t)a.group.p3[0][l] : l;
        KsAcc<2> acc;
        WordRange range;
        acc.start();
        for (int t = 0; t < a.nterms; t++) {
            const int64_t x = *kat<int64_t>(a.parts[t], i, j, sk, sl);
            const int64_t y[2] = {*kat<int64_t>(a.keys[t], 0, j, k, l), *kat<int64_t>(a.keys[t], 1, j, k, l)};
            range.see(y[0], y[1]);
            acc.add(x, y);
            if ((t + 1) % (LIMB_TERMS2 - 1) == 0) acc.fold();
        }
        acc.fold();
        if (range.beyond()) {
            acc.start();
            for (int t = 0; t < a.nterms; t++) {
                const int64_t x = *kat<int64_t>(a.parts[t], i, j, sk, sl);
                for (int q = 0; q < 2; q++) acc.add_wide(q, x, *kat<int64_t>(a.keys[t], q, j, k, l));
            }
        }
        const int64_t o = one[j];
        if (a.has_add0) acc.add_wide(0, *kat<int64_t>(a.add0, i, j, sk, sl), o);
        if (a.has_add1) acc.add_wide(1, *kat<int64_t>(a.add1, i, j, sk, sl), o);
        const MontLimbs ml = mont_limbs(m.n[j], m.ninv[j]);
        *kat<int64_t>(a.dst, 2 * i, j, k, l) = finish_wide(acc.lo[0], acc.hi[0], a.full0, ml, m.r2[j]);
        *kat<int64_t>(a.dst, 2 * i + 1, j, k, l) = finish_wide(acc.lo[1], acc.hi[1], a.full1, ml, m.r2[j]);
    }
}

/// The key-switch inner product with two adjacent positions l, l + 1 per thread: the keys and the
/// output are read and written as 16-byte pairs (dimension 3 is contiguous and even), the parts
/// and summands gathered singly (through the automorphism's permutation when one is fused). The
/// terms' reads (the two digit words and the two key pairs of each gadget digit) are staged
/// through shared memory by asynchronous copies, KS_STAGES digits ahead of the products, so that
/// the reads in flight do not occupy registers; each thread copies and reads only its own slots
/// (no barrier). Tiles run as ((j, k), chunk, i) with the ciphertext index innermost: the B tiles
/// that read one block of the key are adjacent, so the key comes from DRAM once and B - 1 reads
/// hit L2.
/// A launch takes up to KS_GROUP keys over the same digits (a keyset's automorphisms), factor by factor, so
/// that a factor's digits (7 MB for three field_49152 ciphertexts of six) come from DRAM once for all of them: the
/// homomorphic CRT step at r = 23 (12 keys) 4979 -> 4892 us, at r = 12 with 40 coefficients 636 -> 604.
/// COMMON: every term's digit view shares the strides of parts[0] and every key view those of
/// keys[0] (the layouts the ring layer passes), so each thread forms its offsets once and a term's
/// addresses are one addition each.
constexpr int KS_STAGES = 3;

/// FOLD: more digits than the column sums hold (LIMB_TERMS2), folded into 128-bit sums on the way.
template <bool COMMON, bool FOLD>
__global__ void __launch_bounds__(256, 4) keyswitch_async_kernel(KsArgs a, KMods m, const int64_t* one,
                                                                 int64_t lines, int chunks) {
    grid_wait();
    __shared__ int64_t sx[KS_STAGES][2][256];
    __shared__ longlong2 skey[KS_STAGES][2][256];
    const int tid = threadIdx.x;
    const uint32_t tiles = (uint32_t)lines * (uint32_t)chunks * (uint32_t)a.group.n;
    const uint32_t per = (uint32_t)a.batch * (uint32_t)a.dst.n2 * (uint32_t)chunks;  // tiles of one factor under one key
    for (uint32_t t0 = blockIdx.x; t0 < tiles; t0 += gridDim.x) {
        const uint32_t tile = a.reverse ? tiles - 1 - t0 : t0;
        const uint32_t j = tile / (per * (uint32_t)a.group.n), e = tile - j * per * (uint32_t)a.group.n;
        const uint32_t key = e / per, w = e - key * per;
        const uint32_t u = w / (uint32_t)a.batch, i = w - u * (uint32_t)a.batch;
        const uint32_t k = u / (uint32_t)chunks;
        const int64_t l = 2 * (int64_t)((u - k * (uint32_t)chunks) * blockDim.x + tid);
        if (l >= a.dst.n3) continue;
        const uint32_t* p2 = a.group.p2[key];
        const uint32_t* p3 = a.group.p3[key];
        const int64_t sk = p2 ? (int64_t)p2[k] : k;
        const int64_t sl0 = p3 ? (int64_t)p3[l] : l, sl1 = p3 ? (int64_t)p3[l + 1] : l + 1;
        // COMMON offsets (in words) of this thread's digit words and key pairs within every term
        const KView& P = a.parts[0];
        const KView& K = a.keys[0];
        const int64_t po = i * P.s0 + j * P.s1 + sk * P.s2, po0 = po + (P.b3 ? 0 : sl0), po1 = po + (P.b3 ? 0 : sl1);
        const int64_t ko0 = j * K.s1 + k * K.s2 + l + a.group.off[key], ko1 = ko0 + K.s0;
        auto issue = [&](int t) {
            if (t < a.nterms) {
                const int s = t % KS_STAGES;
                if (COMMON) {
                    const int64_t* pp = reinterpret_cast<const int64_t*>(a.parts[t].p);
                    const int64_t* kp = reinterpret_cast<const int64_t*>(a.keys[t].p);
                    cp_async8(&sx[s][0][tid], pp + po0);
                    cp_async8(&sx[s][1][tid], pp + po1);
                    cp_async16(&skey[s][0][tid], kp + ko0);
                    cp_async16(&skey[s][1][tid], kp + ko1);
                } else {
                    cp_async8(&sx[s][0][tid], kat<int64_t>(a.parts[t], i, j, sk, sl0));
                    cp_async8(&sx[s][1][tid], kat<int64_t>(a.parts[t], i, j, sk, sl1));
                    cp_async16(&skey[s][0][tid], kat<int64_t>(a.keys[t], 0, j, k, l) + a.group.off[key]);
                    cp_async16(&skey[s][1][tid], kat<int64_t>(a.keys[t], 1, j, k, l) + a.group.off[key]);
                }
            }
            cp_async_commit();  // an empty group past the end keeps the count uniform
        };
#pragma unroll
        for (int t = 0; t < KS_STAGES - 1; t++) issue(t);
        KsAcc<2> acc0, acc1;  // rows 0, 1 of the two positions
        WordRange range;
        acc0.start(), acc1.start();
        for (int t = 0; t < a.nterms; t++) {
            issue(t + KS_STAGES - 1);
            cp_async_wait<KS_STAGES - 1>();  // digit t's group has landed
            const int s = t % KS_STAGES;
            const longlong2 k0 = skey[s][0][tid], k1 = skey[s][1][tid];
            const int64_t y0[2] = {k0.x, k1.x}, y1[2] = {k0.y, k1.y};
            range.see(k0.x, k0.y), range.see(k1.x, k1.y);
            acc0.add(sx[s][0][tid], y0);
            acc1.add(sx[s][1][tid], y1);
            if (FOLD && (t + 1) % (LIMB_TERMS2 - 1) == 0) acc0.fold(), acc1.fold();
        }
        cp_async_wait<0>();
        const int64_t mone = one[j];
        int64_t c0[2] = {0, 0}, c1[2] = {0, 0};  // the summands of the two positions, in flight during the fold
        if (a.has_add0) c0[0] = *kat<int64_t>(a.add0, i, j, sk, sl0), c0[1] = *kat<int64_t>(a.add0, i, j, sk, sl1);
        if (a.has_add1) c1[0] = *kat<int64_t>(a.add1, i, j, sk, sl0), c1[1] = *kat<int64_t>(a.add1, i, j, sk, sl1);
        acc0.fold(), acc1.fold();
        if (range.beyond()) {
            acc0.start(), acc1.start();
            for (int t = 0; t < a.nterms; t++) {
                const int64_t x0 = *kat<int64_t>(a.parts[t], i, j, sk, sl0), x1 = *kat<int64_t>(a.parts[t], i, j, sk, sl1);
                for (int q = 0; q < 2; q++) {
                    const int64_t* y = kat<int64_t>(a.keys[t], q, j, k, l) + a.group.off[key];
                    acc0.add_wide(q, x0, y[0]), acc1.add_wide(q, x1, y[1]);
                }
            }
        }
        if (a.has_add0) acc0.add_wide(0, c0[0], mone), acc1.add_wide(0, c0[1], mone);
        if (a.has_add1) acc0.add_wide(1, c1[0], mone), acc1.add_wide(1, c1[1], mone);
        const MontLimbs ml = mont_limbs(m.n[j], m.ninv[j]);
        const int64_t r2 = m.r2[j];
        longlong2 w0, w1;
        w0.x = finish_wide(acc0.lo[0], acc0.hi[0], a.full0, ml, r2), w0.y = finish_wide(acc1.lo[0], acc1.hi[0], a.full0, ml, r2);
        w1.x = finish_wide(acc0.lo[1], acc0.hi[1], a.full1, ml, r2), w1.y = finish_wide(acc1.lo[1], acc1.hi[1], a.full1, ml, r2);
        int64_t* o = a.group.dst[key] + 2 * i * a.dst.s0 + j * a.dst.s1 + k * a.dst.s2 + l;
        *reinterpret_cast<longlong2*>(o) = w0;
        *reinterpret_cast<longlong2*>(o + a.dst.s0) = w1;
    }
}

/// W consecutive words at p (W = 2: one 16-byte access; p must be 16-byte aligned).
template <int W>
__device__ __forceinline__ void load_words(const int64_t* p, int64_t (&v)[W]) {
    if constexpr (W == 2) {
        const longlong2 t = *reinterpret_cast<const longlong2*>(p);
        v[0] = t.x, v[1] = t.y;
    } else {
        v[0] = *p;
    }
}
template <int W>
__device__ __forceinline__ void store_words(int64_t* p, const int64_t (&v)[W]) {
    if constexpr (W == 2) {
        longlong2 t;
        t.x = v[0], t.y = v[1];
        *reinterpret_cast<longlong2*>(p) = t;
    } else {
        *p = v[0];
    }
}

/// tensor_kernel's three products of `count` positions in 128 bits, for ciphertexts (the caller's) with words beyond the
/// limb sums; the rows' reductions as bits of `full`.
__device__ __noinline__ void tensor_any(const int64_t* lp, int64_t ls, const int64_t* rp, int64_t rs, int64_t* d01, int64_t ds,
                                        int64_t* d2, int count, int64_t n, int64_t ninv, int64_t r2, int full) {
    auto finish = [&](u128 v, int q) { return finish_any((uint64_t)v, (int64_t)(v >> 64), (full >> q) & 1, n, ninv, r2); };
    auto prod = [](int64_t x, int64_t y) { return (u128)((i128)x * (i128)y); };
#pragma unroll 1
    for (int w = 0; w < count; w++) {
        const int64_t l0 = lp[w], l1 = lp[w + ls], r0 = rp[w], r1 = rp[w + rs];
        d01[w] = finish(prod(l0, r0), 0);
        d01[w + ds] = finish(prod(l0, r1) + prod(l1, r0), 1);
        d2[w] = finish(prod(l1, r1), 2);
    }
}

/// (l0 r0, l0 r1 + l1 r0, l1 r1) of B pairs of 2-row ciphertext tensors ([2B, ...] each),
/// reduced per row into [3B, ...]: rows 2i and 2i + 1 receive the first two components of pair i,
/// row 2B + i the third. Each operand comes in two parts along the RNS dimension: rows j < rsplit
/// from *_lo, rows j >= rsplit from *_hi (row j - rsplit). W adjacent positions per thread (W = 2
/// needs an even dimension 3 and 16-byte aligned rows in every view).
template <int W>
__global__ void __launch_bounds__(256) tensor_kernel(KView d, KView lhs_lo, KView lhs_hi, KView rhs_lo, KView rhs_hi,
                                                     int rsplit, KMods m, int full0, int full1, int full2,
                                                     int64_t lines, int chunks) {
    grid_wait();
    const int64_t tiles = lines * chunks;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        int64_t line = tile / chunks;  // (i, j, k)
        int64_t l = W * ((tile - line * chunks) * blockDim.x + threadIdx.x);
        if (l >= d.n3) continue;
        int64_t k = line % d.n2, r = line / d.n2;
        int64_t j = r % d.n1, i = r / d.n1;
        const bool lo = j < rsplit;
        const int64_t js = lo ? j : j - rsplit;
        const int64_t* lp = lo ? kat<int64_t>(lhs_lo, 2 * i, js, k, l) : kat<int64_t>(lhs_hi, 2 * i, js, k, l);
        const int64_t* rp = lo ? kat<int64_t>(rhs_lo, 2 * i, js, k, l) : kat<int64_t>(rhs_hi, 2 * i, js, k, l);
        const int64_t ls = lo ? lhs_lo.s0 : lhs_hi.s0, rs = lo ? rhs_lo.s0 : rhs_hi.s0;
        const MontLimbs ml = mont_limbs(m.n[j], m.ninv[j]);
        const int64_t r2 = m.r2[j];
        int64_t l0[W], l1[W], r0[W], r1[W], o0[W], o1[W], o2[W];
        load_words<W>(lp, l0), load_words<W>(lp + ls, l1);
        load_words<W>(rp, r0), load_words<W>(rp + rs, r1);
        WordRange range;
#pragma unroll
        for (int w = 0; w < W; w++) {
            range.see(l0[w], l1[w]), range.see(r0[w], r1[w]);
            const int2 x0 = limb_split(l0[w]), x1 = limb_split(l1[w]), y0 = limb_split(r0[w]), y1 = limb_split(r1[w]);
            const int xs0 = x0.x + x0.y, xs1 = x1.x + x1.y, ys0 = y0.x + y0.y, ys1 = y1.x + y1.y;
            LimbSum s[3];
            uint64_t lo[3] = {0, 0, 0};
            int64_t hi[3] = {0, 0, 0};
#pragma unroll
            for (int q = 0; q < 3; q++) s[q].zero();
            s[0].mac(x0, xs0, y0, ys0);
            s[1].mac(x0, xs0, y1, ys1), s[1].mac(x1, xs1, y0, ys0);
            s[2].mac(x1, xs1, y1, ys1);
#pragma unroll
            for (int q = 0; q < 3; q++) s[q].fold(lo[q], hi[q]);
            o0[w] = finish_wide(lo[0], hi[0], full0, ml, r2);
            o1[w] = finish_wide(lo[1], hi[1], full1, ml, r2);
            o2[w] = finish_wide(lo[2], hi[2], full2, ml, r2);
        }
        const int64_t B = d.n0 / 3;
        store_words<W>(kat<int64_t>(d, 2 * i, j, k, l), o0);
        store_words<W>(kat<int64_t>(d, 2 * i + 1, j, k, l), o1);
        store_words<W>(kat<int64_t>(d, 2 * B + i, j, k, l), o2);
        if (range.beyond())
            tensor_any(lp, ls, rp, rs, kat<int64_t>(d, 2 * i, j, k, l), d.s0, kat<int64_t>(d, 2 * B + i, j, k, l), W, m.n[j],
                       m.ninv[j], r2, full0 | full1 << 1 | full2 << 2);
    }
}

/// The three-component products of two dBFV ciphertexts' digits with reduce_wide (dbfv_mul_convolve,
/// src/dbfv.rs:1081-1126): output digit o (rows 2o, 2o + 1 and, its c2, 2 dout + o of d) sums the products
/// of lhs digit q and rhs digit o - q, operands within 2p, folded every DBFV_FOLD digit pairs. Sums of more
/// than full_above terms take the double reduction (the wide accumulator's bound).
/// What bounds it: memory and the multiply pipe about equally (a position's 2 (d1 + d2) words in, 3 dout out, three
/// products per pair of digits in four limb sums and 3 dout reductions): 84 us for three digits each at
/// field_49152 with 34 factors. As nine inner products into a 128-bit tensor, its reduction and rescale's
/// product by t (now in the inverse transform's last pass) 305 us.
constexpr int DBFV_FOLD = (LIMB_TERMS2 - 1) / 2;
template <int W>
__global__ void __launch_bounds__(256) dbfv_tensor_kernel(KView d, KView lhs, KView rhs, int d1, int d2, int dout, KMods m,
                                                          int full_above, int64_t lines, int chunks) {
    grid_wait();
    const int64_t tiles = lines * chunks;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int64_t line = tile / chunks;  // (j, k)
        const int64_t l = W * ((tile - line * chunks) * blockDim.x + threadIdx.x);
        if (l >= d.n3) continue;
        const int64_t k = line % d.n2, j = line / d.n2;
        const int64_t* lp = kat<int64_t>(lhs, 0, j, k, l);
        const int64_t* rp = kat<int64_t>(rhs, 0, j, k, l);
        const MontLimbs ml = mont_limbs(m.n[j], m.ninv[j]);
        const int64_t r2 = m.r2[j];
        for (int o = 0; o < dout; o++) {
            const int q0 = o >= d2 ? o - (d2 - 1) : 0, q1 = o < d1 ? o : d1 - 1;
            LimbSum s[3][W];
            uint64_t lo[3][W];
            int64_t hi[3][W];
#pragma unroll
            for (int c = 0; c < 3; c++)
#pragma unroll
                for (int w = 0; w < W; w++) s[c][w].zero(), lo[c][w] = 0, hi[c][w] = 0;
            auto fold = [&] {
#pragma unroll
                for (int c = 0; c < 3; c++)
#pragma unroll
                    for (int w = 0; w < W; w++) s[c][w].fold(lo[c][w], hi[c][w]), s[c][w].zero();
            };
            int until = DBFV_FOLD;
            for (int q = q0; q <= q1; q++) {
                int64_t l0[W], l1[W], r0[W], r1[W];
                load_words<W>(lp + 2 * q * lhs.s0, l0), load_words<W>(lp + (2 * q + 1) * lhs.s0, l1);
                load_words<W>(rp + 2 * (o - q) * rhs.s0, r0), load_words<W>(rp + (2 * (o - q) + 1) * rhs.s0, r1);
#pragma unroll
                for (int w = 0; w < W; w++) {
                    const int2 x0 = limb_split(l0[w]), x1 = limb_split(l1[w]), y0 = limb_split(r0[w]), y1 = limb_split(r1[w]);
                    const int xs0 = x0.x + x0.y, xs1 = x1.x + x1.y, ys0 = y0.x + y0.y, ys1 = y1.x + y1.y;
                    s[0][w].mac(x0, xs0, y0, ys0);
                    s[1][w].mac(x0, xs0, y1, ys1), s[1][w].mac(x1, xs1, y0, ys0);
                    s[2][w].mac(x1, xs1, y1, ys1);
                }
                if (--until == 0) fold(), until = DBFV_FOLD;
            }
            fold();
            const int n = q1 - q0 + 1;
            int64_t v[3][W];
#pragma unroll
            for (int c = 0; c < 3; c++)
#pragma unroll
                for (int w = 0; w < W; w++)
                    v[c][w] = finish_wide(lo[c][w], hi[c][w], (c == 1 ? 2 * n : n) > full_above, ml, r2);
            store_words<W>(kat<int64_t>(d, 2 * o, j, k, l), v[0]);
            store_words<W>(kat<int64_t>(d, 2 * o + 1, j, k, l), v[1]);
            store_words<W>(kat<int64_t>(d, 2 * dout + o, j, k, l), v[2]);
        }
    }
}

/// One giant step of the homomorphic CRT transform: output digit o (rows 2o, 2o + 1 of dst) is
/// sum over the baby steps j and input digits i of baby(j, i) * L(coef_j, o - i), plus the carried
/// digit o through mont(1), reduced. Each thread holds the accumulators of up to GIANT_OUT output
/// digits, so every baby-step digit is read once for all the outputs it feeds.
constexpr int GIANT_OUT = 4;
constexpr int GIANT_MAX_BABY = 256;

struct GiantArgs {
    KView babies;   // [nbaby * 2d, r, dl, dk]: block j holds sigma^j of the d input digits (rows 2i, 2i + 1)
    KView lcoef;    // [nt, r, dl, 1]: balanced digits of the L' coefficients (CRT basis), broadcast on dim 3
    int nbaby, d;
    short lfirst[GIANT_MAX_BABY];  // row in lcoef of digit 0 of baby j's coefficient
    short lcount[GIANT_MAX_BABY];  // its digit count
    int out0, nout;                // output digits [out0, out0 + nout) of this launch (nout <= GIANT_OUT)
    KView add;                     // the carried digits [2 nadd, ...] (through mont(1))
    int nadd;
    unsigned full;                 // bit o - out0: output digit o needs the full double reduction
    KView dst;                     // [2 used, ...]
    const int* beyond;             // not 0: block 0, the caller's ciphertext, has words beyond the limb sums
};

/// The lcoef values of a tile's line (j, k) are the same for all its positions: the CTA stages
/// them in shared memory once per tile (nt words, dynamic shared memory, after the staging
/// buffers). The (baby step, input digit) units that feed an output digit of the launch are listed
/// by the host (`units`, in giant step order); each thread copies its positions' two words of the
/// next GIANT_STAGES - 1 units into shared memory with cp.async while it multiplies the current
/// one, so that its loads in flight take no registers, and forms every address from one base
/// offset and the row stride. Each thread copies and reads only its own slots.
constexpr int GIANT_STAGES = 4;
constexpr int GIANT_MAX_UNITS = 1024;

/// The (baby step j, input digit i) units of one launch, prepared on the host: the unit's first
/// row in the baby-step tensor (2 d j + 2 i), the output digits o it feeds (bit o of the mask: 0 <=
/// out0 + o - i < lcount[j]) and the coefficient-digit row of output 0 (lfirst[j] + out0 - i;
/// output o reads row fb + o).
struct GiantUnits {
    unsigned int w[GIANT_MAX_UNITS];  // row | mask << 16
    short fb[GIANT_MAX_UNITS];
    int n;
};

/// A copy of a ciphertext that notes in `beyond` whether a word lies beyond the limb sums. The giant steps read it
/// once per CTA: seeing the words on the way, in their loop, cost them 5 % (the step at r = 23 4765 -> 4879 us).
/// CTAs over (COPY_SPAN positions, line), the line split once per thread (split per element 41 us for the step's six
/// rows, a plain copy 16).
constexpr int COPY_SPAN = 1024;
__global__ void __launch_bounds__(256) copy_range_kernel(KView d, KView s, int* beyond, int lines) {
    grid_wait();
    const int64_t l0 = (int64_t)blockIdx.x * COPY_SPAN + threadIdx.x;
    for (int line = blockIdx.y; line < lines; line += gridDim.y) {
        const int k = line % (int)d.n2, r = line / (int)d.n2, j = r % (int)d.n1, i = r / (int)d.n1;
        const int64_t* sp = kat<int64_t>(s, i, j, k, 0);
        int64_t* dp = kat<int64_t>(d, i, j, k, 0);
        int64_t v[COPY_SPAN / 256];
        WordRange range;
#pragma unroll
        for (int q = 0; q < COPY_SPAN / 256; q++) v[q] = l0 + 256 * q < d.n3 ? sp[l0 + 256 * q] : 0;
#pragma unroll
        for (int q = 0; q < COPY_SPAN / 256; q++) {
            range.see(v[q], v[q]);
            if (l0 + 256 * q < d.n3) dp[l0 + 256 * q] = v[q];
        }
        if (range.beyond()) *beyond = 1;
    }
}

/// Component `row` of the launch's output digits at one position in 128-bit sums: for ciphertexts (block 0 of the
/// baby steps, the caller's) with words beyond the limb sums. The other blocks are key switches' results.
__device__ __noinline__ void giant_any(const GiantArgs& a, int64_t n, int64_t ninv, int64_t r2, int64_t one, int64_t j, int64_t k,
                                       int64_t l, int row) {
    for (int o = a.out0; o < a.out0 + a.nout; o++) {
        u128 v = o < a.nadd ? (u128)((i128)*kat<int64_t>(a.add, 2 * o + row, j, k, l) * (i128)one) : 0;
        for (int q = 0; q < a.nbaby; q++)
            for (int i = 0; i < a.d && i <= o; i++)
                if (o - i < a.lcount[q])
                    v += (u128)((i128)*kat<int64_t>(a.babies, 2 * (a.d * q + i) + row, j, k, l) *
                                (i128)*kat<int64_t>(a.lcoef, a.lfirst[q] + o - i, j, k, 0));
        *kat<int64_t>(a.dst, 2 * o + row, j, k, l) =
            finish_any((uint64_t)v, (int64_t)(v >> 64), (a.full >> (o - a.out0)) & 1, n, ninv, r2);
    }
}

template <int NOUT>
__global__ void __launch_bounds__(256, NOUT <= 2 ? 4 : 3) giant_kernel(const __grid_constant__ GiantArgs a, GiantUnits un, KMods m, const int64_t* one,
                                                             int64_t lines, int chunks) {
    grid_wait();
    extern __shared__ __align__(16) int64_t gsm[];  // [GIANT_STAGES][2][256] staging, then the tile's lcoef as limb pairs
    int2* slc = reinterpret_cast<int2*>(gsm + GIANT_STAGES * 2 * 256);
    const int64_t tiles = lines * chunks;
    const int nt = (int)a.lcoef.n0;
    const int tid = threadIdx.x;
    const bool beyond = *a.beyond != 0;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int64_t line = tile / chunks;  // (j, k)
        const int64_t l = (tile - line * chunks) * blockDim.x + tid;
        const int64_t k = line % a.dst.n2, j = line / a.dst.n2;
        __syncthreads();  // the previous tile's readers of slc are done
        for (int t = tid; t < nt; t += blockDim.x) slc[t] = limb_split(*kat<int64_t>(a.lcoef, t, j, k, 0));
        __syncthreads();
        if (l >= a.dst.n3) continue;
        if (beyond) {
            for (int row = 0; row < 2; row++) giant_any(a, m.n[j], m.ninv[j], m.r2[j], one[j], j, k, l, row);
            continue;
        }
        const int64_t rs = a.babies.s0;  // row stride of the baby-step tensor
        const int64_t* xb = kat<int64_t>(a.babies, 0, j, k, l);
        auto issue = [&](int u) {
            if (u < un.n) {
                const int64_t* xr = xb + (int64_t)(un.w[u] & 0xffff) * rs;
                int64_t* slot = gsm + (u % GIANT_STAGES) * 512;
                cp_async8(slot + tid, xr);
                cp_async8(slot + 256 + tid, xr + rs);
            }
            cp_async_commit();  // an empty group past the end keeps the count uniform
        };
#pragma unroll
        for (int u = 0; u < GIANT_STAGES - 1; u++) issue(u);
        LimbSum s0[NOUT], s1[NOUT];
        uint64_t lo0[NOUT], lo1[NOUT];
        int64_t hi0[NOUT], hi1[NOUT];
#pragma unroll
        for (int o = 0; o < NOUT; o++) s0[o].zero(), s1[o].zero(), lo0[o] = lo1[o] = 0, hi0[o] = hi1[o] = 0;
        auto fold = [&] {
#pragma unroll
            for (int o = 0; o < NOUT; o++) {
                s0[o].fold(lo0[o], hi0[o]), s1[o].fold(lo1[o], hi1[o]);
                s0[o].zero(), s1[o].zero();
            }
        };
        for (int u = 0; u < un.n; u++) {
            issue(u + GIANT_STAGES - 1);
            cp_async_wait<GIANT_STAGES - 1>();  // unit u's words have landed
            const unsigned mask = un.w[u] >> 16;
            const int fb = un.fb[u];
            const int64_t* slot = gsm + (u % GIANT_STAGES) * 512;
            const int2 x0 = limb_split(slot[tid]), x1 = limb_split(slot[256 + tid]);
            const int xs0 = x0.x + x0.y, xs1 = x1.x + x1.y;
#pragma unroll
            for (int o = 0; o < NOUT; o++) {
                if ((mask >> o) & 1) {
                    const int2 f = slc[fb + o];
                    s0[o].mac(x0, xs0, f, f.x + f.y);
                    s1[o].mac(x1, xs1, f, f.x + f.y);
                }
            }
            if ((u + 1) % (LIMB_TERMS2 - 1) == 0) fold();
        }
        cp_async_wait<0>();
        const int64_t on = one[j];
        const int2 w = limb_split(on);
#pragma unroll
        for (int o = 0; o < NOUT; o++) {
            if (a.out0 + o < a.nadd) {
                const int2 v0 = limb_split(*kat<int64_t>(a.add, 2 * (a.out0 + o), j, k, l));
                const int2 v1 = limb_split(*kat<int64_t>(a.add, 2 * (a.out0 + o) + 1, j, k, l));
                s0[o].mac(v0, v0.x + v0.y, w, w.x + w.y);
                s1[o].mac(v1, v1.x + v1.y, w, w.x + w.y);
            }
        }
        fold();
        const MontLimbs ml = mont_limbs(m.n[j], m.ninv[j]);
        const int64_t r2 = m.r2[j];
#pragma unroll
        for (int o = 0; o < NOUT; o++) {
            const bool full = (a.full >> o) & 1;
            const int od = a.out0 + o;
            *kat<int64_t>(a.dst, 2 * od, j, k, l) = finish_wide(lo0[o], hi0[o], full, ml, r2);
            *kat<int64_t>(a.dst, 2 * od + 1, j, k, l) = finish_wide(lo1[o], hi1[o], full, ml, r2);
        }
    }
}

/// giant_kernel where output digits 0 .. NOUT - 1 start at digit 0 and every baby step's coefficient has at
/// least NOUT digits (any dense transform): input digit i < NOUT then feeds the outputs o >= i with
/// coefficient digit o - i, so a baby step is straight-line code over its NOUT rows and NOUT
/// coefficient digits. A thread takes two adjacent positions (16-byte copies and stores) of one of the
/// two rows; half of the CTA's threads take each row. n0: input digits used (min(d, NOUT)).
/// What bounds it: memory and the multiply pipe about equally (a step reads every baby row once); the
/// unit list, masks and single-word copies of giant_kernel kept it issue-bound: 237 us per giant step of
/// 13 baby steps and three digits at field_49152 r = 23, here 159 us.
/// One output digit has few sums, so four CTAs per SM and four stages keep more reads in flight: a step at r = 12
/// with 40 one-digit coefficients 601 -> 580 us; with more digits four CTAs spill (5138 us against 4896 at three digits)
/// and two are 1 % slower.
constexpr int TRI_STAGES = 4;

template <int NOUT>
__global__ void __launch_bounds__(256, NOUT == 4 ? 2 : NOUT >= 2 ? 3 : 4)
    giant_tri_kernel(const __grid_constant__ GiantArgs a, KMods m, const int64_t* one, int n0, int64_t lines, int chunks) {
    grid_wait();
    extern __shared__ __align__(16) int64_t gsm[];  // [TRI_STAGES][NOUT][256] position pairs, then the lcoef limb pairs
    longlong2* sx = reinterpret_cast<longlong2*>(gsm);
    int2* slc = reinterpret_cast<int2*>(sx + TRI_STAGES * NOUT * 256);
    const int64_t tiles = lines * chunks;
    const int nt = (int)a.lcoef.n0, tid = threadIdx.x;
    const bool beyond = *a.beyond != 0;
    const int row = tid >> 7, lane = tid & 127;  // the ciphertext component, the pair of positions
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int64_t line = tile / chunks;  // (j, k)
        const int64_t l = (tile - line * chunks) * 256 + 2 * lane;
        const int64_t k = line % a.dst.n2, j = line / a.dst.n2;
        __syncthreads();  // the previous tile's readers of slc are done
        for (int t = tid; t < nt; t += 256) slc[t] = limb_split(*kat<int64_t>(a.lcoef, t, j, k, 0));
        __syncthreads();
        if (l >= a.dst.n3) continue;
        if (beyond) {
            for (int p = 0; p < 2; p++) giant_any(a, m.n[j], m.ninv[j], m.r2[j], one[j], j, k, l + p, row);
            continue;
        }
        const int64_t rs = a.babies.s0;
        const int64_t* next = kat<int64_t>(a.babies, row, j, k, l);  // baby step q's rows of this thread, in turn
        auto issue = [&](int q, int slot) {
            if (q < a.nbaby) {
#pragma unroll
                for (int i = 0; i < NOUT; i++)
                    if (i < n0) cp_async16(sx + (slot * NOUT + i) * 256 + tid, next + 2 * i * rs);
                next += 2 * a.d * rs;
            }
            cp_async_commit();  // an empty group past the end keeps the count uniform
        };
#pragma unroll
        for (int q = 0; q < TRI_STAGES - 1; q++) issue(q, q);
        LimbSum s[NOUT][2];
        uint64_t lo[NOUT][2];
        int64_t hi[NOUT][2];
#pragma unroll
        for (int o = 0; o < NOUT; o++)
#pragma unroll
            for (int p = 0; p < 2; p++) s[o][p].zero(), lo[o][p] = 0, hi[o][p] = 0;
        auto fold = [&] {
#pragma unroll
            for (int o = 0; o < NOUT; o++)
#pragma unroll
                for (int p = 0; p < 2; p++) s[o][p].fold(lo[o][p], hi[o][p]), s[o][p].zero();
        };
        constexpr int FOLD = (LIMB_TERMS2 - 1) / NOUT;  // baby steps whose terms the sums hold
        int until = FOLD, slot = 0;
        for (int q = 0; q < a.nbaby; q++) {
            issue(q + TRI_STAGES - 1, slot == 0 ? TRI_STAGES - 1 : slot - 1);
            cp_async_wait<TRI_STAGES - 1>();  // baby step q's rows have landed
            const int2* fc = slc + a.lfirst[q];
            int2 f[NOUT];
#pragma unroll
            for (int o = 0; o < NOUT; o++) f[o] = fc[o];
#pragma unroll
            for (int i = 0; i < NOUT; i++) {
                if (i < n0) {
                    const longlong2 v = sx[(slot * NOUT + i) * 256 + tid];
                    const int2 x0 = limb_split(v.x), x1 = limb_split(v.y);
                    const int xs0 = x0.x + x0.y, xs1 = x1.x + x1.y;
#pragma unroll
                    for (int o = i; o < NOUT; o++) {
                        const int2 w = f[o - i];
                        s[o][0].mac(x0, xs0, w, w.x + w.y);
                        s[o][1].mac(x1, xs1, w, w.x + w.y);
                    }
                }
            }
            if (--until == 0) fold(), until = FOLD;
            slot = slot == TRI_STAGES - 1 ? 0 : slot + 1;
        }
        cp_async_wait<0>();
        const int2 w = limb_split(one[j]);
#pragma unroll
        for (int o = 0; o < NOUT; o++) {
            if (o < a.nadd) {
                const longlong2 v = *reinterpret_cast<const longlong2*>(kat<int64_t>(a.add, 2 * o + row, j, k, l));
                const int2 x0 = limb_split(v.x), x1 = limb_split(v.y);
                s[o][0].mac(x0, x0.x + x0.y, w, w.x + w.y);
                s[o][1].mac(x1, x1.x + x1.y, w, w.x + w.y);
            }
        }
        fold();
        const MontLimbs ml = mont_limbs(m.n[j], m.ninv[j]);
        const int64_t r2 = m.r2[j];
#pragma unroll
        for (int o = 0; o < NOUT; o++) {
            const bool full = (a.full >> o) & 1;
            longlong2 r;
            r.x = finish_wide(lo[o][0], hi[o][0], full, ml, r2), r.y = finish_wide(lo[o][1], hi[o][1], full, ml, r2);
            *reinterpret_cast<longlong2*>(kat<int64_t>(a.dst, 2 * o + row, j, k, l)) = r;
        }
    }
}

void grid_lines(hc_context ctx, int64_t n3, int64_t lines, int* chunks, unsigned* blocks) {
    *chunks = (int)((n3 + 255) / 256);
    int64_t tiles = lines * *chunks;
    int64_t cap = (int64_t)hc::num_sms(ctx) * 32;
    *blocks = (unsigned)(tiles < cap ? (tiles > 0 ? tiles : 1) : cap);
}

}  // namespace

namespace hc {

hc_status launch_bconv_fused(hc_context ctx, const KView& src, const KView& dst, const BconvConsts& c, int r, int rd,
                             int nb, const KMods& sm, const KMods& dm, int64_t ns, const BarrettLimbs* sub_mul) {
    BconvArgs a;
    a.src = src;
    a.dst = dst;
    a.c = c;
    a.r = r, a.rd = rd, a.nb = nb;
    a.sub_mul = sub_mul;
    a.npos = src.n2 * src.n3;
    if (a.npos == 0 || ns == 0 || rd == 0) return HC_OK;
    if (ns * nb > 65535) return fail(HC_ERR_UNSUPPORTED, "base conversion: batch too large");
    const size_t smem = (size_t)r * BCONV_THREADS * 8;
    if (smem > max_smem_optin(ctx)) return fail(HC_ERR_UNSUPPORTED, "base conversion: too many source rows");
    const bool one_chunk = c.chunk >= r, sub = sub_mul != nullptr;
    // the outputs of a position are split over CTAs while the grid leaves SMs short of work; each
    // split lifts the block's columns again. An SM is busy with four CTAs, so chunks of `oc` outputs
    // take about max(CTAs per SM, 4) times a CTA's cost, in wide products: 8 per lifted column, and per
    // output 3 per column and 32 of reductions ([2, 16 -> 18] of field_36864: 24 us whole, 28 us in two)
    const int64_t cols = (a.npos + BCONV_THREADS - 1) / BCONV_THREADS, base_ctas = cols * ns * nb;
    const int64_t sms = num_sms(ctx);
    const int lifted = (r + nb - 1) / nb;  // columns of a block
    int64_t best = -1;
    for (int oc = (rd + 1) / 2 * 2; oc >= 2; oc -= 2) {
        const int64_t n = (base_ctas * ((rd + oc - 1) / oc) + sms - 1) / sms;
        const int64_t cost = std::max<int64_t>(n, 4) * (8 * lifted + oc * (3 * lifted + 32));
        if (best < 0 || cost < best) best = cost, a.ochunk = oc;
    }
    dim3 grid((unsigned)cols, (unsigned)(ns * nb), (unsigned)((rd + a.ochunk - 1) / a.ochunk));
    auto run = [&](auto kern, const auto& mx) {
        if (smem > 49152) {
            cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (e != cudaSuccess) return cuda_check(e, "bconv smem attribute");
        }
        hc::launch_kernel(kern, grid, BCONV_THREADS, smem, stream_of(ctx), a, sm, dm, mx);
        count_launch(ctx);
        return cuda_check(cudaGetLastError(), "bconv kernel launch");
    };
    auto param = [&](auto mx) {
        typedef decltype(mx) MAT;
        std::memcpy(mx.m, c.hmat, (size_t)c.hwords * sizeof(int2));
        return sub ? run(bconv_fused_kernel<true, true, MAT>, mx) : run(bconv_fused_kernel<true, false, MAT>, mx);
    };
    if (one_chunk && c.hwords > 0 && c.hwords <= BconvSmall::ENTRIES) return param(BconvSmall());
    if (one_chunk && c.hwords > 0 && c.hwords <= BconvParam::ENTRIES) return param(BconvParam());
    const BconvMemory none{};
    if (one_chunk)
        return sub ? run(bconv_fused_kernel<true, true, BconvMemory>, none)
                   : run(bconv_fused_kernel<true, false, BconvMemory>, none);
    return sub ? run(bconv_fused_kernel<false, true, BconvMemory>, none)
               : run(bconv_fused_kernel<false, false, BconvMemory>, none);
}

hc_status launch_dbfv_split(hc_context ctx, const KView& x, const KView& src, const KView& carry, const DbfvSplit& d,
                            const KMods& m) {
    const int r = (int)x.n1;
    const int64_t npos = x.n2 * x.n3;
    if (npos == 0 || x.n0 == 0) return HC_OK;
    const size_t smem = (size_t)r * BCONV_THREADS * 8;
    if (smem > max_smem_optin(ctx) || x.n0 > 65535) return fail(HC_ERR_UNSUPPORTED, "dBFV reduction: too many rows");
    if (smem > 49152) {
        cudaError_t e = cudaFuncSetAttribute(dbfv_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return cuda_check(e, "dBFV reduction smem attribute");
    }
    dim3 grid((unsigned)((npos + BCONV_THREADS - 1) / BCONV_THREADS), (unsigned)x.n0);
    hc::launch_kernel(dbfv_split_kernel, grid, BCONV_THREADS, smem, stream_of(ctx), x, src, carry, d, r, m, npos);
    count_launch(ctx);
    return cuda_check(cudaGetLastError(), "dBFV reduction launch");
}

hc_status launch_copy_range(hc_context ctx, const KView& d, const KView& s, int* beyond) {
    const int64_t lines = d.n0 * d.n1 * d.n2;
    if (lines == 0 || d.n3 == 0) return HC_OK;
    if (lines > INT32_MAX) return fail(HC_ERR_UNSUPPORTED, "too many ciphertext rows");
    dim3 grid((unsigned)((d.n3 + COPY_SPAN - 1) / COPY_SPAN), (unsigned)std::min<int64_t>(lines, 65535));
    hc::launch_kernel(copy_range_kernel, grid, 256, 0, stream_of(ctx), d, s, beyond, (int)lines);
    count_launch(ctx);
    return cuda_check(cudaGetLastError(), "ciphertext copy launch");
}

hc_status launch_galois(hc_context ctx, const KView& d, const KView& s, const uint32_t* p2, const uint32_t* p3) {
    int64_t lines = d.n0 * d.n1 * d.n2;
    if (lines == 0 || d.n3 == 0) return HC_OK;
    int chunks;
    unsigned blocks;
    grid_lines(ctx, d.n3, lines, &chunks, &blocks);
    hc::launch_kernel(galois_kernel, blocks, 256, 0, stream_of(ctx), d, s, p2, p3, lines, chunks);
    count_launch(ctx);
    return cuda_check(cudaGetLastError(), "galois kernel launch");
}

hc_status launch_keyswitch(hc_context ctx, const KView* parts, const KView* keys, int nterms, const KView* add0,
                           const KView* add1, int full0, int full1, const KView& dst, const KMods& m,
                           const int64_t* one_dev, const KsGroup& group, bool reverse) {
    if (nterms > HC_MAX_TERMS) return fail(HC_ERR_UNSUPPORTED, "too many gadget digits");
    KsArgs a;
    a.reverse = reverse;
    for (int t = 0; t < nterms; t++) a.parts[t] = parts[t], a.keys[t] = keys[t];
    a.nterms = nterms;
    a.has_add0 = add0 != nullptr;
    a.has_add1 = add1 != nullptr;
    if (add0) a.add0 = *add0;
    if (add1) a.add1 = *add1;
    a.full0 = full0, a.full1 = full1;
    a.dst = dst;
    a.group = group;
    a.batch = dst.n0 / 2;
    int64_t lines = a.batch * dst.n1 * dst.n2;
    if (lines == 0 || dst.n3 == 0) return HC_OK;
    // the paired kernel needs an even dimension 3 and 16-byte aligned key and output rows
    auto aligned = [](const KView& v) {
        return ((uintptr_t)v.p % 16) == 0 && v.s0 % 2 == 0 && v.s1 % 2 == 0 && v.s2 % 2 == 0 && !v.b3;
    };
    bool pair = dst.n3 % 2 == 0 && aligned(dst);
    for (int g = 0; g < group.n; g++) pair = pair && ((uintptr_t)group.dst[g] % 16) == 0 && group.off[g] % 2 == 0;
    for (int t = 0; t < nterms; t++) pair = pair && aligned(keys[t]);
    int chunks;
    unsigned blocks;
    if (!pair) {
        grid_lines(ctx, dst.n3, lines, &chunks, &blocks);
        for (int g = 0; g < group.n; g++) {
            a.dst.p = (char*)group.dst[g];
            a.group.p2[0] = group.p2[g], a.group.p3[0] = group.p3[g];
            for (int t = 0; t < nterms; t++) a.keys[t].p = keys[t].p + 8 * group.off[g];
            hc::launch_kernel(keyswitch1_kernel, blocks, 256, 0, stream_of(ctx), a, m, one_dev, lines, chunks);
            count_launch(ctx);
            hc_status st = cuda_check(cudaGetLastError(), "keyswitch kernel launch");
            if (st) return st;
        }
        return HC_OK;
    }
    grid_lines(ctx, dst.n3 / 2, lines * group.n, &chunks, &blocks);
    if (lines * chunks * group.n > INT32_MAX) return fail(HC_ERR_UNSUPPORTED, "key switch: too many positions");
    bool common = true;
    for (int t = 1; t < nterms; t++) {
        const KView &p = parts[t], &p0 = parts[0], &k = keys[t], &k0 = keys[0];
        common = common && p.s0 == p0.s0 && p.s1 == p0.s1 && p.s2 == p0.s2 && p.b3 == p0.b3 && k.s0 == k0.s0 &&
                 k.s1 == k0.s1 && k.s2 == k0.s2;
    }
    const bool fold = nterms >= LIMB_TERMS2;  // the sums fold every LIMB_TERMS2 - 1 digits
    auto kern = common ? (fold ? keyswitch_async_kernel<true, true> : keyswitch_async_kernel<true, false>)
                       : (fold ? keyswitch_async_kernel<false, true> : keyswitch_async_kernel<false, false>);
    hc::launch_kernel(kern, blocks, 256, 0, stream_of(ctx), a, m, one_dev, lines, chunks);
    count_launch(ctx);
    return cuda_check(cudaGetLastError(), "keyswitch kernel launch");
}

hc_status launch_giant(hc_context ctx, const KView& babies, const KView& lcoef, int nbaby, int d, const int* lfirst,
                       const int* lcount, const KView* add, int nadd, const unsigned char* full, int used,
                       const KView& dst, const KMods& m, const int64_t* one_dev, const int* beyond) {
    if (nbaby > GIANT_MAX_BABY) return fail(HC_ERR_UNSUPPORTED, "too many baby steps");
    int64_t lines = dst.n1 * dst.n2;
    if (lines == 0 || dst.n3 == 0 || used == 0) return HC_OK;
    GiantArgs a;
    a.babies = babies;
    a.lcoef = lcoef;
    a.lcoef.b3 = 1;  // broadcast along dimension 3
    a.nbaby = nbaby, a.d = d;
    a.beyond = beyond;
    for (int j = 0; j < nbaby; j++) {
        if (lfirst[j] > 32767 || lcount[j] > 32767) return fail(HC_ERR_UNSUPPORTED, "too many coefficient digits");
        a.lfirst[j] = (short)lfirst[j], a.lcount[j] = (short)lcount[j];
    }
    a.nadd = add ? nadd : 0;
    if (add) a.add = *add;
    a.dst = dst;
    int chunks;
    unsigned blocks;
    grid_lines(ctx, dst.n3, lines, &chunks, &blocks);
    // the staging buffers and the tile's lcoef words
    const size_t smem = (size_t)(GIANT_STAGES * 2 * 256 + std::max<int64_t>(lcoef.n0, 1)) * 8;
    if (smem > 49152) return fail(HC_ERR_UNSUPPORTED, "too many coefficient digits");
    if (d >= 64) return fail(HC_ERR_UNSUPPORTED, "too many dBFV digits");
    // 16-byte accesses of every row, and coefficients with a digit for each output
    auto pairs = [](const KView& v) {
        return ((uintptr_t)v.p % 16) == 0 && v.s0 % 2 == 0 && v.s1 % 2 == 0 && v.s2 % 2 == 0 && !v.b3;
    };
    bool tri = used <= GIANT_OUT && dst.n3 % 2 == 0 && pairs(babies) && pairs(dst) && (!add || pairs(*add));
    for (int bj = 0; bj < nbaby; bj++) tri = tri && lcount[bj] >= used;
    const size_t tri_smem = (size_t)TRI_STAGES * used * 256 * 16 + (size_t)std::max<int64_t>(lcoef.n0, 1) * 8;
    if (tri && tri_smem <= max_smem_optin(ctx)) {
        a.out0 = 0, a.nout = used;
        a.full = 0;
        for (int o = 0; o < used; o++) a.full |= (unsigned)(full[o] != 0) << o;
        auto kern = used == 1 ? giant_tri_kernel<1> : used == 2 ? giant_tri_kernel<2> : used == 3 ? giant_tri_kernel<3> : giant_tri_kernel<4>;
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tri_smem);
        if (e != cudaSuccess) return cuda_check(e, "giant-step smem attribute");
        hc::launch_kernel(kern, blocks, 256, tri_smem, stream_of(ctx), a, m, one_dev, std::min(d, used), lines, chunks);
        count_launch(ctx);
        return cuda_check(cudaGetLastError(), "giant-step kernel launch");
    }
    for (int o0 = 0; o0 < used; o0 += GIANT_OUT) {
        a.out0 = o0;
        a.nout = std::min(GIANT_OUT, used - o0);
        a.full = 0;
        for (int o = 0; o < a.nout; o++) a.full |= (unsigned)(full[o0 + o] != 0) << o;
        GiantUnits un;  // the (baby step, input digit) units that feed an output digit of this launch
        un.n = 0;
        for (int bj = 0; bj < nbaby; bj++)
            for (int i = 0; i < d; i++) {
                unsigned mask = 0;
                for (int o = 0; o < a.nout; o++) {
                    const int jj = a.out0 + o - i;
                    if (jj >= 0 && jj < lcount[bj]) mask |= 1u << o;
                }
                if (!mask) continue;
                const int row = bj * 2 * d + 2 * i, fb = lfirst[bj] + a.out0 - i;
                if (un.n == GIANT_MAX_UNITS || row > 0xffff || fb < -32768 || fb > 32767)
                    return fail(HC_ERR_UNSUPPORTED, "too many baby-step units");
                un.w[un.n] = (unsigned)row | (mask << 16);
                un.fb[un.n++] = (short)fb;
            }
        auto kern = a.nout == 1   ? giant_kernel<1>
                    : a.nout == 2 ? giant_kernel<2>
                    : a.nout == 3 ? giant_kernel<3>
                                  : giant_kernel<4>;
        hc::launch_kernel(kern, blocks, 256, smem, stream_of(ctx), a, un, m, one_dev, lines, chunks);
        count_launch(ctx);
        hc_status st = cuda_check(cudaGetLastError(), "giant-step kernel launch");
        if (st) return st;
    }
    return HC_OK;
}

hc_status launch_dbfv_tensor(hc_context ctx, const KView& d, const KView& lhs, const KView& rhs, int dout, const KMods& m,
                             int full_above) {
    const int64_t lines = d.n1 * d.n2;
    if (lines == 0 || d.n3 == 0) return HC_OK;
    auto aligned = [](const KView& v) { return ((uintptr_t)v.p % 16) == 0 && v.s0 % 2 == 0 && v.s1 % 2 == 0 && v.s2 % 2 == 0; };
    const bool pair = d.n3 % 2 == 0 && aligned(d) && aligned(lhs) && aligned(rhs);
    int chunks;
    unsigned blocks;
    grid_lines(ctx, pair ? d.n3 / 2 : d.n3, lines, &chunks, &blocks);
    hc::launch_kernel(pair ? dbfv_tensor_kernel<2> : dbfv_tensor_kernel<1>, blocks, 256, 0, stream_of(ctx), d, lhs, rhs,
                      (int)(lhs.n0 / 2), (int)(rhs.n0 / 2), dout, m, full_above, lines, chunks);
    count_launch(ctx);
    return cuda_check(cudaGetLastError(), "dBFV tensor kernel launch");
}

hc_status launch_tensor(hc_context ctx, const KView& d, const KView& lhs_lo, const KView& lhs_hi, const KView& rhs_lo,
                        const KView& rhs_hi, int rsplit, const KMods& m, int f0, int f1, int f2) {
    int64_t lines = (d.n0 / 3) * d.n1 * d.n2;
    if (lines == 0 || d.n3 == 0) return HC_OK;
    // two adjacent positions per thread where every view allows 16-byte accesses
    auto aligned = [](const KView& v) {
        return ((uintptr_t)v.p % 16) == 0 && v.s0 % 2 == 0 && v.s1 % 2 == 0 && v.s2 % 2 == 0 && !v.b3;
    };
    const bool pair = d.n3 % 2 == 0 && aligned(d) && aligned(lhs_lo) && aligned(lhs_hi) && aligned(rhs_lo) &&
                      aligned(rhs_hi);
    int chunks;
    unsigned blocks;
    if (pair) {
        grid_lines(ctx, d.n3 / 2, lines, &chunks, &blocks);
        hc::launch_kernel(tensor_kernel<2>, blocks, 256, 0, stream_of(ctx), d, lhs_lo, lhs_hi, rhs_lo, rhs_hi, rsplit, m, f0, f1, f2,
                                                              lines, chunks);
    } else {
        grid_lines(ctx, d.n3, lines, &chunks, &blocks);
        hc::launch_kernel(tensor_kernel<1>, blocks, 256, 0, stream_of(ctx), d, lhs_lo, lhs_hi, rhs_lo, rhs_hi, rsplit, m, f0, f1, f2,
                                                              lines, chunks);
    }
    count_launch(ctx);
    return cuda_check(cudaGetLastError(), "tensor kernel launch");
}

}  // namespace hc
