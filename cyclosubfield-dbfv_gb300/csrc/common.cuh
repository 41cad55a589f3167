// Shared definitions of the sm_103a ring-arithmetic backend: tensor views as kernels see them,
// exact 64/128-bit modular arithmetic, and launch helpers.
//
// The arithmetic reproduces the reference's integer formulas exactly (same inputs -> same
// representatives), because downstream base-conversion corrections depend on the
// representative, not only on the residue:
//   Barrett multiplication by a constant   cyclosubfield-dbfv/src/hal/ntt.rs:126-158
//   Montgomery reductions (R = 2^64)       cyclosubfield-dbfv/src/hal/mont.rs:36-76
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "../../include/halcuda.h"
#include "../../include/ringcuda.h"

typedef __int128 i128;
typedef unsigned __int128 u128;

#define HC_MAX_MODS 96     // RNS rows per call whose moduli travel as kernel parameters
#define HC_MAX_TERMS 64    // inner-product terms per call
#define HC_MAX_STAGES 40   // NTT stages per plan (2^40-point transforms)

// ------------------------------------------------------------------------------------------
// Views
// ------------------------------------------------------------------------------------------

/// A kernel-side 4-D view: shape plus element strides; `s3` is implicitly 1. Broadcast
/// sources carry stride 0 in the broadcast dimensions (`b3` marks a broadcast dimension 3).
struct KView {
    char* p;
    int64_t n0, n1, n2, n3;
    int64_t s0, s1, s2;
    int32_t b3;
};

template <typename T>
__device__ __forceinline__ T* kat(const KView& v, int64_t i, int64_t j, int64_t k, int64_t l) {
    return reinterpret_cast<T*>(v.p) + i * v.s0 + j * v.s1 + k * v.s2 + (v.b3 ? 0 : l);
}

struct BarrettLimbs;

/// Device tables of one base conversion (built by the ring layer; bconv_fused_kernel reads them).
struct BconvConsts {
    const BarrettLimbs* qinv;  // [r] Montgomery factors of the plain lifts of (Q_b / p_u)^-1 mod p_u
    const int64_t* mat;    // [nb][rd + 1][r] conversion matrix; row rd of each block: correction row
    const int2* mat2;      // [nb][rd][r] rows 0..rd-1 as limbs (m mod 2^29, m >> 29)
    const int64_t* qmodp;  // [nb][rd]
    const int64_t* qtab;   // [nb][rd][2 qhalf + 1] mul_mont(q, qmodp) for |q| <= qhalf
    const BarrettLimbs* r2;  // [rd] Montgomery factors R^2 mod p_j
    const int32_t* ucol;   // [nb][2] source column range of output block b
    int qhalf;
    int corr_limb;         // the correction row fits the limb products
    int shift;             // log2 of the correction's fixed-point scale
    int chunk;             // acc_before_reduce of the reference
    const int2* hmat;      // host: each block's own columns of mat2, [nb][rd][columns], hwords entries (0: none)
    int hwords;
};

/// First statement of every kernel: its launch may begin before the stream's previous kernel has finished
/// (launch_kernel). Waits until that kernel has completed and its writes are visible; before it only
/// constants (plans, twiddles, conversion tables: written by copies, never by kernels) may be read. Every
/// kernel launched by launch_kernel waits, so that a finished kernel implies all before it.
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

/// Keys of one launch of the key switch over the same gadget digits and summands (launch_keyswitch): each
/// with its automorphism and its output.
constexpr int KS_GROUP = 16;
struct KsGroup {
    int n;
    int64_t off[KS_GROUP];        // words from the first key's tensor to this key's (equal strides)
    int64_t* dst[KS_GROUP];       // [2B, r, dl, dk], equal strides
    const uint32_t* p2[KS_GROUP]; // optional Galois permutation applied to the digits and summands (apply_galois
    const uint32_t* p3[KS_GROUP]; // fused into the read, src/bfv.rs:819-820); null means identity
};

/// One digit of the dBFV reduction (launch_dbfv_split): its constants, in device memory.
struct DbfvSplit {
    const int64_t* rqinv;    // [r] Montgomery factors of the lifts
    const int64_t* mat;      // [limbs + 1][r]: the sums' matrix, the correction row last
    const int64_t* nbd[2];   // [r] mont^2(-b Delta 2^(64 k)) of overflow limb k
    const int64_t* delta[2]; // [r] mont^2(Delta 2^(64 k)) of carry limb k
    const int64_t* one;      // [r] mont(1)
    i128 f0, f1;             // Q and -Q^-1 modulo 2^log2m
    int limbs, shift, log2m;
    int corr_limb;           // the correction row's products with 29-bit limbs stay in range
    int have_carry, full_in, full_out;  // a carry comes in; the two sums need the double reduction
};

/// Montgomery moduli of one call, by value in the kernel's parameter space.
struct KMods {
    int64_t n[HC_MAX_MODS];
    int64_t ninv[HC_MAX_MODS];
    int64_t r2[HC_MAX_MODS];
    int64_t r3[HC_MAX_MODS];
};

// ------------------------------------------------------------------------------------------
// Exact arithmetic
// ------------------------------------------------------------------------------------------

__device__ __forceinline__ int64_t wadd(int64_t a, int64_t b) { return (int64_t)((uint64_t)a + (uint64_t)b); }
__device__ __forceinline__ int64_t wsub(int64_t a, int64_t b) { return (int64_t)((uint64_t)a - (uint64_t)b); }

/// The Barrett quotient q = floor((u x + 2^63) / 2^64) of signed u, x.
/// The high word of the unsigned 128-bit product U X is accumulated from 32-bit limbs with one
/// carry chain; the signed product follows from u x = U X - 2^64 ([u < 0] X + [x < 0] U), and the
/// rounding bit of "+ 2^63" is bit 63 of the low word (bit 31 of its upper limb).
__device__ __forceinline__ uint64_t barrett_q(int64_t u, int64_t x) {
    const uint32_t u0 = (uint32_t)u, u1 = (uint32_t)((uint64_t)u >> 32);
    const uint32_t x0 = (uint32_t)x, x1 = (uint32_t)((uint64_t)x >> 32);
    uint32_t r1, r2, r3;
    asm("{\n\t"
        "mul.hi.u32 %0, %3, %5;\n\t"
        "mad.lo.cc.u32 %0, %3, %6, %0;\n\t"
        "madc.hi.u32 %1, %3, %6, 0;\n\t"
        "mad.lo.cc.u32 %0, %4, %5, %0;\n\t"
        "madc.hi.cc.u32 %1, %4, %5, %1;\n\t"
        "madc.hi.u32 %2, %4, %6, 0;\n\t"
        "mad.lo.cc.u32 %1, %4, %6, %1;\n\t"
        "addc.u32 %2, %2, 0;\n\t"
        "}"
        : "=&r"(r1), "=&r"(r2), "=&r"(r3)
        : "r"(u0), "r"(u1), "r"(x0), "r"(x1));
    const uint64_t mx = (uint64_t)(x >> 63), mu = (uint64_t)(u >> 63);
    return ((((uint64_t)r3 << 32) | r2) - ((uint64_t)u & mx) - ((uint64_t)x & mu)) + (r1 >> 31);
}

/// Barrett multiplication by the constant (z, u): result z x + q n in wrapping 64-bit arithmetic
/// (|result| <= 3n/4 for |x| <= 2^63), q = barrett_q(u, x).
__device__ __forceinline__ int64_t bmul(int64_t z, int64_t u, int64_t x, int64_t n) {
    return (int64_t)((uint64_t)z * (uint64_t)x + barrett_q(u, x) * (uint64_t)n);
}

/// bmul by the Barrett constant of 1, the reduction step of the lazy transforms: that constant's
/// z is 1 for every odd modulus n >= 3 (1 is its own balanced residue), so z x is x and only the
/// quotient's product remains - the same result as bmul(1, u, x, n) with one product fewer.
__device__ __forceinline__ int64_t bmul1(int64_t u, int64_t x, int64_t n) {
    return (int64_t)((uint64_t)x + barrett_q(u, x) * (uint64_t)n);
}

/// Montgomery reduction of the 128-bit value hi:lo: ((x + m n) >> 64) with m = lo * (-n^-1).
/// The low words of x and m n cancel, so the carry out of the low word is (lo != 0).
__device__ __forceinline__ int64_t red128(uint64_t lo, int64_t hi, int64_t n, int64_t ninv) {
    int64_t m = (int64_t)(lo * (uint64_t)ninv);
    int64_t thi = __mul64hi(m, n);
    return (int64_t)((uint64_t)hi + (uint64_t)thi + (uint64_t)(lo != 0));
}
__device__ __forceinline__ int64_t red128(i128 x, int64_t n, int64_t ninv) {
    return red128((uint64_t)x, (int64_t)(x >> 64), n, ninv);
}

/// Montgomery product of two i64 values (the i128 product must stay within 2^63 n).
__device__ __forceinline__ int64_t mul_mont(int64_t a, int64_t b, int64_t n, int64_t ninv) {
    uint64_t lo = (uint64_t)a * (uint64_t)b;
    int64_t hi = __mul64hi(a, b);
    return red128(lo, hi, n, ninv);
}

/// Double Montgomery reduction of any i128 (x 2^-128 mod n, in [-n, n]).
__device__ __forceinline__ int64_t double_red128(i128 x, int64_t n, int64_t ninv) {
    uint64_t lo = (uint64_t)x;
    int64_t m = (int64_t)(lo * (uint64_t)ninv);
    i128 t = (i128)m * (i128)n;
    i128 carry = (i128)(((u128)lo + (u128)(uint64_t)t) >> 64);
    i128 r1 = (x >> 64) + (t >> 64) + carry;
    return red128(r1, n, ninv);
}

__device__ __forceinline__ int64_t to_mont64(int64_t x, int64_t n, int64_t ninv, int64_t r2) {
    return mul_mont(x, r2, n, ninv);
}
__device__ __forceinline__ int64_t to_mont128(i128 x, int64_t n, int64_t ninv, int64_t r3) {
    return mul_mont(red128(x, n, ninv), r3, n, ninv);
}

// ------------------------------------------------------------------------------------------
// The Barrett and Montgomery products in 32-bit limbs
// ------------------------------------------------------------------------------------------
// What bounds them: sm_103a multiplies 32 x 32 -> 64 bits (with a 64-bit addend) in 4 cycles per
// warp and SM partition and 32 x 32 -> 32 in 2, on one pipe; everything else can run beside it. So a
// product costs (4 x its wide products + 2 x its low ones) cycles, and these forms have as few of
// both as the exact result allows. The wide products are written as mad.lo.cc / madc.hi pairs,
// which ptxas fuses into one multiply-add; mad.wide with an addend becomes a multiply and two
// additions (measured: 6.3 against 4.2 cycles). Limbs are balanced: v = v1 2^32 + v0, v0 a signed word.

/// a b + c, signed 32 x 32 -> 64.
__device__ __forceinline__ int64_t mad_wide(int32_t a, int32_t b, int64_t c) {
    int64_t r;
    asm("{\n\t"
        ".reg .s32 l, h, cl, ch;\n\t"
        "mov.b64 {cl, ch}, %3;\n\t"
        "mad.lo.cc.s32 l, %1, %2, cl;\n\t"
        "madc.hi.s32 h, %1, %2, ch;\n\t"
        "mov.b64 %0, {l, h};\n\t"
        "}"
        : "=l"(r)
        : "r"(a), "r"(b), "l"(c));
    return r;
}
/// a b + c, unsigned 32 x 32 -> 64.
__device__ __forceinline__ uint64_t mad_wide_u(uint32_t a, uint32_t b, uint64_t c) {
    uint64_t r;
    asm("{\n\t"
        ".reg .u32 l, h, cl, ch;\n\t"
        "mov.b64 {cl, ch}, %3;\n\t"
        "mad.lo.cc.u32 l, %1, %2, cl;\n\t"
        "madc.hi.u32 h, %1, %2, ch;\n\t"
        "mov.b64 %0, {l, h};\n\t"
        "}"
        : "=l"(r)
        : "r"(a), "r"(b), "l"(c));
    return r;
}
__host__ __device__ __forceinline__ uint32_t lo32(int64_t x) { return (uint32_t)x; }
__host__ __device__ __forceinline__ uint32_t hi32(int64_t x) { return (uint32_t)((uint64_t)x >> 32); }
/// Upper balanced limb of x (the lower one is its low word, read as signed).
__host__ __device__ __forceinline__ int32_t bal_hi(int64_t x) { return (int32_t)(hi32(x) + (lo32(x) >> 31)); }
__device__ __forceinline__ int64_t pack64(uint32_t lo, uint32_t hi) { return (int64_t)(((uint64_t)hi << 32) | lo); }

/// A Barrett constant (z, u) in limbs (barrett_limbs).
struct __align__(16) BarrettLimbs {
    int32_t u0, u1;  // balanced limbs of u
    int32_t z0;      // z mod 2^32
    int32_t e1;      // upper balanced limb of e = u n + z 2^64 (n times the rounding error of u)
};

/// The modulus of barrett_mul and barrett_red: n = n1 2^32 + n0 balanced.
struct __align__(16) BarrettMod {
    int32_t n0, nn0, nn1;  // n0, -n0, -n1
    int32_t red_add, red_shift;
};

/// bmul(z, u, x, n), the same integer, for n < 2^57 and |x| <= 0.9 x 2^63 (plans whose schedule keeps
/// the lazy bounds there; csrc/ntt.cu checks it). With u x = u1 x1 2^64 + a 2^32 + (a word), the rounded
/// quotient is q = u1 x1 + round(a / 2^32), and the result's low word z x + q n modulo 2^32. The
/// upper word needs no multiple-precision sum: the result is -n f + e x / 2^64 exactly, where f is the
/// signed fraction that the rounding cut off, and x1 e1 - F n1 (F: the leading 32 bits of f) misses
/// that by less than 2^31 - at most 2^30 for n0, 0.9 x 2^30 for e0, 2^25 for F's cut-off and 2^23 for
/// e x0 - so that it and the low word name one integer.
/// Five wide products and three low ones, 27.6 cycles of the multiply pipe by count against 34 of bmul, and 14
/// instructions against 31: register-only chains run at 1367 G/s against 861 G/s (29.5 and 46.8 cycles per product),
/// butterflies at 1209 against 765.
__device__ __forceinline__ int64_t barrett_mul(const BarrettLimbs& w, int64_t x, const BarrettMod& m) {
    const int32_t x0 = (int32_t)lo32(x), x1 = bal_hi(x);
    const int64_t a = wadd(mad_wide(w.u1, x0, (int64_t)w.u0 * x1), __mulhi(w.u0, x0));
    const uint32_t q = (uint32_t)w.u1 * (uint32_t)x1 + (uint32_t)bal_hi(a);
    const uint32_t rl = (uint32_t)x0 * (uint32_t)w.z0 + q * (uint32_t)m.n0;
    const int64_t p = mad_wide((int32_t)lo32(a), m.nn1, mad_wide(x1, w.e1, (int64_t)1 << 31));
    uint32_t rh;  // (p - rl) >> 32
    asm("{\n\t"
        ".reg .u32 d;\n\t"
        "sub.cc.u32 d, %1, %2;\n\t"
        "subc.u32 %0, %3, 0;\n\t"
        "}"
        : "=r"(rh)
        : "r"(lo32(p)), "r"(rl), "r"(hi32(p)));
    return pack64(rl, rh);
}

/// Limbs of the constant (z, u) modulo n. u is taken modulo 2^64 into the range of two balanced
/// words, with z changed by the same multiple of n: q changes by a multiple of x and z x + q n keeps
/// its value.
inline BarrettLimbs barrett_limbs(i128 z, i128 u, int64_t n) {
    if (u >= ((i128)1 << 63) - ((i128)1 << 31)) u -= (i128)1 << 64, z += n;
    BarrettLimbs w;
    w.u0 = (int32_t)(uint32_t)u;
    w.u1 = (int32_t)((u - w.u0) >> 32);
    w.z0 = (int32_t)(uint32_t)z;
    w.e1 = bal_hi((int64_t)(u * n + (z << 64)));
    return w;
}

/// bmul1(u, x, n), the same integer, for a modulus whose constant of 1 is u = -2^k exactly: the
/// quotient is -ceil(x / 2^(64 - k) - 1/2), a shift of the upper word (red_add = 2^(31 - k) - 1,
/// red_shift = 32 - k). One wide product and a low one: 4156 G/s against 935 G/s.
__device__ __forceinline__ int64_t barrett_red(int64_t x, const BarrettMod& m) {
    int32_t t;
    asm("{\n\t"
        ".reg .u32 d;\n\t"
        "add.cc.u32 d, %1, 0xffffffff;\n\t"
        "addc.u32 %0, %2, %3;\n\t"
        "}"
        : "=r"(t)
        : "r"(lo32(x)), "r"(hi32(x)), "r"(m.red_add));
    const int32_t s = t >> m.red_shift;
    const int64_t r = mad_wide(s, m.nn0, x);
    return pack64(lo32(r), hi32(r) + (uint32_t)s * (uint32_t)m.nn1);
}

/// Montgomery modulus of mont_mul in limbs.
struct MontLimbs {
    int32_t n0, n1;  // balanced limbs of n
    uint32_t i0, i1;  // -n^-1 mod 2^64
    int64_t k;
};
__device__ __forceinline__ MontLimbs mont_limbs(int64_t n, int64_t ninv) {
    MontLimbs m;
    m.n0 = (int32_t)lo32(n), m.n1 = bal_hi(n);
    m.i0 = lo32(ninv), m.i1 = hi32(ninv);
    m.k = m.n0 >= 0 ? 0xc0000000ll : 0x40000000ll;
    return m;
}

/// mul_mont(a, b, n, ninv), the same integer, for n < 2^57, |a b| <= 2^63 n and |a|, |b| <= 0.9 x 2^63.
/// With m = m1 2^32 + m0 (m1 signed, m0 unsigned) the sum a b + m n is 2^64 (a1 b1 + m1 n1) + 2^32 M +
/// (a0 b0 + m0 n0) with M = a1 b0 + a0 b1 + m1 n0 + m0 n1, and divisible by 2^64. The last term lies
/// within [-2^62, 2^62 + 2^63) for n0 >= 0 and (-2^62 - 2^63, 2^62] for n0 < 0, an interval of
/// length 2^64, so M alone rounds to the right carry and its products are never formed: 12 products
/// instead of 18, 17 instructions instead of 44 (890 G/s against 524 G/s).
__device__ __forceinline__ int64_t mont_mul(int64_t a, int64_t b, const MontLimbs& m) {
    const int32_t a0 = (int32_t)lo32(a), a1 = bal_hi(a), b0 = (int32_t)lo32(b), b1 = bal_hi(b);
    const uint64_t l = (uint64_t)(uint32_t)a0 * (uint32_t)b0;
    const uint32_t l0 = lo32((int64_t)l);
    const uint32_t l1 = hi32((int64_t)l) + hi32(a) * (uint32_t)b0 + (uint32_t)a0 * hi32(b);
    const uint64_t q = (uint64_t)l0 * m.i0;
    const uint32_t q0 = lo32((int64_t)q);
    const int32_t q1 = (int32_t)(hi32((int64_t)q) + l1 * m.i0 + l0 * m.i1);
    int64_t c = mad_wide(q1, m.n0, mad_wide(a0, b1, mad_wide(a1, b0, m.k)));
    c = (int64_t)mad_wide_u(q0, (uint32_t)m.n1, (uint64_t)c);
    return mad_wide(q1, m.n1, mad_wide(a1, b1, c >> 32));
}

/// The Montgomery reduction (hi 2^64 + lo + m n) / 2^64 = red128(lo, hi, n, ninv), the same integer, for
/// n < 2^57 and |hi| <= 2^62: as in mont_mul only the middle limbs of m n are formed, here with the
/// upper word of lo beside them; what is left out lies in [0, 2^31 + 1) 2^32 for n0 >= 0 and (-2^31, 1) 2^32
/// for n0 < 0. Six products (21 cycles) instead of eight and their sign corrections.
__device__ __forceinline__ int64_t mont_red(uint64_t lo, int64_t hi, const MontLimbs& m) {
    const uint32_t l0 = lo32((int64_t)lo), l1 = hi32((int64_t)lo);
    const uint64_t q = (uint64_t)l0 * m.i0;
    const uint32_t q0 = lo32((int64_t)q);
    const int32_t q1 = (int32_t)(hi32((int64_t)q) + l1 * m.i0 + l0 * m.i1);
    const int64_t k = m.n0 >= 0 ? 0x80000001ll : 1;
    int64_t c = mad_wide(q1, m.n0, (int64_t)((uint64_t)l1 + (uint64_t)k));
    c = (int64_t)mad_wide_u(q0, (uint32_t)m.n1, (uint64_t)c);
    return mad_wide(q1, m.n1, wadd(c >> 32, hi));
}
/// double_red128 of hi 2^64 + lo (|hi| <= 2^62), the same integer: the first reduction fits one word, the
/// second has its sign as the upper word (floor division keeps the middle limbs' carry exact).
__device__ __forceinline__ int64_t mont_red_double(uint64_t lo, int64_t hi, const MontLimbs& m) {
    const int64_t r = mont_red(lo, hi, m);
    return mont_red((uint64_t)r, r >> 63, m);
}

/// mul_mont(a, b, n, ninv) for a constant b in the limbs of a Barrett product, for n < 2^57 and |a| <= 0.9 x
/// 2^63: with b' = b 2^-64 mod n and s = (b' 2^64 - b) / n the Montgomery product is b' a - q n, q =
/// round(s a / 2^64) (|a b / 2^64 - b' a + q n| <= n / 2, ties as the signed quotient of the reduction
/// takes them), which is barrett_mul modulo -n. 8 products instead of 12 of mont_mul.
__host__ __device__ __forceinline__ BarrettMod mont_const_mod(int64_t n) {
    BarrettMod m;
    m.n0 = (int32_t)(0u - lo32(n)), m.nn0 = (int32_t)lo32(n), m.nn1 = bal_hi(n);
    m.red_add = m.red_shift = 0;
    return m;
}
inline BarrettLimbs mont_const_limbs(int64_t b, int64_t n, int64_t ninv) {
    // b' 2^64 = b + n s with s = -b n^-1 mod 2^64; signed s keeps b' centred
    const i128 s = (int64_t)((uint64_t)b * (uint64_t)ninv);
    const i128 z = ((i128)b + s * n) >> 64;
    i128 u = s, zz = z;
    if (u >= ((i128)1 << 63) - ((i128)1 << 31)) u -= (i128)1 << 64, zz -= n;
    BarrettLimbs w;
    w.u0 = (int32_t)(uint32_t)u;
    w.u1 = (int32_t)((u - w.u0) >> 32);
    w.z0 = (int32_t)(uint32_t)zz;
    w.e1 = bal_hi(b);
    return w;
}
/// Whether |x| stays within the range of the limb products' variable operand, 0.9 x 2^63.
__device__ __forceinline__ bool limb_range(int64_t x) { return hi32(x) + 0x73000000u < 0xe6000000u; }
/// The constant b of mont_const_limbs: u = b ninv and n ninv = -1, both modulo 2^64.
__device__ __forceinline__ int64_t mont_const_value(const BarrettLimbs& w, int64_t n) {
    return (int64_t)(0 - (((uint64_t)(uint32_t)w.u1 << 32) + (uint64_t)(int64_t)w.u0) * (uint64_t)n);
}
__device__ __forceinline__ BarrettLimbs load_limbs(const BarrettLimbs* p) {
    const int4 a = __ldg(reinterpret_cast<const int4*>(p));
    return BarrettLimbs{a.x, a.y, a.z, a.w};
}

__device__ __forceinline__ i128 ld128(const void* p) {
    longlong2 v = *reinterpret_cast<const longlong2*>(p);
    return (i128)(((u128)(uint64_t)v.y << 64) | (uint64_t)v.x);
}
__device__ __forceinline__ void st128(void* p, i128 x) {
    longlong2 v;
    v.x = (long long)(uint64_t)x;
    v.y = (long long)(x >> 64);
    *reinterpret_cast<longlong2*>(p) = v;
}

// ------------------------------------------------------------------------------------------
// Batched CRT transforms
// ------------------------------------------------------------------------------------------

/// One (ring element, RNS factor) slab of a batched transform: deg_L' rows of deg_K residues.
struct CrtSlab {
    const void* plan2;     // NTT plan along dimension 2 (length deg_L')
    const void* plan3;     // NTT plan along dimension 3 (length deg_K)
    int64_t* data;         // row k at data + k * s2, contiguous
    const int64_t* op;     // operand slab (HC_CRT_MUL), row k at op + k * op_s2
    // CRT kernel of this factor along dimension 2 (deg_L' entries) and 3 (deg_K entries): Montgomery
    // words, or BarrettLimbs where the dimension's shape is specialised and its plan fixed (`shapes`)
    const int64_t* kl;
    const int64_t* kk;
    const int64_t* ikl;    // inverse kernels
    const int64_t* ikk;
    int64_t s2, op_s2;
    int64_t n, ninv;       // Montgomery modulus of the factor
    int32_t dl, dk;
    int32_t ops;           // HC_CRT_* bits
    int32_t shapes;        // specialised kernel shapes: dimension 3 | dimension 2 << 8 (0: generic)
};

/// Launch shape of the persistent batched-transform kernel (chosen by the autotuner).
struct CrtLaunch {
    int threads;      // per CTA
    int ctas_per_sm;  // persistent grid = SMs x this
    int logv;         // dimension-2 tile: 2^logv columns
};

// ------------------------------------------------------------------------------------------
// Host-side helpers shared by the translation units
// ------------------------------------------------------------------------------------------
namespace hc {

void set_error(const std::string& msg);
hc_status fail(hc_status st, const std::string& msg);
hc_status cuda_check(cudaError_t e, const char* what);
cudaStream_t stream_of(hc_context ctx);
void count_launch(hc_context ctx, uint64_t n = 1);
/// Every device or pinned-host allocation call of the library counts itself (hc_memory_stats).
void count_alloc();
uint64_t alloc_calls();
int num_sms(hc_context ctx);
size_t max_smem_optin(hc_context ctx);
int device_of(hc_context ctx);
hc_status intt_mul_mont64_dim(hc_context ctx, hc_view dst, const hc_ntt_plan* plans, size_t nplans, hc_data_dim dim,
                              hc_view mul, const hc_modulus* mods, size_t nmods);
hc_status ntt_kernel_dim(hc_context ctx, hc_view dst, const hc_view* src, const hc_ntt_plan* plans, size_t nplans,
                         hc_data_dim dim, hc_view mul, const BarrettLimbs* limbs, const hc_modulus* mods, size_t nmods);


/// kernel<<<grid, block, smem, stream>>>(args...), placed on the SMs as soon as the CTAs of the stream's previous
/// kernel have exited instead of after that kernel's completion has come back through the queue: the calls
/// here are chains of 3 to 80 short dependent launches (two transforms and a product of one field_36864 element at r = 16 72 ->
/// 52 us, a ct-mult at r = 5 215 -> 171, the homomorphic CRT step 5.25 -> 4.91 ms). No kernel lets its
/// successor start earlier (griddepcontrol.launch_dependents): waiting CTAs then hold slots that the rest
/// of the kernel and the ring's other stream use (64 us, 191 us, 5.13 ms; for grids of up to 608 or 2000 CTAs only 64, 195, 5.25).
template <class... P, class... A>
void launch_kernel(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, const A&... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid, cfg.blockDim = block, cfg.dynamicSmemBytes = smem, cfg.stream = stream;
    cfg.attrs = &attr, cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, args...);  // its error is the last error, which every caller reads
}

}  // namespace hc
