// Exact sums of products of 64-bit words in 29-bit limbs.
#pragma once
#include "common.cuh"

namespace {

// Exact multiply-accumulate of 64-bit words in limbs: v = v1 2^29 + v0 with 0 <= v0 < 2^29, three wide
// products per term (12.75 cycles of the multiply pipe; a 64 x 64 -> 128 product and its 128-bit
// addition take 33). The middle column x0 y1 + x1 y0 is the Karatsuba difference of the column sums, which
// may wrap: it is right modulo 2^64, so only x0 y0 (unsigned) and the middle column itself must stay
// in range.
constexpr int LIMB_BITS = 29;
constexpr int LIMB_TERMS = 28;   // terms whose column sums fit, for |x| < 2^57, |y| < 2^57 (middle: 28 2^58 < 2^63)
constexpr int LIMB_TERMS2 = 15;  // the same for |x|, |y| <= 2^58, twice a factor (middle: 15 2^59 < 2^63)

__device__ __forceinline__ int2 limb_split(int64_t v) {
    return make_int2((int)(v & ((1 << LIMB_BITS) - 1)), (int)(v >> LIMB_BITS));
}

/// hi:lo += a00 + a01 2^29 + a11 2^58 (a00 unsigned).
__device__ __forceinline__ void fold_limbs(uint64_t& lo, int64_t& hi, int64_t a00, int64_t a01, int64_t a11) {
    const u128 s = (u128)lo + (uint64_t)a00 + ((uint64_t)a01 << LIMB_BITS) + ((uint64_t)a11 << (2 * LIMB_BITS));
    lo = (uint64_t)s;
    hi = (int64_t)((uint64_t)hi + (uint64_t)(a01 >> (64 - LIMB_BITS)) + (uint64_t)(a11 >> (64 - 2 * LIMB_BITS)) +
                   (uint64_t)(s >> 64));
}

/// Column sums x0 y0, x1 y1 and (x0 + x1) (y0 + y1) of up to LIMB_TERMS terms.
struct LimbSum {
    int64_t a, b, m;
    __device__ __forceinline__ void zero() { a = b = m = 0; }
    __device__ __forceinline__ void mac(int2 x, int xs, int2 y, int ys) {
        a = mad_wide(x.x, y.x, a);
        b = mad_wide(x.y, y.y, b);
        m = mad_wide(xs, ys, m);
    }
    __device__ __forceinline__ void fold(uint64_t& lo, int64_t& hi) const { fold_limbs(lo, hi, a, wsub(wsub(m, a), b), b); }
};

}  // namespace
