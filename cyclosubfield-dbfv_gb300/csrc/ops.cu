// Pointwise, contraction, correction and permutation kernels of the Backend trait
// (cyclosubfield-dbfv/src/hal/cpu.rs:591-1122). Every kernel walks the destination as
// (line, l) with l the contiguous dimension 3; sources are broadcast through zero strides.
#include "limb_sum.cuh"

namespace {

enum PwOp {
    OP_ASSIGN,
    OP_ASSIGN_NARROW,
    OP_ASSIGN_I128,
    OP_ADD_I64,
    OP_SUB_I64,
    OP_ADD_I128,
    OP_FMA_I64,
    OP_MUL_I64,
    OP_MUL_MONT,
    OP_ADD_RED_DOUBLE,
    OP_RED_DOUBLE,
    OP_ADD_RED,
    OP_RED,
    OP_I128_TO_MONT,
    OP_I64_TO_MONT,
};

/// What operation OP reads at one position: the destination's old value (p, wp) and its operands, 8-byte
/// words or 16-byte ones (w*).
struct PwIn {
    int64_t p, a, b;
    i128 wp, wa;
};

constexpr bool pw_wide_dst(int op) { return op == OP_ASSIGN_I128 || op == OP_ADD_I128 || op == OP_FMA_I64 || op == OP_MUL_I64; }
constexpr bool pw_wide_src(int op) {
    return op == OP_ASSIGN_NARROW || op == OP_ASSIGN_I128 || op == OP_ADD_I128 || op == OP_ADD_RED_DOUBLE ||
           op == OP_RED_DOUBLE || op == OP_ADD_RED || op == OP_RED || op == OP_I128_TO_MONT;
}
constexpr bool pw_reads_dst(int op) {
    return op == OP_ADD_I64 || op == OP_SUB_I64 || op == OP_ADD_I128 || op == OP_FMA_I64 || op == OP_MUL_MONT ||
           op == OP_ADD_RED_DOUBLE || op == OP_ADD_RED || op == OP_I64_TO_MONT;
}

template <int OP>
__device__ __forceinline__ void pw_load(PwIn& v, const KView& d, const KView& a, const KView& b, int64_t i, int64_t j,
                                        int64_t k, int64_t l) {
    if constexpr (pw_reads_dst(OP)) {
        if constexpr (pw_wide_dst(OP)) v.wp = ld128(kat<longlong2>(d, i, j, k, l));
        else v.p = *kat<int64_t>(d, i, j, k, l);
    }
    if constexpr (pw_wide_src(OP)) v.wa = ld128(kat<longlong2>(a, i, j, k, l));
    else if constexpr (OP != OP_I64_TO_MONT) v.a = *kat<int64_t>(a, i, j, k, l);
    if constexpr (OP == OP_FMA_I64 || OP == OP_MUL_I64) v.b = *kat<int64_t>(b, i, j, k, l);
}

template <int OP>
__device__ __forceinline__ void pw_store(const PwIn& v, const KView& d, const KMods& m, int64_t i, int64_t j, int64_t k,
                                         int64_t l) {
    if constexpr (pw_wide_dst(OP)) {
        i128 r;
        if constexpr (OP == OP_ASSIGN_I128) r = v.wa;
        else if constexpr (OP == OP_ADD_I128) r = (i128)((u128)v.wp + (u128)v.wa);
        else if constexpr (OP == OP_FMA_I64) r = (i128)((u128)v.wp + (u128)((i128)v.a * (i128)v.b));
        else r = (i128)v.a * (i128)v.b;
        st128(kat<longlong2>(d, i, j, k, l), r);
    } else {
        int64_t r;
        if constexpr (OP == OP_ASSIGN) r = v.a;
        else if constexpr (OP == OP_ASSIGN_NARROW) r = (int64_t)(uint64_t)v.wa;  // low word of the i128
        else if constexpr (OP == OP_ADD_I64) r = wadd(v.p, v.a);
        else if constexpr (OP == OP_SUB_I64) r = wsub(v.p, v.a);
        else if constexpr (OP == OP_MUL_MONT) r = mul_mont(v.p, v.a, m.n[j], m.ninv[j]);
        else if constexpr (OP == OP_RED_DOUBLE) r = double_red128(v.wa, m.n[j], m.ninv[j]);
        else if constexpr (OP == OP_ADD_RED_DOUBLE) r = wadd(v.p, double_red128(v.wa, m.n[j], m.ninv[j]));
        else if constexpr (OP == OP_RED) r = red128(v.wa, m.n[j], m.ninv[j]);
        else if constexpr (OP == OP_ADD_RED) r = wadd(v.p, red128(v.wa, m.n[j], m.ninv[j]));
        else if constexpr (OP == OP_I128_TO_MONT) r = to_mont128(v.wa, m.n[j], m.ninv[j], m.r3[j]);
        else r = to_mont64(v.p, m.n[j], m.ninv[j], m.r2[j]);
        *kat<int64_t>(d, i, j, k, l) = r;
    }
}

template <int OP>
__global__ void __launch_bounds__(256) pw_kernel(KView d, KView a, KView b, KMods m, int64_t lines, int chunks) {
    grid_wait();
    const int64_t tiles = lines * chunks;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        int64_t line = tile / chunks;
        int64_t l = (tile - line * chunks) * blockDim.x + threadIdx.x;
        if (l >= d.n3) continue;
        int64_t k = line % d.n2, r = line / d.n2;
        int64_t j = r % d.n1, i = r / d.n1;
        PwIn v;
        pw_load<OP>(v, d, a, b, i, j, k, l);
        pw_store<OP>(v, d, m, i, j, k, l);
    }
}

/// pw_kernel over a 2-D grid: blockIdx.y is the destination line (i, j, k), decomposed once per
/// thread with 32-bit arithmetic, and each thread takes LINE_SPAN / 256 positions of it, so that
/// the per-element work is the operation itself (the tile form pays several 64-bit divisions per
/// element). Used while the line count fits the grid's y dimension. What bounds the short launches of
/// one ciphertext is the latency of the reads, so all of a thread's are in flight before its first store: a
/// trait-path ct-mult at field_36864 r = 16 (42 of its 77 launches are of this file) 842 -> 819 us.
constexpr int LINE_SPAN = 1024, LINE_STEPS = LINE_SPAN / 256;

template <int OP>
__global__ void __launch_bounds__(256) pw_line_kernel(KView d, KView a, KView b, KMods m) {
    grid_wait();
    const int line = (int)blockIdx.y;
    const int k = line % (int)d.n2, r = line / (int)d.n2;
    const int j = r % (int)d.n1, i = r / (int)d.n1;
    const int64_t l0 = (int64_t)blockIdx.x * LINE_SPAN;
    PwIn v[LINE_STEPS];
#pragma unroll
    for (int s = 0; s < LINE_STEPS; s++)
        if (l0 + 256 * s + threadIdx.x < d.n3) pw_load<OP>(v[s], d, a, b, i, j, k, l0 + 256 * s + threadIdx.x);
#pragma unroll
    for (int s = 0; s < LINE_STEPS; s++)
        if (l0 + 256 * s + threadIdx.x < d.n3) pw_store<OP>(v[s], d, m, i, j, k, l0 + 256 * s + threadIdx.x);
}

/// dst[i,j,k,l] = sum_u lhs[li,j,u,0] * rhs[ri,u,k,l] (src/hal/cpu.rs:791-818), i128 wrapping.
/// Four output rows j per pass share each rhs load. The columns u go in chunks of LIMB_TERMS: a warp
/// splits a chunk's matrix entries into limbs and lists its columns that are not zero in all four
/// rows (a gadget conversion matrix is zero outside each digit's columns; the others add nothing), four warps
/// four chunks at a time, so that a short line waits for the matrix once.
/// A chunk whose words are all below 2^57 in absolute value (residues and centred constants are) is summed
/// in limbs, found out for the matrix by the staging warp and for the right-hand side by each warp as it
/// goes; a warp that meets a larger word sums the chunk and the rest of the tile as 128-bit products, so every
/// word is allowed.
/// What bounds it: the multiply pipe, 13 cycles a term instead of 33; a trait-path ct-mult (five
/// products at field_36864 r = 16) 921 -> 839 us. Four columns unrolled in the limb sums or four CTAs per SM spill
/// (852, 854). [2, 18 x 16, 12, 3072] of small words 20.5 us, 33 with larger ones on the right and 30 in the matrix
/// (as 128-bit products alone, two at a time, 37).
constexpr int MATMUL_ROWS = 4, MATMUL_UNROLL = 2;
/// MATMUL_STAGED: 1 for matrices of one chunk, whose staging indexes then fold away, else 4.
template <int MATMUL_STAGED>
__global__ void __launch_bounds__(256, 3) matmul_kernel(KView d, KView lhs, KView rhs, int64_t U, int64_t lines,
                                                        int chunks) {
    grid_wait();
    __shared__ __align__(16) int2 sm[MATMUL_STAGED][LIMB_TERMS][MATMUL_ROWS];
    __shared__ __align__(16) int64_t sw[MATMUL_STAGED][LIMB_TERMS][MATMUL_ROWS];  // the entries whole
    __shared__ int sidx[MATMUL_STAGED][LIMB_TERMS], scount[MATMUL_STAGED], slarge[MATMUL_STAGED];
    const int64_t tiles = lines * chunks;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int64_t line = tile / chunks;  // (i, k)
        const int64_t l = (tile - line * chunks) * blockDim.x + threadIdx.x;
        const int64_t k = line % d.n2, i = line / d.n2;
        // a thread past the line's end reads its last position and stores nothing
        const int64_t* x0 = kat<int64_t>(rhs, i, 0, k, l < d.n3 ? l : d.n3 - 1);
        bool beyond = false;  // the warp has met a larger word of this tile
        for (int64_t j = 0; j < d.n1; j += MATMUL_ROWS) {
            const int rows = (int)(d.n1 - j < MATMUL_ROWS ? d.n1 - j : MATMUL_ROWS);
            uint64_t lo[MATMUL_ROWS] = {};
            int64_t hi[MATMUL_ROWS] = {};
            for (int64_t u0 = 0; u0 < U; u0 += LIMB_TERMS) {
                const int g = (int)(u0 / LIMB_TERMS) % MATMUL_STAGED;
                if (g == 0) {
                    __syncthreads();  // the previous chunks' readers are done
                    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
                    const int64_t u = u0 + LIMB_TERMS * warp + lane;
                    if (warp < MATMUL_STAGED && u0 + LIMB_TERMS * warp < U) {
                        const bool in = lane < LIMB_TERMS && u < U;
                        int64_t c[MATMUL_ROWS];
                        uint64_t any = 0, large = 0;
#pragma unroll
                        for (int q = 0; q < MATMUL_ROWS; q++) {
                            c[q] = in && q < rows ? *kat<int64_t>(lhs, i, j + q, u, 0) : 0;
                            any |= (uint64_t)c[q];
                            large |= ((uint64_t)c[q] + ((uint64_t)1 << 57)) >> 58;
                        }
                        const unsigned mask = __ballot_sync(0xffffffffu, any != 0);
                        const int wide = __any_sync(0xffffffffu, large != 0);
                        if (any != 0) {
                            const int at = __popc(mask & ((1u << lane) - 1));
                            sidx[warp][at] = lane;
#pragma unroll
                            for (int q = 0; q < MATMUL_ROWS; q++) sm[warp][at][q] = limb_split(c[q]), sw[warp][at][q] = c[q];
                        }
                        if (lane == 0) scount[warp] = __popc(mask), slarge[warp] = wide;
                    }
                    __syncthreads();
                }
                const int n = scount[g];
                const int64_t* xu = x0 + u0 * rhs.s1;
                if (!beyond && !slarge[g]) {
                    uint64_t large = 0;
                    LimbSum s[MATMUL_ROWS];
#pragma unroll
                    for (int q = 0; q < MATMUL_ROWS; q++) s[q].zero();
#pragma unroll MATMUL_UNROLL
                    for (int t = 0; t < n; t++) {
                        const int64_t v = xu[sidx[g][t] * rhs.s1];
                        large |= ((uint64_t)v + ((uint64_t)1 << 57)) >> 58;
                        const int2 x = limb_split(v);
                        const int xs = x.x + x.y;
#pragma unroll
                        for (int q = 0; q < MATMUL_ROWS; q++) {
                            const int2 w = sm[g][t][q];
                            s[q].mac(x, xs, w, w.x + w.y);
                        }
                    }
                    beyond = __any_sync(0xffffffffu, large != 0);
                    if (!beyond) {
#pragma unroll
                        for (int q = 0; q < MATMUL_ROWS; q++) s[q].fold(lo[q], hi[q]);
                        continue;
                    }
                }
#pragma unroll 4
                for (int t = 0; t < n; t++) {
                    const int64_t v = xu[sidx[g][t] * rhs.s1];
#pragma unroll
                    for (int q = 0; q < MATMUL_ROWS; q++) {
                        const u128 s = (((u128)(uint64_t)hi[q] << 64) | lo[q]) + (u128)((i128)sw[g][t][q] * (i128)v);
                        lo[q] = (uint64_t)s, hi[q] = (int64_t)(s >> 64);
                    }
                }
            }
            if (l < d.n3)
#pragma unroll
                for (int q = 0; q < MATMUL_ROWS; q++)
                    if (q < rows) st128(kat<longlong2>(d, i, j + q, k, l), (i128)(((u128)(uint64_t)hi[q] << 64) | lo[q]));
        }
    }
}

struct Terms {
    KView l[HC_MAX_TERMS];
    KView r[HC_MAX_TERMS];
    int n;
};

/// dst = sum_t lhs[t] * rhs[t], overwriting (src/hal/cpu.rs:707-788).
__global__ void __launch_bounds__(256) inner_product_kernel(KView d, Terms terms, int64_t lines, int chunks) {
    grid_wait();
    const int64_t tiles = lines * chunks;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        int64_t line = tile / chunks;
        int64_t l = (tile - line * chunks) * blockDim.x + threadIdx.x;
        if (l >= d.n3) continue;
        int64_t k = line % d.n2, r = line / d.n2;
        int64_t j = r % d.n1, i = r / d.n1;
        i128 acc = 0;
        for (int t = 0; t < terms.n; t++) {
            i128 prod = (i128)*kat<int64_t>(terms.l[t], i, j, k, l) * (i128)*kat<int64_t>(terms.r[t], i, j, k, l);
            acc = (i128)((u128)acc + (u128)prod);
        }
        st128(kat<longlong2>(d, i, j, k, l), acc);
    }
}

/// inner_product_kernel over the line grid of pw_line_kernel. FULL: the CTA's span lies within the line; a
/// shorter line's threads read only what they store (repeating its last position instead, 100 x 8 x 2 lines of 96
/// positions took 36.0 us for twelve terms, 31.5 this way), at the price of reads that wait for their own test.
template <bool FULL>
__device__ __forceinline__ void inner_product_span(const KView& d, const Terms& terms, int i, int j, int k, int64_t l0) {
    auto in = [&](int s) { return FULL || l0 + 256 * s + threadIdx.x < d.n3; };
    i128 acc[LINE_STEPS];
#pragma unroll
    for (int s = 0; s < LINE_STEPS; s++) acc[s] = 0;
    for (int t = 0; t < terms.n; t++) {
        int64_t x[LINE_STEPS] = {}, y[LINE_STEPS] = {};
#pragma unroll
        for (int s = 0; s < LINE_STEPS; s++)
            if (in(s)) {
                x[s] = *kat<int64_t>(terms.l[t], i, j, k, l0 + 256 * s + threadIdx.x);
                y[s] = *kat<int64_t>(terms.r[t], i, j, k, l0 + 256 * s + threadIdx.x);
            }
#pragma unroll
        for (int s = 0; s < LINE_STEPS; s++) acc[s] = (i128)((u128)acc[s] + (u128)((i128)x[s] * (i128)y[s]));
    }
#pragma unroll
    for (int s = 0; s < LINE_STEPS; s++)
        if (in(s)) st128(kat<longlong2>(d, i, j, k, l0 + 256 * s + threadIdx.x), acc[s]);
}
__global__ void __launch_bounds__(256) inner_product_line_kernel(KView d, Terms terms) {
    grid_wait();
    const int line = (int)blockIdx.y;
    const int k = line % (int)d.n2, r = line / (int)d.n2;
    const int j = r % (int)d.n1, i = r / (int)d.n1;
    const int64_t l0 = (int64_t)blockIdx.x * LINE_SPAN;
    if (l0 + LINE_SPAN <= d.n3) inner_product_span<true>(d, terms, i, j, k, l0);
    else inner_product_span<false>(d, terms, i, j, k, l0);
}

/// dst[i,j,k,l] += red(((lhs[i,0,k,l] + 2^(shift-1)) >> shift) * rhs[ri,j,0,0])
/// (src/hal/cpu.rs:950-980)
__global__ void __launch_bounds__(256) bconv_correct_kernel(KView d, KView lhs, KView rhs, KMods m, int shift,
                                                            int64_t lines, int chunks) {
    grid_wait();
    const i128 half = (i128)1 << (shift - 1);
    const int64_t tiles = lines * chunks;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        int64_t line = tile / chunks;
        int64_t l = (tile - line * chunks) * blockDim.x + threadIdx.x;
        if (l >= d.n3) continue;
        int64_t k = line % d.n2, r = line / d.n2;
        int64_t j = r % d.n1, i = r / d.n1;
        i128 x = ld128(kat<longlong2>(lhs, i, 0, k, l));
        int64_t q = (int64_t)((i128)((u128)x + (u128)half) >> shift);
        int64_t c = *kat<int64_t>(rhs, i, j, 0, 0);
        int64_t* p = kat<int64_t>(d, i, j, k, l);
        *p = wadd(*p, mul_mont(q, c, m.n[j], m.ninv[j]));
    }
}

/// bconv_correct_kernel over the line grid of pw_line_kernel. AHEAD: a thread's positions whose reads are in flight
/// together: all while the tensor stays in L2 ([2, 23, 4, 12288] 13.5 us, one at a time 14.5), one beyond
/// ([24, 34, 12, 3072] 138 us, where four together took 155).
template <int AHEAD>
__global__ void __launch_bounds__(256) bconv_correct_line_kernel(KView d, KView lhs, KView rhs, KMods m, int shift) {
    grid_wait();
    const i128 half = (i128)1 << (shift - 1);
    const int line = (int)blockIdx.y;
    const int k = line % (int)d.n2, r = line / (int)d.n2;
    const int j = r % (int)d.n1, i = r / (int)d.n1;
    const int64_t c = *kat<int64_t>(rhs, i, j, 0, 0);
    const int64_t n = m.n[j], ninv = m.ninv[j];
    const int64_t l0 = (int64_t)blockIdx.x * LINE_SPAN;
    auto add = [&](i128 x, int64_t v, int64_t l) {
        *kat<int64_t>(d, i, j, k, l) = wadd(v, mul_mont((int64_t)((i128)((u128)x + (u128)half) >> shift), c, n, ninv));
    };
    if constexpr (AHEAD == 1) {
        const int64_t l1 = min(l0 + LINE_SPAN, d.n3);
        for (int64_t l = l0 + threadIdx.x; l < l1; l += 256) add(ld128(kat<longlong2>(lhs, i, 0, k, l)), *kat<int64_t>(d, i, j, k, l), l);
    } else {
        i128 x[LINE_STEPS];
        int64_t v[LINE_STEPS];
#pragma unroll
        for (int s = 0; s < LINE_STEPS; s++) {
            const int64_t l = min(l0 + 256 * s + threadIdx.x, d.n3 - 1);  // past the end: the last position again
            x[s] = ld128(kat<longlong2>(lhs, i, 0, k, l)), v[s] = *kat<int64_t>(d, i, j, k, l);
        }
#pragma unroll
        for (int s = 0; s < LINE_STEPS; s++)
            if (l0 + 256 * s + threadIdx.x < d.n3) add(x[s], v[s], l0 + 256 * s + threadIdx.x);
    }
}

/// src/hal/cpu.rs:983-1015 (wide == 0) and :1018-1057 (wide == 1)
__global__ void __launch_bounds__(256) bconv_pow2_kernel(KView d, KView src, i128 f0, i128 f1, int shift, int log2m,
                                                         int wide, int64_t lines, int chunks) {
    grid_wait();
    const i128 half = (i128)1 << (shift - 1);
    const u128 mask = ((u128)1 << log2m) - 1;
    const i128 modulus = (i128)1 << log2m;
    const i128 mhalf = modulus / 2;
    const int64_t tiles = lines * chunks;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        int64_t line = tile / chunks;  // (i, k)
        int64_t l = (tile - line * chunks) * blockDim.x + threadIdx.x;
        if (l >= d.n3) continue;
        int64_t k = line % d.n2, i = line / d.n2;
        i128 v, corr;
        if (wide) {
            i128 lo = ld128(kat<longlong2>(src, i, 0, k, l)), hi = ld128(kat<longlong2>(src, i, 1, k, l));
            v = (i128)((u128)lo + ((u128)hi << 64));
            corr = ld128(kat<longlong2>(src, i, 2, k, l));
        } else {
            v = ld128(kat<longlong2>(src, i, 0, k, l));
            corr = ld128(kat<longlong2>(src, i, 1, k, l));
        }
        i128 quot = (i128)((u128)corr + (u128)half) >> shift;
        u128 x = ((u128)v - (u128)quot * (u128)f0) * (u128)f1;
        i128 red = (i128)(x & mask);
        i128 c = red > mhalf ? red - modulus : red;
        if (wide) {
            int64_t lo = (int64_t)(uint64_t)c;
            int64_t hi = (int64_t)((c - (i128)lo) >> 64);
            *kat<int64_t>(d, i, 0, k, l) = lo;
            *kat<int64_t>(d, i, 1, k, l) = hi;
        } else {
            *kat<int64_t>(d, i, 0, k, l) = (int64_t)c;
        }
    }
}

/// dst[e] = src[perm[e]] along dimension 2 or 3 (src/hal/cpu.rs:1086-1122)
__global__ void __launch_bounds__(256) permute_kernel(KView d, KView s, const uint32_t* perm, int dim, int64_t lines,
                                                      int chunks) {
    grid_wait();
    const int64_t tiles = lines * chunks;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        int64_t line = tile / chunks;
        int64_t l = (tile - line * chunks) * blockDim.x + threadIdx.x;
        if (l >= d.n3) continue;
        int64_t k = line % d.n2, r = line / d.n2;
        int64_t j = r % d.n1, i = r / d.n1;
        int64_t v = dim == 2 ? *kat<int64_t>(s, i, j, perm[k], l) : *kat<int64_t>(s, i, j, k, perm[l]);
        *kat<int64_t>(d, i, j, k, l) = v;
    }
}

/// Grid of the line kernels, or false when the line count exceeds the grid's y dimension.
bool line_grid(const KView& d, int64_t lines, dim3* grid) {
    if (lines > 65535 || d.n1 > INT32_MAX || d.n2 > INT32_MAX) return false;
    *grid = dim3((unsigned)((d.n3 + LINE_SPAN - 1) / LINE_SPAN), (unsigned)lines, 1);
    return true;
}

void grid_for(hc_context ctx, const KView& d, int64_t lines, int* chunks, unsigned* blocks) {
    *chunks = (int)((d.n3 + 255) / 256);
    int64_t tiles = lines * *chunks;
    int64_t cap = (int64_t)hc::num_sms(ctx) * 32;
    *blocks = (unsigned)(tiles < cap ? (tiles > 0 ? tiles : 1) : cap);
}

}  // namespace

namespace hc {

hc_status launch_pointwise(hc_context ctx, int op, const KView& d, const KView& a, const KView& b, const KMods& m) {
    int64_t lines = d.n0 * d.n1 * d.n2;
    if (lines == 0 || d.n3 == 0) return HC_OK;
    int chunks;
    unsigned blocks;
    grid_for(ctx, d, lines, &chunks, &blocks);
    cudaStream_t s = stream_of(ctx);
    dim3 lg;
    const bool by_line = line_grid(d, lines, &lg);
#define HC_PW(OPV)                                                      \
    case OPV:                                                           \
        if (by_line) hc::launch_kernel(pw_line_kernel<OPV>, lg, 256, 0, s, d, a, b, m); \
        else hc::launch_kernel(pw_kernel<OPV>, blocks, 256, 0, s, d, a, b, m, lines, chunks); \
        break;
    switch (op) {
        HC_PW(OP_ASSIGN)
        HC_PW(OP_ASSIGN_NARROW)
        HC_PW(OP_ASSIGN_I128)
        HC_PW(OP_ADD_I64)
        HC_PW(OP_SUB_I64)
        HC_PW(OP_ADD_I128)
        HC_PW(OP_FMA_I64)
        HC_PW(OP_MUL_I64)
        HC_PW(OP_MUL_MONT)
        HC_PW(OP_ADD_RED_DOUBLE)
        HC_PW(OP_RED_DOUBLE)
        HC_PW(OP_ADD_RED)
        HC_PW(OP_RED)
        HC_PW(OP_I128_TO_MONT)
        HC_PW(OP_I64_TO_MONT)
        default: return fail(HC_ERR_ARG, "unknown pointwise operation");
    }
#undef HC_PW
    count_launch(ctx);
    return cuda_check(cudaGetLastError(), "pointwise kernel launch");
}

hc_status launch_matmul(hc_context ctx, const KView& d, const KView& lhs, const KView& rhs, int64_t U) {
    int64_t lines = d.n0 * d.n2;
    if (lines == 0 || d.n3 == 0 || d.n1 == 0) return HC_OK;
    int chunks;
    unsigned blocks;
    grid_for(ctx, d, lines, &chunks, &blocks);
    hc::launch_kernel(U <= LIMB_TERMS ? matmul_kernel<1> : matmul_kernel<4>, blocks, 256, 0, stream_of(ctx), d, lhs, rhs, U, lines,
                      chunks);
    count_launch(ctx);
    return cuda_check(cudaGetLastError(), "matmul kernel launch");
}

hc_status launch_inner_product(hc_context ctx, const KView& d, const KView* l, const KView* r, int n) {
    int64_t lines = d.n0 * d.n1 * d.n2;
    if (lines == 0 || d.n3 == 0) return HC_OK;
    Terms t;
    for (int i = 0; i < n; i++) t.l[i] = l[i], t.r[i] = r[i];
    t.n = n;
    int chunks;
    unsigned blocks;
    dim3 lg;
    if (line_grid(d, lines, &lg)) {
        hc::launch_kernel(inner_product_line_kernel, lg, 256, 0, stream_of(ctx), d, t);
    } else {
        grid_for(ctx, d, lines, &chunks, &blocks);
        hc::launch_kernel(inner_product_kernel, blocks, 256, 0, stream_of(ctx), d, t, lines, chunks);
    }
    count_launch(ctx);
    return cuda_check(cudaGetLastError(), "inner product kernel launch");
}

hc_status launch_bconv_correct(hc_context ctx, const KView& d, const KView& lhs, const KView& rhs, const KMods& m,
                               int shift) {
    int64_t lines = d.n0 * d.n1 * d.n2;
    if (lines == 0 || d.n3 == 0) return HC_OK;
    int chunks;
    unsigned blocks;
    dim3 lg;
    if (line_grid(d, lines, &lg)) {
        const bool in_l2 = d.n0 * d.n1 * d.n2 * d.n3 * 8 <= ((int64_t)64 << 20);
        hc::launch_kernel(in_l2 ? bconv_correct_line_kernel<LINE_STEPS> : bconv_correct_line_kernel<1>, lg, 256, 0, stream_of(ctx), d,
                          lhs, rhs, m, shift);
    } else {
        grid_for(ctx, d, lines, &chunks, &blocks);
        hc::launch_kernel(bconv_correct_kernel, blocks, 256, 0, stream_of(ctx), d, lhs, rhs, m, shift, lines, chunks);
    }
    count_launch(ctx);
    return cuda_check(cudaGetLastError(), "bconv correction kernel launch");
}

hc_status launch_bconv_pow2(hc_context ctx, const KView& d, const KView& src, i128 f0, i128 f1, int shift, int log2m,
                            int wide) {
    int64_t lines = d.n0 * d.n2;
    if (lines == 0 || d.n3 == 0) return HC_OK;
    int chunks;
    unsigned blocks;
    grid_for(ctx, d, lines, &chunks, &blocks);
    hc::launch_kernel(bconv_pow2_kernel, blocks, 256, 0, stream_of(ctx), d, src, f0, f1, shift, log2m, wide, lines, chunks);
    count_launch(ctx);
    return cuda_check(cudaGetLastError(), "bconv pow2 kernel launch");
}

hc_status launch_permute(hc_context ctx, const KView& d, const KView& s, const uint32_t* perm, int dim) {
    int64_t lines = d.n0 * d.n1 * d.n2;
    if (lines == 0 || d.n3 == 0) return HC_OK;
    int chunks;
    unsigned blocks;
    grid_for(ctx, d, lines, &chunks, &blocks);
    hc::launch_kernel(permute_kernel, blocks, 256, 0, stream_of(ctx), d, s, perm, dim, lines, chunks);
    count_launch(ctx);
    return cuda_check(cudaGetLastError(), "permute kernel launch");
}

}  // namespace hc
