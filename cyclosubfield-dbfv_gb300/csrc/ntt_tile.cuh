// The generic tile programme: any plan's stage program executed over a tile in shared memory (or, for
// lines that exceed it, in place in global memory). ntt_tile_kernel runs one HAL call with it, the
// batched-transform kernel the slabs without specialised shapes.
#pragma once
#include "ntt_plan.cuh"

namespace {

__device__ __forceinline__ uint32_t fdiv(uint32_t n, const FastDiv& f) {
    uint32_t t = __umulhi(f.m, n);
    return (t + ((n - t) >> f.s1)) >> f.s2;
}

/// Shared-memory slot of tile element i: for single lines (one vector) the low four index bits
/// are XOR-ed with the next four, so that groups of consecutive elements read by consecutive
/// threads fall into distinct banks; blocks of 16 stay in place, so the map is a permutation
/// whenever the line length is a multiple of 16.
__device__ __forceinline__ int sw(int i, bool on) { return on ? (i ^ ((i >> 4) & 15)) : i; }

/// Butterfly b of a stage -> position of its first leg (element index within the tile's
/// transform axis) and its twiddle block. Groups of `span` butterflies share a block; the legs of
/// a butterfly are `span` elements apart.
__device__ __forceinline__ int leg0(uint32_t bb, const DevStage& st, int* block) {
    uint32_t g = fdiv(bb, st.div_span);
    uint32_t off = bb - g * (uint32_t)st.span;
    uint32_t q = fdiv(g, st.div_nblocks);
    *block = (int)(g - q * st.div_nblocks.d);
    return (int)(g * (uint32_t)(st.stage_len * st.stride) + off);
}

struct Tile {
    int64_t* __restrict__ s;
    int len, logv;
    bool swz;
    __device__ __forceinline__ int64_t& at(int e, int v) const { return s[sw((e << logv) + v, swz)]; }
    /// n items per vector: their number over all vectors, and item b's index and vector.
    __device__ __forceinline__ int count(int n) const { return n << logv; }
    __device__ __forceinline__ uint32_t split(int b, int& v) const {
        v = b & ((1 << logv) - 1);
        return (uint32_t)(b >> logv);
    }
};

/// A whole slab of V vectors in shared memory: element e of vector v at e * se + v * sv.
struct SlabTile {
    int64_t* __restrict__ s;
    int len, V, se, sv;
    FastDiv div_v;
    __device__ __forceinline__ int64_t& at(int e, int v) const { return s[e * se + v * sv]; }
    __device__ __forceinline__ int count(int n) const { return n * V; }
    __device__ __forceinline__ uint32_t split(int b, int& v) const {
        const uint32_t q = fdiv((uint32_t)b, div_v);
        v = b - (int)q * V;
        return q;
    }
};

/// One forward stage (radix 2 or 3) over the tile in shared memory.
template <class TILE>
__device__ __forceinline__ void fwd_stage(const TILE& T, const DevStage st, const int64_t* __restrict__ tw,
                                          int64_t n, int64_t one_z, int64_t one_u, bool reduce_output) {
    const int radix = st.radix;
    const bool fuse = st.last && reduce_output;
    const int nbf = T.count(T.len / radix);
    for (int b = threadIdx.x; b < nbf; b += blockDim.x) {
        int block, v;
        const uint32_t bb = T.split(b, v);
        const int e = leg0(bb, st, &block);
        int64_t& x = T.at(e, v);
        int64_t& y = T.at(e + st.span, v);
        if (radix == 2) {
            int64_t z = tw[2 * (st.tw_off + block)], u = tw[2 * (st.tw_off + block) + 1];
            bool skip = st.skip_ok && z == 1;
            int64_t a = x, yv = y;
            if (st.reduce_before) {  // the reference's reduction pass, applied as the operands are read
                a = bmul1(one_u, a, n);
                yv = bmul1(one_u, yv, n);
            }
            int64_t t = skip ? yv : bmul(z, u, yv, n);
            int64_t o0 = wadd(a, t), o1 = wsub(a, t);
            if (fuse) {
                o0 = bmul1(one_u, o0, n);
                o1 = bmul1(one_u, o1, n);
            }
            x = o0;
            y = o1;
        } else {
            int64_t& zr = T.at(e + 2 * st.span, v);
            const int64_t* w = tw + 2 * (st.tw_off + 6 * block);
            bool skip = st.skip_ok && w[0] == 1;
            int64_t a = x, bv = y, c = zr;
            if (st.reduce_before) {
                a = bmul1(one_u, a, n);
                bv = bmul1(one_u, bv, n);
                c = bmul1(one_u, c, n);
            }
            int64_t t_b = skip ? bv : bmul(w[0], w[1], bv, n);
            int64_t t_bz = bmul(w[2], w[3], bv, n);
            int64_t t_bzz = bmul(w[4], w[5], bv, n);
            int64_t t_c = skip ? c : bmul(w[6], w[7], c, n);
            int64_t t_cz = bmul(w[8], w[9], c, n);
            int64_t t_czz = bmul(w[10], w[11], c, n);
            int64_t o0 = wadd(wadd(a, t_b), t_c), o1 = wadd(wadd(a, t_bz), t_czz), o2 = wadd(wadd(a, t_bzz), t_cz);
            if (fuse) {
                o0 = bmul1(one_u, o0, n);
                o1 = bmul1(one_u, o1, n);
                o2 = bmul1(one_u, o2, n);
            }
            x = o0;
            y = o1;
            zr = o2;
        }
    }
}

/// One inverse stage (radix 2 or 3) over the tile in shared memory.
template <class TILE>
__device__ __forceinline__ void inv_stage(const TILE& T, const DevStage st, const int64_t* __restrict__ tw,
                                          int64_t n, int64_t il_z, int64_t il_u, int64_t one_z, int64_t one_u) {
    const int radix = st.radix;
    const bool fused = st.last;
    const int nbf = T.count(T.len / radix);
    for (int b = threadIdx.x; b < nbf; b += blockDim.x) {
        int block, v;
        const uint32_t bb = T.split(b, v);
        const int e = leg0(bb, st, &block);
        int64_t& x = T.at(e, v);
        int64_t& y = T.at(e + st.span, v);
        if (radix == 2) {
            int64_t yz, yu;
            if (fused) {
                yz = il_z;
                yu = il_u;
            } else {
                yz = tw[2 * (st.tw_off + block)];
                yu = tw[2 * (st.tw_off + block) + 1];
            }
            bool skip = !fused && yz == 1;
            int64_t y0 = x, y1 = y;
            if (st.reduce_before) {
                y0 = bmul1(one_u, y0, n);
                y1 = bmul1(one_u, y1, n);
            }
            int64_t sum = wadd(y0, y1), dif = wsub(y0, y1);
            x = fused ? bmul(yz, yu, sum, n) : sum;
            y = skip ? dif : bmul(yz, yu, dif, n);
        } else {
            int64_t& zr = T.at(e + 2 * st.span, v);
            int64_t yz, yu, zz, zu;
            if (fused) {
                yz = zz = il_z;
                yu = zu = il_u;
            } else {
                const int64_t* w = tw + 2 * (st.tw_off + 2 * block);
                yz = w[0], yu = w[1], zz = w[2], zu = w[3];
            }
            bool skip = !fused && yz == 1;
            const int64_t* zt = tw + 2 * st.zeta_off;
            int64_t y0 = x, y1 = y, y2 = zr;
            if (st.reduce_before) {
                y0 = bmul1(one_u, y0, n);
                y1 = bmul1(one_u, y1, n);
                y2 = bmul1(one_u, y2, n);
            }
            int64_t y1z = bmul(zt[0], zt[1], y1, n), y1zz = bmul(zt[2], zt[3], y1, n);
            int64_t y2z = bmul(zt[0], zt[1], y2, n), y2zz = bmul(zt[2], zt[3], y2, n);
            int64_t s0 = wadd(wadd(y0, y1), y2);
            int64_t sy = wadd(wadd(y0, y1zz), y2z), sz = wadd(wadd(y0, y1z), y2zz);
            x = fused ? bmul(yz, yu, s0, n) : s0;
            y = skip ? sy : bmul(yz, yu, sy, n);
            zr = skip ? sz : bmul(zz, zu, sz, n);
        }
    }
}

/// K consecutive forward radix-2 stages of one factor in registers. Group element m lies at
/// g * glen + o + m * span; at the q-th stage of the pass the butterflies pair m with
/// m + 2^(K-1-q) and use the twiddle of block block0 * 2^q + (m >> (K-q)).
template <int K, class TILE>
__device__ __forceinline__ void fwd_pass_r2(const TILE& T, const DevPass ps, const DevStage* sts,
                                            const int64_t* __restrict__ tw, int64_t n, int64_t one_z, int64_t one_u,
                                            bool reduce_output) {
    constexpr int M = 1 << K;
    // the stage parameters, read once into registers
    int tw_off[K];
    bool red[K], skip_ok[K], fuse[K];
#pragma unroll
    for (int q = 0; q < K; q++) {
        const DevStage& st = sts[ps.first + q];
        tw_off[q] = st.tw_off;
        red[q] = st.reduce_before;
        skip_ok[q] = st.skip_ok;
        fuse[q] = st.last && reduce_output;
    }
    const int ng = T.count(T.len >> K);
    for (int gi = threadIdx.x; gi < ng; gi += blockDim.x) {
        int v;
        const uint32_t gg = T.split(gi, v);
        const uint32_t g = fdiv(gg, ps.div_span);
        const int o = (int)(gg - g * (uint32_t)ps.span);
        const int block0 = (int)(g - fdiv(g, ps.div_nb) * (uint32_t)ps.nb);
        const int base = (int)g * ps.glen + o;
        int64_t x[M];
#pragma unroll
        for (int m = 0; m < M; m++) x[m] = T.at(base + m * ps.span, v);
#pragma unroll
        for (int q = 0; q < K; q++) {
            if (red[q]) {
#pragma unroll
                for (int m = 0; m < M; m++) x[m] = bmul1(one_u, x[m], n);
            }
            const int half = M >> (q + 1);
#pragma unroll
            for (int j = 0; j < M / 2; j++) {
                const int m1 = ((j / half) * 2 * half) + (j % half), m2 = m1 + half;
                const int tb = block0 * (1 << q) + (m1 >> (K - q));
                const int64_t z = tw[2 * (tw_off[q] + tb)], u = tw[2 * (tw_off[q] + tb) + 1];
                const bool skip = skip_ok[q] && z == 1;
                const int64_t a = x[m1];
                const int64_t t = skip ? x[m2] : bmul(z, u, x[m2], n);
                int64_t o0 = wadd(a, t), o1 = wsub(a, t);
                if (fuse[q]) {
                    o0 = bmul1(one_u, o0, n);
                    o1 = bmul1(one_u, o1, n);
                }
                x[m1] = o0;
                x[m2] = o1;
            }
        }
#pragma unroll
        for (int m = 0; m < M; m++) T.at(base + m * ps.span, v) = x[m];
    }
}

/// K consecutive inverse radix-2 stages (stage lengths growing) in registers: at the q-th stage
/// of the pass the butterflies pair m with m + 2^q and use the twiddle of block
/// blockK * 2^(K-1-q) + (m >> (q+1)), blockK being the group's block at the pass's last stage.
template <int K, class TILE>
__device__ __forceinline__ void inv_pass_r2(const TILE& T, const DevPass ps, const DevStage* sts,
                                            const int64_t* __restrict__ tw, int64_t n, int64_t il_z, int64_t il_u,
                                            int64_t one_z, int64_t one_u) {
    constexpr int M = 1 << K;
    int tw_off[K];
    bool red[K], fused[K];
#pragma unroll
    for (int q = 0; q < K; q++) {
        const DevStage& st = sts[ps.first + q];
        tw_off[q] = st.tw_off;
        red[q] = st.reduce_before;
        fused[q] = st.last;
    }
    const int ng = T.count(T.len >> K);
    for (int gi = threadIdx.x; gi < ng; gi += blockDim.x) {
        int v;
        const uint32_t gg = T.split(gi, v);
        const uint32_t g = fdiv(gg, ps.div_span);
        const int o = (int)(gg - g * (uint32_t)ps.span);
        const int blockK = (int)(g - fdiv(g, ps.div_nb) * (uint32_t)ps.nb);
        const int base = (int)g * ps.glen + o;
        int64_t x[M];
#pragma unroll
        for (int m = 0; m < M; m++) x[m] = T.at(base + m * ps.span, v);
#pragma unroll
        for (int q = 0; q < K; q++) {
            if (red[q]) {
#pragma unroll
                for (int m = 0; m < M; m++) x[m] = bmul1(one_u, x[m], n);
            }
            const int dist = 1 << q;
#pragma unroll
            for (int j = 0; j < M / 2; j++) {
                const int m1 = ((j >> q) << (q + 1)) | (j & (dist - 1)), m2 = m1 + dist;
                const int tb = blockK * (1 << (K - 1 - q)) + (m1 >> (q + 1));
                int64_t yz, yu;
                if (fused[q]) {
                    yz = il_z;
                    yu = il_u;
                } else {
                    yz = tw[2 * (tw_off[q] + tb)];
                    yu = tw[2 * (tw_off[q] + tb) + 1];
                }
                const bool skip = !fused[q] && yz == 1;
                const int64_t y0 = x[m1], y1 = x[m2];
                const int64_t sum = wadd(y0, y1), dif = wsub(y0, y1);
                x[m1] = fused[q] ? bmul(yz, yu, sum, n) : sum;
                x[m2] = skip ? dif : bmul(yz, yu, dif, n);
            }
        }
#pragma unroll
        for (int m = 0; m < M; m++) T.at(base + m * ps.span, v) = x[m];
    }
}

/// A plan's stage programme and constants, in global or shared memory.
struct Program {
    const DevStage *fwd, *inv;
    const DevPass *fpass, *ipass;
    int nfpass, nipass;
    int64_t n, one_z, one_u, il_z, il_u;
    const int64_t* tw;
};
__device__ __forceinline__ Program program_of(const DevPlanHeader* P, const int64_t* tw) {
    return Program{P->fwd, P->inv, P->fpass, P->ipass, P->nfpass, P->nipass, P->n, P->one_z, P->one_u, P->invlen_z, P->invlen_u, tw};
}

/// All passes of a programme over a tile in place (modes as tile_run, without the multiplication); a
/// block barrier after each.
template <class TILE>
__device__ __forceinline__ void run_passes(const TILE& T, const Program& P, int mode) {
    const bool inverse = mode & 1;
    const int npass = inverse ? P.nipass : P.nfpass;
    for (int pi = 0; pi < npass; pi++) {
        const DevPass ps = inverse ? P.ipass[pi] : P.fpass[pi];
        if (ps.kind == 0) {
            if (inverse) inv_stage(T, P.inv[ps.first], P.tw, P.n, P.il_z, P.il_u, P.one_z, P.one_u);
            else fwd_stage(T, P.fwd[ps.first], P.tw, P.n, P.one_z, P.one_u, mode == 0);
        } else if (inverse) {
            if (ps.k == 3) inv_pass_r2<3>(T, ps, P.inv, P.tw, P.n, P.il_z, P.il_u, P.one_z, P.one_u);
            else if (ps.k == 2) inv_pass_r2<2>(T, ps, P.inv, P.tw, P.n, P.il_z, P.il_u, P.one_z, P.one_u);
            else inv_pass_r2<1>(T, ps, P.inv, P.tw, P.n, P.il_z, P.il_u, P.one_z, P.one_u);
        } else {
            if (ps.k == 3) fwd_pass_r2<3>(T, ps, P.fwd, P.tw, P.n, P.one_z, P.one_u, mode == 0);
            else if (ps.k == 2) fwd_pass_r2<2>(T, ps, P.fwd, P.tw, P.n, P.one_z, P.one_u, mode == 0);
            else fwd_pass_r2<1>(T, ps, P.fwd, P.tw, P.n, P.one_z, P.one_u, mode == 0);
        }
        __syncthreads();
    }
    // plans without factors (length 1): the inverse scales by 1^-1, the reduced forward
    // reduces; an unreduced forward leaves the data unchanged
    if (npass == 0 && (mode == 0 || inverse)) {
        const int64_t fz = inverse ? P.il_z : P.one_z, fu = inverse ? P.il_u : P.one_u;
        for (int b = threadIdx.x; b < T.count(T.len); b += blockDim.x) {
            int v;
            const int e = (int)T.split(b, v);
            T.at(e, v) = bmul(fz, fu, T.at(e, v), P.n);
        }
        __syncthreads();
    }
}

/// Where one tile lives in global memory and where its Montgomery multiplier (modes 2 and 3)
/// comes from: element (e, v) of the tile is g[e * ge + v] and is multiplied by
/// mulp[e * me + v * mv] modulo (mn, mi).
struct TileIO {
    int64_t* g;
    int64_t ge;
    int64_t ncol;  // valid columns of the tile (a dimension-2 block at the end of the axis)
    const int64_t* mulp;
    int64_t me, mv;
    int64_t mn, mi;
};

/// One tile transformed by plan P, twiddles `tw` already staged. mode 0: forward (reduced),
/// 1: inverse, 2: forward unreduced + Montgomery multiplication, 3: inverse + Montgomery
/// multiplication. With `use_smem` the tile is copied to `s` (len x 2^logv elements) and back;
/// otherwise (single lines too long for shared memory) it is worked on in place in global memory.
/// Ends with a block barrier, so the caller may reuse the shared memory at once.
__device__ __forceinline__ void tile_run(const DevPlanHeader* __restrict__ P, const int64_t* __restrict__ tw,
                                         int64_t* s, int len, int logv, bool use_smem, int mode,
                                         const TileIO& io) {
    const int V = 1 << logv, vmask = V - 1;
    const int total = len * V;
    Tile T{use_smem ? s : io.g, len, logv, use_smem && logv == 0 && (len & 15) == 0};
    if (use_smem) {
        for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
            int e = idx >> logv, v = idx & vmask;
            T.at(e, v) = v < io.ncol ? io.g[e * io.ge + v] : 0;
        }
    }
    __syncthreads();
    run_passes(T, program_of(P, tw), mode);
    if (mode & 2) {
        for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
            int e = idx >> logv, v = idx & vmask;
            if (v >= io.ncol) continue;
            T.at(e, v) = mul_mont(T.at(e, v), io.mulp[e * io.me + v * io.mv], io.mn, io.mi);
        }
        __syncthreads();
    }
    if (use_smem) {
        for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
            int e = idx >> logv, v = idx & vmask;
            if (v < io.ncol) io.g[e * io.ge + v] = T.at(e, v);
        }
    }
    __syncthreads();
}

/// Copies the twiddle table of plan P to shared memory (no barrier).
__device__ __forceinline__ void stage_twiddles(const DevPlanHeader* P, int64_t* dst) {
    const int64_t* twg = reinterpret_cast<const int64_t*>(P + 1);
    for (int idx = threadIdx.x; idx < 2 * P->ntw; idx += blockDim.x) dst[idx] = twg[idx];
}

}  // namespace
