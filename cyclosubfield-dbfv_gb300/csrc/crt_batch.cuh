// The persistent batched-transform kernel; crt_batch*.cu instantiate one slab class each.
#pragma once
#include "ntt_run.cuh"
#include "ntt_tile.cuh"

namespace {

/// Whether a slab has field_49152's shapes with fixed plans in both dimensions (slab12288_half).
__host__ __device__ inline bool crt_slab_12288(int32_t shapes) {
    return (shapes & 0x3ffff) == (HC_SHAPE_L12288 | HC_SHAPE_C4 << 8 | 3 << 16);
}

/// Half a transform of a field_49152 slab, as crt_slab.cu's two kernels run it: the lead pass over its
/// positions, then its twelve blocks one after the other. MODE 6: forward, times the kernels kl [4] and
/// kk [12288] (limbs); 1: inverse; 11: inverse, times the operand.
template <int MODE>
__device__ __forceinline__ void slab12288_half(const CrtSlab& S, const DevPlanHeader* P2, const DevPlanHeader* P3, int64_t* s,
                                               const int64_t* kl, const int64_t* kk) {
    const fast::CtxL c3 = make_ctx<fast::CtxL>(P3);
    {
        const fast::CtxL c2 = make_ctx<fast::CtxL>(P2);
        const BarrettLimbs* m2 = reinterpret_cast<const BarrettLimbs*>(kl);
        for (int p = threadIdx.x; p < 4096; p += blockDim.x) {
            if (P3->cls == 57) lead12288<(MODE & 1), 57>(c2, c3, S.data + p, S.s2, S.data + p, S.s2, m2, S.n);
            else lead12288<(MODE & 1), 56>(c2, c3, S.data + p, S.s2, S.data + p, S.s2, m2, S.n);
        }
    }
    __syncthreads();
    const auto mont = fast::make_mont<fast::CtxL, MODE>(S.n, S.ninv);
    with_sched<HC_SHAPE_L12288, (MODE & 1) != 0, true>(P3, [&](const auto& sch) {
        int4* tws = reinterpret_cast<int4*>(s + 4096);
        fast::stage_tail_twiddles<(MODE & 1) != 0>(fast::CtaTeam{}, c3, sch, tws, 1, 63, 7);
        for (int q = 0; q < 12; q++) {
            const int k = q / 3, blk = q - 3 * (q / 3);
            const int64_t* mulp = MODE == 6    ? fast::block_multiplier<MODE>(kk, 1, blk)
                                  : MODE == 11 ? S.op + k * S.op_s2 + 4096 * blk
                                               : nullptr;
            fast::block4096<MODE>(fast::CtaTeam{}, sch, c3, s, tws, S.data + k * S.s2 + 4096 * blk, mulp, 1, mont);
            __syncthreads();  // the tile is refilled by the next block
        }
    });
}

/// The [2, 3, 8, 64] lines of a slab. 256 threads work as two teams of 128 with a tile each: a line's
/// 384 register groups and 12 tail rows fill 128 threads exactly and 256 to three quarters.
template <int MODE>
__device__ __forceinline__ void slab_lines3072(const CrtSlab& S, const DevPlanHeader* P, int64_t* s, const int64_t* mulrow) {
    const int teams = blockDim.x == 256 ? 2 : 1, t = (int)threadIdx.x / 128 % teams;
    const fast::PartTeam tm{(int)threadIdx.x - 128 * t, (int)blockDim.x / teams, 1 + t};
    int64_t* tile = s + t * LINE3072_WORDS;
    for (int k = t; k < S.dl; k += teams) {
        run_line3072<MODE, true>(tm, P, tile, S.data + k * S.s2, MODE == 11 ? S.op + k * S.op_s2 : mulrow, 1, S.n,
                                 S.ninv, k == t);
        tm.sync();
    }
    __syncthreads();
}

/// One pass of a batched transform over a whole slab: its deg_L' lines (dimension 3) or its
/// column blocks of 2^logv columns (dimension 2). Modes as tile_run; `mulrow` is the CRT kernel
/// row of the pass (modes 2 and 3 along dimension 2, mode 2 along dimension 3), while mode 3
/// along dimension 3 multiplies by the slab's operand.
template <bool GENERIC, int CLS>
__device__ __forceinline__ void slab_pass(const CrtSlab& S, const DevPlanHeader* P, const int64_t* tw, int64_t* s,
                                          int dim, int mode, const int64_t* mulrow, int logv) {
    // specialised kernels for slabs whose plans are fixed (bit 16: dimension-3 plan, bit 17: dimension-2
    // plan), the generic tile programme otherwise
    const int shape = dim == 3 ? (S.shapes & 0xff) : ((S.shapes >> 8) & 0xff);
    const bool fix = CLS != 3 && ((S.shapes >> (dim == 3 ? 16 : 17)) & 1);
    if (fix && dim == 3 && shape == HC_SHAPE_L3072) {
        if (mode == 2) slab_lines3072<6>(S, P, s, mulrow);
        else if (mode == 3) slab_lines3072<11>(S, P, s, mulrow);
        else slab_lines3072<1>(S, P, s, mulrow);
        return;
    }
    if (fix && dim == 2 && shape == HC_SHAPE_C12) {
        for (int l = threadIdx.x; l < S.dk; l += blockDim.x) {
            int64_t* g = S.data + l;
            if (mode == 2) run_column<HC_SHAPE_C12, 6, true>(P, g, S.s2, g, S.s2, mulrow, 1, S.n, S.ninv);
            else run_column<HC_SHAPE_C12, 1, true>(P, g, S.s2, g, S.s2, mulrow, 1, S.n, S.ninv);
        }
        __syncthreads();
        return;
    }
    if constexpr (!GENERIC) return;  // the launcher sends only specialised slabs to this form
    TileIO io;
    io.mn = S.n, io.mi = S.ninv;
    io.me = 1, io.mv = 0;
    if (dim == 3) {
        io.ge = 1, io.ncol = 1;
        for (int k = 0; k < S.dl; k++) {
            io.g = S.data + k * S.s2;
            io.mulp = mode == 3 ? S.op + k * S.op_s2 : mulrow;
            tile_run(P, tw, s, S.dk, 0, true, mode, io);
        }
    } else {
        const int V = 1 << logv;
        io.ge = S.s2;
        io.mulp = mulrow;
        for (int c0 = 0; c0 < S.dk; c0 += V) {
            io.g = S.data + c0;
            io.ncol = S.dk - c0 < V ? S.dk - c0 : V;
            tile_run(P, tw, s, S.dl, logv, true, mode, io);
        }
    }
}

/// Persistent batched CRT transforms: every CTA takes the next slab from `counter` and runs the
/// slab's whole operation (period -> CRT, Montgomery product with the operand, CRT -> period, as
/// its `ops` say) before taking another. Slabs of different fields and RNS lengths mix freely;
/// the passes are the HAL transforms' passes in the same order (src/ring.rs:1118-1161), the
/// operand product fused into the epilogue of the forward transform's last pass.
/// GENERIC = false: every slab has the specialised line and column shapes with compiled-in
/// schedules (both large fields' rings), so the generic tile programme is left out; MINB: the CTAs
/// of MAXT threads per SM the register allocation must allow (256 threads: 2 -> 128 registers,
/// 3 -> 80, 4 -> 64 with some spilling), chosen through the autotuned launch shape. GENERIC = true serves other slabs. CLS: the slabs' shape class - 1 every slab has
/// field_36864's [4, 3] x [2, 3, 8, 64] shapes, 2 field_49152's [4] x [3, 64, 64], 3 none with a specialised
/// dimension, 0 any - so that a launch carries only its class's code (pb_to_crt of four field_18 elements 22.7 us
/// with all of it, 18.5 as class 3).
template <bool GENERIC, int CLS, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB)
    crt_batch_kernel(const CrtSlab* __restrict__ slabs, int nslabs, int* counter, int logv, int tile_words) {
    grid_wait();
    extern __shared__ __align__(16) int64_t smem[];
    __shared__ int s_next;
    for (;;) {
        __syncthreads();  // every thread has read s_next and left the previous slab's tiles
        if (threadIdx.x == 0) s_next = atomicAdd(counter, 1);
        __syncthreads();
        const int si = s_next;
        if (si >= nslabs) return;
        const CrtSlab S = slabs[si];
        const DevPlanHeader* P2 = reinterpret_cast<const DevPlanHeader*>(S.plan2);
        const DevPlanHeader* P3 = reinterpret_cast<const DevPlanHeader*>(S.plan3);
        int64_t* tw2 = smem + tile_words;
        int64_t* tw3 = tw2 + 2 * P2->ntw;
        if constexpr (GENERIC) {  // the specialised passes stage theirs with each tile
            stage_twiddles(P2, tw2);
            stage_twiddles(P3, tw3);
            __syncthreads();
        }
        // one half of a transform: dimension 2, then dimension 3 (modes as slab_pass)
        const bool slab12288 = CLS == 2 || (CLS == 0 && crt_slab_12288(S.shapes));
        auto half = [&](auto mode3, int mode2, const int64_t* kl, const int64_t* kk) {
            constexpr int M = decltype(mode3)::value;
            if constexpr (CLS == 0 || CLS == 2) {
                if (slab12288) return slab12288_half<M == 2 ? 6 : M == 3 ? 11 : M>(S, P2, P3, smem, kl, kk);
            }
            if constexpr (CLS != 2) {
                slab_pass<GENERIC, CLS>(S, P2, tw2, smem, 2, mode2, kl, logv);
                slab_pass<GENERIC, CLS>(S, P3, tw3, smem, 3, M, kk, logv);
            }
        };
        if (S.ops & HC_CRT_FORWARD) {
            half(std::integral_constant<int, 2>{}, 2, S.kl, S.kk);
            if (S.ops & HC_CRT_MUL) half(std::integral_constant<int, 3>{}, 1, nullptr, nullptr);
            else half(std::integral_constant<int, 1>{}, 1, nullptr, nullptr);
        } else if (S.ops & HC_CRT_MUL) {
            const int total = S.dl * S.dk;
            for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
                const int k = idx / S.dk, l = idx - k * S.dk;
                int64_t* x = S.data + k * S.s2 + l;
                *x = mul_mont(*x, S.op[k * S.op_s2 + l], S.n, S.ninv);
            }
            __syncthreads();
        }
        if (S.ops & HC_CRT_INVERSE) {
            half(std::integral_constant<int, 2>{}, 2, S.ikl, S.ikk);
            half(std::integral_constant<int, 1>{}, 1, nullptr, nullptr);
        }
    }
}

/// The specialised kernel of class CLS for a launch shape.
typedef void (*CrtBatchKernel)(const CrtSlab*, int, int*, int, int);
template <int CLS>
CrtBatchKernel crt_batch_variant(int ctas_per_sm) {
    return ctas_per_sm >= 4   ? crt_batch_kernel<false, CLS, 256, 4>
           : ctas_per_sm == 3 ? crt_batch_kernel<false, CLS, 256, 3>
                              : crt_batch_kernel<false, CLS, 256, 2>;
}

}  // namespace
