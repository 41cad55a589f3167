// The persistent batched-transform kernel; crt_batch*.cu instantiate one slab class each.
#pragma once
#include "ntt_run.cuh"
#include "ntt_tile.cuh"

namespace {

/// One pass of a batched transform over a whole slab: its deg_L' lines (dimension 3) or its
/// column blocks of 2^logv columns (dimension 2). Modes as tile_run; `mulrow` is the CRT kernel
/// row of the pass (modes 2 and 3 along dimension 2, mode 2 along dimension 3), while mode 3
/// along dimension 3 multiplies by the slab's operand.
template <bool GENERIC, int CLS>
__device__ __forceinline__ void slab_pass(const CrtSlab& S, const DevPlanHeader* P, const int64_t* tw, int64_t* s,
                                          int dim, int mode, const int64_t* mulrow, int logv) {
    // specialised kernels for slabs whose plans have the fixed schedule (bit 16: dimension-3
    // plan, bit 17: dimension-2 plan), the generic tile programme otherwise
    const int shape = dim == 3 ? (S.shapes & 0xff) : ((S.shapes >> 8) & 0xff);
    const bool fix = (S.shapes >> (dim == 3 ? 16 : 17)) & 1;
    if (fix && dim == 3 && (shape == HC_SHAPE_L3072 || shape == HC_SHAPE_L12288)) {
        for (int k = 0; k < S.dl; k++) {
            int64_t* g = S.data + k * S.s2;
            const int64_t* mulp = mode == 3 ? S.op + k * S.op_s2 : mulrow;
            if (CLS != 2 && (CLS == 1 || shape == HC_SHAPE_L3072)) {
                if (mode == 2) run_line3072<6, true>(P, s, g, mulp, 1, S.n, S.ninv);
                else if (mode == 3) run_line3072<3, true>(P, s, g, mulp, 1, S.n, S.ninv);
                else run_line3072<1, true>(P, s, g, mulp, 1, S.n, S.ninv);
            } else if (CLS != 1) {
                // one 4096-residue block in shared memory at a time (crt_slab_tile_words)
                const auto c = make_ctx<fast::CtxL>(P);
                if (mode & 1) {  // modes 1 (inverse) and 3 (inverse, then the operand product)
                    with_sched<HC_SHAPE_L12288, true, true>(P, [&](const auto& sch) {
                        if (mode == 3) fast::line12288_seq<3>(sch, c, s, g, mulp, 1, S.n, S.ninv);
                        else fast::line12288_seq<1>(sch, c, s, g, mulp, 1, S.n, S.ninv);
                    });
                } else {  // mode 2: forward, then the kernel product
                    with_sched<HC_SHAPE_L12288, false, true>(
                        P, [&](const auto& sch) { fast::line12288_seq<6>(sch, c, s, g, mulp, 1, S.n, S.ninv); });
                }
            }
            __syncthreads();
        }
        return;
    }
    if (fix && dim == 2 && (shape == HC_SHAPE_C12 || shape == HC_SHAPE_C4)) {
        for (int l = threadIdx.x; l < S.dk; l += blockDim.x) {
            int64_t* g = S.data + l;
            if (CLS != 2 && (CLS == 1 || shape == HC_SHAPE_C12)) {
                if (mode == 2) run_column<HC_SHAPE_C12, 6, true>(P, g, S.s2, g, S.s2, mulrow, 1, S.n, S.ninv);
                else run_column<HC_SHAPE_C12, 1, true>(P, g, S.s2, g, S.s2, mulrow, 1, S.n, S.ninv);
            } else if (CLS != 1) {
                if (mode == 2) run_column<HC_SHAPE_C4, 6, true>(P, g, S.s2, g, S.s2, mulrow, 1, S.n, S.ninv);
                else run_column<HC_SHAPE_C4, 1, true>(P, g, S.s2, g, S.s2, mulrow, 1, S.n, S.ninv);
            }
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
/// field_36864's [4, 3] x [2, 3, 8, 64] shapes, 2 field_49152's [4] x [3, 64, 64], 0 any - so that
/// a launch carries only its class's code.
template <bool GENERIC, int CLS, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB)
    crt_batch_kernel(const CrtSlab* __restrict__ slabs, int nslabs, int* counter, int logv, int tile_words) {
    extern __shared__ int64_t smem[];
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
        if constexpr (GENERIC) {  // the specialised passes read theirs from the plan (L1-cached)
            stage_twiddles(P2, tw2);
            stage_twiddles(P3, tw3);
            __syncthreads();
        }
        if (S.ops & HC_CRT_FORWARD) {
            slab_pass<GENERIC, CLS>(S, P2, tw2, smem, 2, 2, S.kl, logv);
            slab_pass<GENERIC, CLS>(S, P3, tw3, smem, 3, 2, S.kk, logv);
            slab_pass<GENERIC, CLS>(S, P2, tw2, smem, 2, 1, nullptr, logv);
            slab_pass<GENERIC, CLS>(S, P3, tw3, smem, 3, (S.ops & HC_CRT_MUL) ? 3 : 1, nullptr, logv);
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
            slab_pass<GENERIC, CLS>(S, P2, tw2, smem, 2, 2, S.ikl, logv);
            slab_pass<GENERIC, CLS>(S, P3, tw3, smem, 3, 2, S.ikk, logv);
            slab_pass<GENERIC, CLS>(S, P2, tw2, smem, 2, 1, nullptr, logv);
            slab_pass<GENERIC, CLS>(S, P3, tw3, smem, 3, 1, nullptr, logv);
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
