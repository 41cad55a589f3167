// Dimension-2 columns [4, 3] (field_36864) and [4] (field_49152): one thread per column.
#include "ntt_run.cuh"

namespace {

#ifndef HC_COL12_MIN_BLOCKS
#define HC_COL12_MIN_BLOCKS 4  // resident CTAs per SM the [4, 3] column kernel's registers must allow
#endif

/// Specialised dimension-2 NTT: one thread per column (i, j, l), CTAs over (i, j, column block).
template <int SHAPE, int MODE, bool FIX>
__global__ void __launch_bounds__(HC_COL_THREADS, SHAPE == HC_SHAPE_C12 ? HC_COL12_MIN_BLOCKS : MODE == 2 && FIX ? 6 : 4) ntt_col_kernel(KView t, PlanPtrs plans, KView mul, KMods mods,
                                                                    int ncb, KView src) {
    grid_wait();
    // tiles last to first: a transform's column pass follows a line pass (or the input's producer)
    // that wrote the tensor first to last, so the CTAs scheduled first read what is still in L2,
    // and the next line pass, first to last, starts on what this pass wrote last
    const int64_t tile = gridDim.x - 1 - blockIdx.x;
    const int64_t cb = tile % ncb, r = tile / ncb;
    const int64_t j = r % t.n1, i = r / t.n1;
    const DevPlanHeader* P = plans.p[j];
    const int64_t l = cb * HC_COL_THREADS + threadIdx.x;
    if (l >= t.n3) return;
    int64_t* g = reinterpret_cast<int64_t*>(t.p) + i * t.s0 + j * t.s1 + l;
    const int64_t* mulp = nullptr;
    int64_t ms = 0, mn = 0, mi = 0;
    if (MODE & 2) {
        mulp = multiplier<MODE>(mul, i, j, 0, l);
        ms = mul.s2;
        mn = mods.n[j], mi = mods.ninv[j];
    }
    // out of place (src.p set): the column is read from src, written to t
    const int64_t* gs = src.p ? reinterpret_cast<const int64_t*>(src.p) + i * src.s0 + j * src.s1 + l : g;
    run_column<SHAPE, MODE, FIX>(P, g, t.s2, gs, src.p ? src.s2 : t.s2, mulp, ms, mn, mi);
}

template <int SHAPE, int MODE, bool FIX>
hc_status launch(hc_context ctx, const KView& t, const PlanPtrs& pp, const KView& mul, const KMods& mods, int64_t tiles, int ncb,
                      const KView& src) {
    hc::launch_kernel(ntt_col_kernel<SHAPE, MODE, FIX>, (unsigned)tiles, HC_COL_THREADS, 0, hc::stream_of(ctx), t, pp, mul, mods, ncb, src);
    hc::count_launch(ctx);
    return hc::cuda_check(cudaGetLastError(), "ntt kernel launch");
}

template <int SHAPE, bool FIX>
hc_status launch_mode(hc_context ctx, int mode, const KView& t, const PlanPtrs& pp, const KView& mul, const KMods& mods, int64_t tiles, int ncb,
                      const KView& src) {
    if (mode == 0) return launch<SHAPE, 0, FIX>(ctx, t, pp, mul, mods, tiles, ncb, src);
    if (mode == 1) return launch<SHAPE, 1, FIX>(ctx, t, pp, mul, mods, tiles, ncb, src);
    if (mode == 2) return launch<SHAPE, 2, FIX>(ctx, t, pp, mul, mods, tiles, ncb, src);
    if (FIX && mode == 6) return launch<SHAPE, 6, true>(ctx, t, pp, mul, mods, tiles, ncb, src);
    return launch<SHAPE, 3, FIX>(ctx, t, pp, mul, mods, tiles, ncb, src);
}

}  // namespace

namespace hc {

hc_status launch_ntt_col(hc_context ctx, int shape, int mode, bool fix, const KView& t, const PlanPtrs& pp, const KView& mul, const KMods& mods, int64_t tiles, int ncb,
                      const KView& src) {
    if (shape == HC_SHAPE_C12)
        return fix ? launch_mode<HC_SHAPE_C12, true>(ctx, mode, t, pp, mul, mods, tiles, ncb, src)
                   : launch_mode<HC_SHAPE_C12, false>(ctx, mode, t, pp, mul, mods, tiles, ncb, src);
    return fix ? launch_mode<HC_SHAPE_C4, true>(ctx, mode, t, pp, mul, mods, tiles, ncb, src)
               : launch_mode<HC_SHAPE_C4, false>(ctx, mode, t, pp, mul, mods, tiles, ncb, src);
}

}  // namespace hc
