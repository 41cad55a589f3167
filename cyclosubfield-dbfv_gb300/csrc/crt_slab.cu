// CRT transforms of field_49152 (slabs of 4 rows of 12288 residues, dimension 2 = [4], dimension 3 =
// [3, 64, 64]) in four launches with the passes split where the data's coupling splits.
//
// The reference transforms a batch [count, r, deg_L', deg_K] in four HAL calls (src/ring.rs:1118-1161):
// ntt_mul along dimension 2 (times the kernel K_L'), ntt_mul along dimension 3 (times K_K), intt along
// dimension 2, intt along dimension 3. A dimension-3 line is too long for a CTA's share of an SM, and
// its leading radix-3 stage is the only one that couples its three blocks of 4096. So each half runs
// as
//   lead:   a thread takes positions p, p + 4096, p + 8192 of all four rows (12 residues, coalesced along
//           dimension 3) through the four-point columns, the kernel product and the radix-3 stage of
//           each row, all in registers;
//   blocks: a CTA takes one block of 4096 through the twelve radix-2 stages in its shared memory, six
//           CTAs per SM, independent of one another (ntt_fast.cuh, block4096).
// What bounds them: the lead kernel memory, the block kernel the multiply pipe. Butterflies, their order
// and the reduction / skip / fused-final schedule are exactly those of the single-dimension kernels,
// so the results are bit-identical. Holding a slab in the shared memory of a 12-CTA cluster between
// the two kernels saves half the traffic, but its CTAs wait for one another and for twelve free places
// at once: pb_to_crt of [24, 23, 4, 12288] 563 us against 510 us, of [8, 23, 4, 12288] 202 against 186.
#include "common.cuh"
#include "ntt_run.cuh"

namespace hc {
const void* plan_device(hc_ntt_plan p);
int32_t plan_shape(hc_ntt_plan p);
}  // namespace hc

namespace {

constexpr int LEAD_THREADS = 256;
constexpr size_t SMEM4096 = (size_t)BLOCK4096_WORDS * 8;

/// lead: CTAs over (slab, 256 positions). DIR 0: forward, times the dimension-2 kernel m2 [r][4] (limbs),
/// reading src, writing t; DIR 1: inverse, in place (src = t).
template <int DIR>
__global__ void __launch_bounds__(LEAD_THREADS, 4)
    lead12288_kernel(KView t, KView src, PlanPtrs p2, PlanPtrs p3, const BarrettLimbs* m2, KMods mods) {
    grid_wait();
    // tiles last to first (as the column kernel's: what the last launch wrote last is still in L2)
    const int64_t tile = gridDim.x - 1 - blockIdx.x;
    const int64_t slab = tile / (4096 / LEAD_THREADS), j = slab % t.n1, i = slab / t.n1;
    const int p = (int)(tile % (4096 / LEAD_THREADS)) * LEAD_THREADS + threadIdx.x;
    const DevPlanHeader* P3 = p3.p[j];
    const fast::CtxL c2 = make_ctx<fast::CtxL>(p2.p[j]), c3 = make_ctx<fast::CtxL>(P3);
    const int64_t* gs = reinterpret_cast<const int64_t*>(src.p) + i * src.s0 + j * src.s1 + p;
    int64_t* g = reinterpret_cast<int64_t*>(t.p) + i * t.s0 + j * t.s1 + p;
    if (P3->cls == 57) lead12288<DIR, 57>(c2, c3, gs, src.s2, g, t.s2, m2 + 4 * j, mods.n[j]);
    else lead12288<DIR, 56>(c2, c3, gs, src.s2, g, t.s2, m2 + 4 * j, mods.n[j]);
}

/// blocks: CTAs over (line, block). MODE 6: forward, times the dimension-3 kernel m3 [r][12288] (limbs); 1:
/// inverse; 3: inverse, times the tensor pm.
template <int MODE, int THREADS>
__global__ void __launch_bounds__(THREADS, 768 / THREADS)
    block4096_kernel(KView t, PlanPtrs p3, const BarrettLimbs* m3, KView pm, KMods mods) {
    grid_wait();
    extern __shared__ __align__(16) int64_t smem[];
    const int64_t tile = blockIdx.x / 3;
    const int blk = (int)(blockIdx.x % 3);
    const int64_t k = tile % t.n2, r = tile / t.n2;
    const int64_t j = r % t.n1, i = r / t.n1;
    const DevPlanHeader* P = p3.p[j];
    const fast::CtxL c = make_ctx<fast::CtxL>(P);
    int64_t* g = reinterpret_cast<int64_t*>(t.p) + i * t.s0 + j * t.s1 + k * t.s2 + 4096 * blk;
    const int64_t* mulp = nullptr;
    int64_t me = 0;
    if constexpr (MODE == 6) {
        mulp = reinterpret_cast<const int64_t*>(m3 + 12288 * j + 4096 * blk), me = 1;
    } else if constexpr (MODE == 3) {
        me = pm.b3 ? 0 : 1;
        mulp = kat<int64_t>(pm, i, j, k, 0) + me * 4096 * blk;
    }
    with_sched<HC_SHAPE_L12288, (MODE & 1) != 0, true>(P, [&](const auto& sch) {
        int4* tws = reinterpret_cast<int4*>(smem + 4096);
        fast::stage_tail_twiddles<(MODE & 1) != 0>(fast::CtaTeam{}, c, sch, tws, 1, 63, 7);
        fast::block4096<MODE>(fast::CtaTeam{}, sch, c, smem, tws, g, mulp, me, fast::make_mont<fast::CtxL, MODE>(mods.n[j], mods.ninv[j]));
    });
}

template <int MODE, int THREADS>
hc_status launch_blocks_as(hc_context ctx, int64_t ctas, const KView& t, const PlanPtrs& p3, const BarrettLimbs* m3,
                           const KView& pm, const KMods& mods) {
    hc::launch_kernel(block4096_kernel<MODE, THREADS>, (unsigned)ctas, THREADS, SMEM4096, hc::stream_of(ctx), t, p3, m3, pm, mods);
    hc::count_launch(ctx);
    return hc::cuda_check(cudaGetLastError(), "CRT block pass launch");
}
/// 128 threads per block, or 256 for calls whose blocks all fit the device at once that way (three per
/// SM), where a block's own latency is the launch's.
template <int MODE>
hc_status launch_blocks(hc_context ctx, const KView& t, const PlanPtrs& p3, const BarrettLimbs* m3, const KView& pm,
                        const KMods& mods) {
    const int64_t ctas = t.n0 * t.n1 * t.n2 * 3;
    if (ctas <= 3 * (int64_t)hc::num_sms(ctx)) return launch_blocks_as<MODE, 256>(ctx, ctas, t, p3, m3, pm, mods);
    return launch_blocks_as<MODE, 128>(ctx, ctas, t, p3, m3, pm, mods);
}

/// Whether a transform's plans are field_49152's shapes ([4] along dimension 2, [3, 64, 64] along
/// dimension 3), fixed, and t has their extents. (field_36864's [2, 3, 8, 64] lines fit a CTA, and its
/// [4, 3] columns already hold 12 residues of one position.)
bool slab_shape(const hc_ntt_plan* plans2, const hc_ntt_plan* plans3, size_t r, const KView& t) {
    if (r == 0 || r > HC_MAX_MODS || (int64_t)r != t.n1) return false;
    const int s2 = hc::plan_shape(plans2[0]), s3 = hc::plan_shape(plans3[0]);
    if (s2 != (HC_SHAPE_C4 | 0x100) || s3 != (HC_SHAPE_L12288 | 0x100) || t.n2 != 4 || t.n3 != 12288) return false;
    for (size_t j = 1; j < r; j++)
        if (hc::plan_shape(plans2[j]) != s2 || hc::plan_shape(plans3[j]) != s3) return false;
    return t.n0 * t.n1 * (4096 / LEAD_THREADS) <= 0x7fffffff;
}

}  // namespace

namespace hc {

/// Whether the slab passes can run this transform (slab_shape).
bool crt_pass_ready(hc_context ctx, const hc_ntt_plan* plans2, const hc_ntt_plan* plans3, size_t r, const KView& t) {
    (void)ctx;
    return slab_shape(plans2, plans3, r, t);
}

/// One half of a CRT transform over t [count, r, deg_L', deg_K] (dimension 3 contiguous):
/// dir 0 = ntt_mul along dimension 2 by the kernels m2 [r][4], then along dimension 3 by m3 [r][12288],
/// both as limbs (mont_const_limbs), reading the input from src when given (the caller's copy folded
/// into the lead kernel; src must not overlap t other than exactly); dir 1 = intt along dimension 2,
/// then along dimension 3, times the tensor pm when `post`.
/// The caller checks crt_pass_ready first.
hc_status launch_crt_pass(hc_context ctx, int dir, const KView& t, const KView* src, const hc_ntt_plan* plans2,
                          const hc_ntt_plan* plans3, size_t r, const BarrettLimbs* m2, const BarrettLimbs* m3,
                          const KView& pm, bool post, const KMods& mods) {
    if (!slab_shape(plans2, plans3, r, t)) return fail(HC_ERR_UNSUPPORTED, "CRT slab pass: plans are not its shapes");
    PlanPtrs p2, p3;
    for (size_t j = 0; j < r; j++) {
        p2.p[j] = reinterpret_cast<const DevPlanHeader*>(plan_device(plans2[j]));
        p3.p[j] = reinterpret_cast<const DevPlanHeader*>(plan_device(plans3[j]));
    }
    const int64_t slabs = t.n0 * t.n1;
    if (slabs == 0) return HC_OK;
    const unsigned grid = (unsigned)(slabs * (4096 / LEAD_THREADS));
    if (dir == 0) hc::launch_kernel(lead12288_kernel<0>, grid, LEAD_THREADS, 0, stream_of(ctx), t, src ? *src : t, p2, p3, m2, mods);
    else hc::launch_kernel(lead12288_kernel<1>, grid, LEAD_THREADS, 0, stream_of(ctx), t, t, p2, p3, nullptr, mods);
    count_launch(ctx);
    hc_status st = cuda_check(cudaGetLastError(), "CRT lead pass launch");
    if (st) return st;
    if (dir == 0) return launch_blocks<6>(ctx, t, p3, m3, pm, mods);
    return post ? launch_blocks<3>(ctx, t, p3, nullptr, pm, mods) : launch_blocks<1>(ctx, t, p3, nullptr, pm, mods);
}

}  // namespace hc
