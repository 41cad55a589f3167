// Whole CRT transforms of small rings (field_2 .. field_192): slabs of deg_L' x deg_K residues that fit a CTA's
// shared memory, one CTA per (element, factor) slab and one launch per transform.
//
// What bounds them: latency. A slab is 2 to 192 residues, so each of the reference's four HAL calls
// (src/ring.rs:1118-1161) is one short launch that fetches its stage programme, its twiddles and its
// line one after the other; here all of it is fetched together once and the four passes run on shared
// memory. The passes are the generic tile programme's (ntt_tile.cuh), in the calls' order.
// One element of field_18 over four factors: 53 us for two transforms and a product in nine launches, 25 us
// in three; 100 elements of field_192 over eight 83 us against 42 us.
#include <algorithm>

#include "ntt_tile.cuh"

namespace hc {
const void* plan_device(hc_ntt_plan p);
int32_t plan_len(hc_ntt_plan p);
int32_t plan_shape(hc_ntt_plan p);
int32_t plan_ntw(hc_ntt_plan p);
void plan_counts(hc_ntt_plan p, int32_t counts[4]);
}  // namespace hc

namespace {

/// What a plan's programme takes in shared memory; the same for every row of a call.
struct SmallPlan {
    int nfwd, ninv, nfpass, nipass;
    int ntw;   // the largest of the rows' twiddle pairs
    int words;  // of the staged programme and twiddles
};
struct SmallArgs {
    KView t, src;
    KView post;  // a factor of the result (p null: none)
    PlanPtrs p2, p3;
    SmallPlan s2, s3;
    const int64_t* kl;  // kernels [r][deg_L'] and [r][deg_K]
    const int64_t* kk;
    FastDiv div_dl, div_dk;
};

/// Starts copying n bytes (a multiple of 8) to shared memory, over the CTA's threads.
__device__ __forceinline__ void stage(int64_t* dst, const void* src, int bytes) {
    const int64_t* g = reinterpret_cast<const int64_t*>(src);
    for (int i = threadIdx.x; i < bytes / 8; i += blockDim.x) dst[i] = g[i];
}
/// Stages plan P's programme at `at`; the copies are complete after the next block barrier.
__device__ __forceinline__ Program stage_program(const DevPlanHeader* P, const SmallPlan& q, int64_t* at) {
    Program r = program_of(P, nullptr);
    auto take = [&](const void* src, int bytes) {
        int64_t* p = at;
        stage(p, src, bytes);
        at += bytes / 8;
        return p;
    };
    r.tw = take(P + 1, q.ntw * 16);
    r.fwd = reinterpret_cast<DevStage*>(take(P->fwd, q.nfwd * (int)sizeof(DevStage)));
    r.inv = reinterpret_cast<DevStage*>(take(P->inv, q.ninv * (int)sizeof(DevStage)));
    r.fpass = reinterpret_cast<DevPass*>(take(P->fpass, q.nfpass * (int)sizeof(DevPass)));
    r.ipass = reinterpret_cast<DevPass*>(take(P->ipass, q.nipass * (int)sizeof(DevPass)));
    return r;
}
static_assert(sizeof(DevStage) % 8 == 0 && sizeof(DevPass) % 8 == 0, "staged in 8-byte words");

__global__ void __launch_bounds__(256) crt_small_kernel(SmallArgs a, KMods mods) {
    grid_wait();
    extern __shared__ __align__(16) int64_t smem[];
    const int dl = (int)a.t.n2, dk = (int)a.t.n3, total = dl * dk;
    const int64_t j = blockIdx.x % a.t.n1, i = blockIdx.x / a.t.n1;
    int64_t* s = smem;
    const int64_t* gs = reinterpret_cast<const int64_t*>(a.src.p) + i * a.src.s0 + j * a.src.s1;
    int64_t* g = reinterpret_cast<int64_t*>(a.t.p) + i * a.t.s0 + j * a.t.s1;
    for (int b = threadIdx.x; b < total; b += blockDim.x) {
        const int k = (int)fdiv((uint32_t)b, a.div_dk), l = b - k * dk;
        s[b] = gs[k * a.src.s2 + l];
    }
    int64_t* kl = s + total;
    int64_t* kk = kl + dl;
    stage(kl, a.kl + j * dl, dl * 8);
    stage(kk, a.kk + j * dk, dk * 8);
    const Program P2 = stage_program(a.p2.p[j], a.s2, kk + dk);
    const Program P3 = stage_program(a.p3.p[j], a.s3, kk + dk + a.s2.words);
    const int64_t n = mods.n[j], ninv = mods.ninv[j];
    const SlabTile T2{s, dl, dk, dk, 1, a.div_dk}, T3{s, dk, dl, 1, dk, a.div_dl};
    __syncthreads();
    run_passes(T2, P2, 2);
    for (int b = threadIdx.x; b < total; b += blockDim.x) s[b] = mul_mont(s[b], kl[fdiv((uint32_t)b, a.div_dk)], n, ninv);
    __syncthreads();
    run_passes(T3, P3, 2);
    for (int b = threadIdx.x; b < total; b += blockDim.x) {
        const int k = (int)fdiv((uint32_t)b, a.div_dk);
        s[b] = mul_mont(s[b], kk[b - k * dk], n, ninv);
    }
    __syncthreads();
    run_passes(T2, P2, 1);
    run_passes(T3, P3, 1);
    for (int b = threadIdx.x; b < total; b += blockDim.x) {
        const int k = (int)fdiv((uint32_t)b, a.div_dk), l = b - k * dk;
        int64_t v = s[b];
        if (a.post.p) v = mul_mont(v, *kat<int64_t>(a.post, i, j, k, l), n, ninv);
        g[k * a.t.s2 + l] = v;
    }
}

/// The rows' plans as one SmallPlan, or false if they differ in more than their constants.
bool small_plan(const hc_ntt_plan* plans, size_t r, int64_t len, SmallPlan* out, PlanPtrs* ptrs) {
    int32_t c0[4], c[4];
    *out = SmallPlan{};
    for (size_t j = 0; j < r; j++) {
        if (hc::plan_len(plans[j]) != len) return false;
        hc::plan_counts(plans[j], c);
        if (j == 0) std::copy(c, c + 4, c0);
        if (!std::equal(c, c + 4, c0)) return false;
        out->ntw = std::max(out->ntw, (int)hc::plan_ntw(plans[j]));
        if (hc::plan_ntw(plans[j]) != hc::plan_ntw(plans[0])) return false;
        ptrs->p[j] = reinterpret_cast<const DevPlanHeader*>(hc::plan_device(plans[j]));
    }
    out->nfwd = c0[0], out->ninv = c0[1], out->nfpass = c0[2], out->nipass = c0[3];
    out->words = 2 * out->ntw + (int)((out->nfwd + out->ninv) * sizeof(DevStage) + (out->nfpass + out->nipass) * sizeof(DevPass)) / 8;
    return true;
}

}  // namespace

namespace hc {

/// Runs a transform of t [count, r, deg_L', deg_K] (dimension 3 contiguous) in one launch, if its slabs and
/// programmes fit 48 KB of shared memory (*done tells): ntt_mul along dimension 2 by kl [r][deg_L'] and along
/// dimension 3 by kk [r][deg_K], intt along both, times `post` when given. src: read instead of t (equal to t
/// or not overlapping it).
hc_status launch_crt_small(hc_context ctx, const KView& t, const KView* src, const hc_ntt_plan* plans2,
                           const hc_ntt_plan* plans3, size_t r, const int64_t* kl, const int64_t* kk, const KView* post,
                           const KMods& mods, bool* done) {
    *done = false;
    if (r == 0 || r > HC_MAX_MODS || (int64_t)r != t.n1 || t.n2 < 1 || t.n3 < 1 || t.n2 * t.n3 > 4096) return HC_OK;
    SmallArgs a;
    if (!small_plan(plans2, r, t.n2, &a.s2, &a.p2) || !small_plan(plans3, r, t.n3, &a.s3, &a.p3)) return HC_OK;
    const int64_t total = t.n2 * t.n3, slabs = t.n0 * t.n1;
    const size_t smem = (size_t)(total + t.n2 + t.n3 + a.s2.words + a.s3.words) * 8;
    if (smem > 49152 || slabs > 0x7fffffff) return HC_OK;
    *done = true;
    if (slabs == 0) return HC_OK;
    a.t = t, a.src = src ? *src : t;
    a.post = post ? *post : KView();
    a.kl = kl, a.kk = kk;
    a.div_dl = make_fastdiv((uint32_t)t.n2), a.div_dk = make_fastdiv((uint32_t)t.n3);
    // a butterfly or two per thread; at least two warps, for the staging
    const int threads = (int)std::min<int64_t>(256, std::max<int64_t>(64, (total / 4 + 31) / 32 * 32));
    hc::launch_kernel(crt_small_kernel, (unsigned)slabs, threads, smem, stream_of(ctx), a, mods);
    count_launch(ctx);
    return cuda_check(cudaGetLastError(), "small CRT transform launch");
}

}  // namespace hc
