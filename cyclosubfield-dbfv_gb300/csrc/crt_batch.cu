// Launches of the batched-transform kernel, and its form for slabs of any shape.
#include <algorithm>

#include "crt_batch.cuh"

namespace hc {

bool crt_slab_limbs(int32_t shapes, int dim);

CrtBatchKernel crt_batch_f36864(int ctas_per_sm);
CrtBatchKernel crt_batch_f49152(int ctas_per_sm);
CrtBatchKernel crt_batch_mixed(int ctas_per_sm);

/// Shared-memory words a slab of the batched transform needs: two 3072-residue lines (one per team of
/// 128 threads), one 4096-residue block of a 12288-residue line, or the generic tile (the whole
/// line, or deg_L' x 2^logv dimension-2 columns); the specialised column passes use none.
size_t crt_slab_tile_words(int32_t shapes, int32_t dl, int32_t dk, int logv) {
    if (crt_slab_12288(shapes)) return BLOCK4096_WORDS;
    const size_t w3 = crt_slab_limbs(shapes, 3) ? 2 * (size_t)LINE3072_WORDS : (size_t)dk;
    const size_t w2 = crt_slab_limbs(shapes, 2) ? 0 : ((size_t)dl << logv);
    const size_t w = std::max(w3, w2);
    return (w + 1) & ~(size_t)1;
}

/// Whether the passes along `dim` run on the specialised code, with the CRT kernels as limbs:
/// field_36864's columns and lines each on their own, field_49152's together.
bool crt_slab_limbs(int32_t shapes, int dim) {
    if (crt_slab_12288(shapes)) return true;
    return dim == 3 ? ((shapes >> 16) & 1) && (shapes & 0xff) == HC_SHAPE_L3072
                    : ((shapes >> 17) & 1) && ((shapes >> 8) & 0xff) == HC_SHAPE_C12;
}

/// Whether a slab runs entirely on the specialised line and column code (crt_batch_kernel<false>).
bool crt_slab_specialised(int32_t shapes) { return crt_slab_limbs(shapes, 3) && crt_slab_limbs(shapes, 2); }

/// Shape class of specialised slab shapes (crt_batch_kernel's CLS): 1 field_36864, 2 field_49152
/// (CLS 0: a launch over both).
int crt_slab_kernel_class(int32_t shapes) { return (shapes & 0xff) == HC_SHAPE_L3072 ? 1 : 2; }

/// Launches the persistent batched-transform kernel over `nslabs` device slab descriptors.
/// `tile_words`: largest tile (deg_K, or deg_L' x 2^logv); `tw_words`: largest pair of twiddle
/// tables (dimension-2 + dimension-3 plan) of a slab. `counter` is reset on the stream first.
hc_status launch_crt_batch(hc_context ctx, cudaStream_t stream, const CrtSlab* slabs, int nslabs, int* counter, size_t tile_words,
                           size_t tw_words, const CrtLaunch& L, bool generic, int cls) {
    if (nslabs <= 0) return HC_OK;
    CrtBatchKernel kern = generic    ? (cls == 3 ? crt_batch_kernel<true, 3, 256, 2> : crt_batch_kernel<true, 0, 256, 2>)
                          : cls == 1 ? crt_batch_f36864(L.ctas_per_sm)
                          : cls == 2 ? crt_batch_f49152(L.ctas_per_sm)
                                     : crt_batch_mixed(L.ctas_per_sm);
    if (L.threads < 32 || L.threads > 256 || L.threads % 32) return fail(HC_ERR_ARG, "batched transform: threads per CTA");
    if (L.logv < 0 || L.logv > 6) return fail(HC_ERR_ARG, "batched transform: dimension-2 tile width");
    const size_t smem = (tile_words + (generic ? tw_words : 0)) * 8;
    if (smem > max_smem_optin(ctx)) return fail(HC_ERR_UNSUPPORTED, "batched transform: slab tiles exceed shared memory");
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return cuda_check(e, "batched transform smem attribute");
    int occ = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, L.threads, smem);
    if (e != cudaSuccess) return cuda_check(e, "batched transform occupancy");
    if (occ < 1) return fail(HC_ERR_UNSUPPORTED, "batched transform: launch shape does not fit an SM");
    int per = L.ctas_per_sm < 1 ? 1 : (L.ctas_per_sm < occ ? L.ctas_per_sm : occ);
    int64_t grid = (int64_t)num_sms(ctx) * per;
    if (grid > nslabs) grid = nslabs;
    hc_status st = cuda_check(cudaMemsetAsync(counter, 0, sizeof(int), stream), "batched transform counter");
    if (st) return st;
    hc::launch_kernel(kern, (unsigned)grid, (unsigned)L.threads, smem, stream, slabs, nslabs, counter, L.logv, (int)tile_words);
    count_launch(ctx);
    return cuda_check(cudaGetLastError(), "batched transform launch");
}

}  // namespace hc
