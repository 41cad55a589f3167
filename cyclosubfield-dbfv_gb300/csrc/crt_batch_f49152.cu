// The batched-transform kernel for field_49152's slabs.
#include "crt_batch.cuh"

namespace hc {

CrtBatchKernel crt_batch_f49152(int ctas_per_sm) { return crt_batch_variant<2>(ctas_per_sm); }

}  // namespace hc
