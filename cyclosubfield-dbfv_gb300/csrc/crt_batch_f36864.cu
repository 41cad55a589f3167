// The batched-transform kernel for field_36864's slabs.
#include "crt_batch.cuh"

namespace hc {

CrtBatchKernel crt_batch_f36864(int ctas_per_sm) { return crt_batch_variant<1>(ctas_per_sm); }

}  // namespace hc
