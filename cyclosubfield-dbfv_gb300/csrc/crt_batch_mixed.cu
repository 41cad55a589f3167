// The batched-transform kernel for both large fields' slabs in one launch.
#include "crt_batch.cuh"

namespace hc {

CrtBatchKernel crt_batch_mixed(int ctas_per_sm) { return crt_batch_variant<0>(ctas_per_sm); }

}  // namespace hc
