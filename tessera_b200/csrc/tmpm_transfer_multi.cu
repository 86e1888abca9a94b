// tmpm_transfer_multi.cu -- transfer kernels: multi-scene batches.
#include "tmpm_transfer.cuh"

namespace tmpm {
TMPM_TRANSFER_VARIANT(kMulti)
TMPM_SEGMENT_VARIANT(kMulti)
template void preload_transfer_variant<kMulti>();
}  // namespace tmpm
