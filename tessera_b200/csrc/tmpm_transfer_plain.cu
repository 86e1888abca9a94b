// tmpm_transfer_plain.cu -- transfer kernels: one scene without obstacles.
#include "tmpm_transfer.cuh"

namespace tmpm {
TMPM_TRANSFER_VARIANT(kPlain)
TMPM_SEGMENT_VARIANT(kPlain)
template void preload_transfer_variant<kPlain>();
}  // namespace tmpm
