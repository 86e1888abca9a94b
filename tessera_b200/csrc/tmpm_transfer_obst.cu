// tmpm_transfer_obst.cu -- transfer kernels: one scene with rigid obstacles, or plastic state.
#include "tmpm_transfer.cuh"

namespace tmpm {
TMPM_TRANSFER_VARIANT(kPlainObst)
TMPM_SEGMENT_VARIANT(kPlainObst)
template void preload_transfer_variant<kPlainObst>();
}  // namespace tmpm
