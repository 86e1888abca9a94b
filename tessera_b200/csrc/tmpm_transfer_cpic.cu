// tmpm_transfer_cpic.cu -- transfer kernels: one scene with CPIC obstacles.
#include "tmpm_transfer.cuh"

namespace tmpm {
TMPM_TRANSFER_VARIANT(kCpic)
}  // namespace tmpm
