// The persistent kernel with the Householder panels of the factored updates.
#include "engine_kernel.cuh"

namespace chb {

template cudaError_t build_launch<EB_PANELS>(const RunArgs&, int, size_t, cudaStream_t);
template cudaError_t build_set_smem<EB_PANELS>(size_t);

}  // namespace chb
