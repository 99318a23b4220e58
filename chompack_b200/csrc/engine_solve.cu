// The persistent kernel with the tasks of the triangular solves and products.
#include "engine_kernel.cuh"

namespace chb {

template cudaError_t build_launch<EB_SOLVE>(const RunArgs&, int, size_t, cudaStream_t);
template cudaError_t build_set_smem<EB_SOLVE>(size_t);

}  // namespace chb
