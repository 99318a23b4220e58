// The persistent kernel with TF32 GEMM tiles on tcgen05.
#include "engine_kernel.cuh"

namespace chb {

template cudaError_t build_launch<EB_TCGEN05>(const RunArgs&, int, size_t, cudaStream_t);
template cudaError_t build_set_smem<EB_TCGEN05>(size_t);
template cudaError_t build_occupancy<EB_TCGEN05>(int*, size_t);

}  // namespace chb
