// Launch of the persistent kernel, and its build for the FP64 sweeps without
// Householder panels and solve tasks.
#include "engine_kernel.cuh"

namespace chb {

template cudaError_t build_launch<EB_BASE>(const RunArgs&, int, size_t, cudaStream_t);

#ifdef CHB_PROFILE_POTRF
// Development builds only: copies out (and optionally clears) the diagonal
// task's phase counters.
extern "C" int chb_dev_potrf_phase(unsigned long long* out, int clear) {
  cudaError_t e = cudaMemcpyFromSymbol(out, g_potrf_phase, sizeof(g_potrf_phase));
  if (e == cudaSuccess && clear) {
    static const unsigned long long zero[32] = {};
    e = cudaMemcpyToSymbol(g_potrf_phase, zero, sizeof(zero));
  }
  return (int)e;
}
#endif

// The other builds (engine_tc.cu, engine_ql.cu, engine_solve.cu).
extern template cudaError_t build_launch<EB_TCGEN05>(const RunArgs&, int, size_t, cudaStream_t);
extern template cudaError_t build_set_smem<EB_TCGEN05>(size_t);
extern template cudaError_t build_occupancy<EB_TCGEN05>(int*, size_t);
extern template cudaError_t build_launch<EB_PANELS>(const RunArgs&, int, size_t, cudaStream_t);
extern template cudaError_t build_set_smem<EB_PANELS>(size_t);
extern template cudaError_t build_launch<EB_SOLVE>(const RunArgs&, int, size_t, cudaStream_t);
extern template cudaError_t build_set_smem<EB_SOLVE>(size_t);

size_t engine_smem_bytes() { return (size_t)ENGINE_SMEM_DOUBLES * sizeof(double); }

// The dynamic shared-memory attribute must have been raised on the current
// device by engine_occupancy() (done when a plan is created).  The launch
// uses ra.smem_doubles (at least the GEMM/POTRF staging).
cudaError_t engine_launch(const RunArgs& ra, int grid, cudaStream_t stream) {
  if (ra.smem_doubles < ENGINE_SMEM_BASE_DOUBLES || ra.smem_doubles > ENGINE_SMEM_DOUBLES) return cudaErrorInvalidValue;
  // the tcgen05 build is sized (engine_occupancy) for the base staging only
  if (ra.panels && ra.solve) return cudaErrorInvalidValue;
  if (ra.tmem && (ra.panels || ra.solve || ra.smem_doubles != ENGINE_SMEM_BASE_DOUBLES)) return cudaErrorInvalidValue;
  const size_t smem = (size_t)ra.smem_doubles * sizeof(double);
  if (ra.tmem) return build_launch<EB_TCGEN05>(ra, grid, smem, stream);
  if (ra.panels) return build_launch<EB_PANELS>(ra, grid, smem, stream);
  if (ra.solve) return build_launch<EB_SOLVE>(ra, grid, smem, stream);
  return build_launch<EB_BASE>(ra, grid, smem, stream);
}

// Resident CTAs per SM of the FP64 build (tc: of the tcgen05 one).  The
// dynamic shared-memory attribute is raised on all builds.  The FP64 builds
// are sized for the largest staging (Householder panels, solve steps); the
// tcgen05 build only runs the TF32 sweeps, which launch with the base
// staging, and is queried at that size (the query still reports one CTA per
// SM for it; the plan launches it as wide as the FP64 build, see
// upload_plan).
int engine_occupancy(int* blocks_per_sm, bool tc) {
  const size_t smem = engine_smem_bytes(), smem_tc = (size_t)ENGINE_SMEM_BASE_DOUBLES * sizeof(double);
  cudaError_t e = build_set_smem<EB_BASE>(smem);
  if (e == cudaSuccess) e = build_set_smem<EB_TCGEN05>(smem);
  if (e == cudaSuccess) e = build_set_smem<EB_PANELS>(smem);
  if (e == cudaSuccess) e = build_set_smem<EB_SOLVE>(smem);
  if (e == cudaSuccess)
    e = tc ? build_occupancy<EB_TCGEN05>(blocks_per_sm, smem_tc) : build_occupancy<EB_BASE>(blocks_per_sm, smem);
  return e == cudaSuccess ? 0 : -1;
}

}  // namespace chb
