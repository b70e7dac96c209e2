// Forward kernels of the quadratic spline with split operands, other base paths.
#include "skv_tc_fwd_kernel.cuh"

namespace skv {
namespace tc {
cudaError_t fwd_launch_split_other(int groups, int fold, const FwdParams& P, dim3 grid, size_t smem, cudaStream_t stream) {
  return fwd_launch<-1, false, true>(groups, fold, P, grid, smem, stream);
}
}  // namespace tc
}  // namespace skv
