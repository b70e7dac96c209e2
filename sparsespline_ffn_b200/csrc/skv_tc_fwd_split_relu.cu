// Forward kernels of the quadratic spline with split operands, ReLU^2 base path.
#include "skv_tc_fwd_kernel.cuh"

namespace skv {
namespace tc {
cudaError_t fwd_launch_split_relu(int groups, int fold, const FwdParams& P, dim3 grid, size_t smem, cudaStream_t stream) {
  return fwd_launch<SKV_ACT_RELU_SQ, false, true>(groups, fold, P, grid, smem, stream);
}
}  // namespace tc
}  // namespace skv
