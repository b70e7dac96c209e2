// Forward kernels of the quadratic spline, ReLU^2 base path.
#include "skv_tc_fwd_kernel.cuh"

namespace skv {
namespace tc {
cudaError_t fwd_launch_quad_relu(int groups, int fold, const FwdParams& P, dim3 grid, size_t smem, cudaStream_t stream) {
  return fwd_launch<SKV_ACT_RELU_SQ, false, false>(groups, fold, P, grid, smem, stream);
}
}  // namespace tc
}  // namespace skv
