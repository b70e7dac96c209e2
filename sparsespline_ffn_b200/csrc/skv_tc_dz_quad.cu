// dz kernels of the quadratic spline.
#include "skv_tc_dz_kernel.cuh"

namespace skv {
namespace tc {
cudaError_t dz_launch_quad(const DzPlan& zp, int L, bool relu, const DzParams& P, dim3 grid, cudaStream_t stream) {
  return dz_launch<false, false>(zp, L, relu, P, grid, stream);
}
}  // namespace tc
}  // namespace skv
