// dz kernels of the quadratic spline with a split table.
#include "skv_tc_dz_kernel.cuh"

namespace skv {
namespace tc {
cudaError_t dz_launch_split(const DzPlan& zp, int L, bool relu, const DzParams& P, dim3 grid, cudaStream_t stream) {
  return dz_launch<false, true>(zp, L, relu, P, grid, stream);
}
}  // namespace tc
}  // namespace skv
