// dC kernels: keys per chunk and, for L = 21 / 22, words per key known at compile time.
#include "skv_tc_dc_kernel.cuh"

namespace skv {
namespace tc {

cudaError_t dc_launch(const DcPlan& dp, bool lin, const DcParams& P, dim3 grid, cudaStream_t stream) {
#define SKV_DC_CASE(KCH_, HLC_)                                                                      \
  return lin ? launch_chained<tc_dc_kernel<KCH_, HLC_, true>>(grid, 320, dp.smem, stream, P)         \
             : launch_chained<tc_dc_kernel<KCH_, HLC_, false>>(grid, 320, dp.smem, stream, P);
  if (dp.kch == 16 && P.LR == 22) SKV_DC_CASE(16, 11)
  if (dp.kch == 16) SKV_DC_CASE(16, 0)
  SKV_DC_CASE(8, 0)
#undef SKV_DC_CASE
}

}  // namespace tc
}  // namespace skv
