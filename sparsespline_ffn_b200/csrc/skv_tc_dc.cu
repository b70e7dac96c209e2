// dC kernels: keys per lane and warps per producer group.
#include "skv_tc_dc_kernel.cuh"

namespace skv {
namespace tc {

namespace {
template <int KJ, int GW, bool RUNS>
cudaError_t dc_launch_case(const DcPlan& dp, bool lin, bool split, const DcParams& P, dim3 grid, cudaStream_t stream) {
  const unsigned threads = (unsigned)(dp.ngroups * dp.gw + kDcIssuers + 1) * 32;
  return lin     ? launch_chained<tc_dc_kernel<KJ, GW, true, true, RUNS>>(grid, threads, dp.smem, stream, P)
         : split ? launch_chained<tc_dc_kernel<KJ, GW, false, true, RUNS>>(grid, threads, dp.smem, stream, P)
                 : launch_chained<tc_dc_kernel<KJ, GW, false, false, RUNS>>(grid, threads, dp.smem, stream, P);
}
}  // namespace

cudaError_t dc_launch(const DcPlan& dp, bool lin, bool split, const DcParams& P, dim3 grid, cudaStream_t stream) {
  const bool segments = dp.runs || dp.run > dp.chain;
#define SKV_DC_CASE(KJ_, GW_)                                                                   \
  if (dp.kj == KJ_ && dp.gw == GW_)                                                             \
    return segments ? dc_launch_case<KJ_, GW_, true>(dp, lin, split, P, grid, stream)           \
                    : dc_launch_case<KJ_, GW_, false>(dp, lin, split, P, grid, stream);
  SKV_DC_CASE(4, 4) SKV_DC_CASE(4, 8) SKV_DC_CASE(2, 4) SKV_DC_CASE(2, 8)
#undef SKV_DC_CASE
  return cudaErrorInvalidValue;
}

}  // namespace tc
}  // namespace skv
