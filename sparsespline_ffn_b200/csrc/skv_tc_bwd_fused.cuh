// Plan and launch of the opt-in one-kernel backward (skv_tc_bwd_fused.cu).
#pragma once

#include "skv_tc_dz_kernel.cuh"

namespace skv {
namespace tc {

struct FusedPlan { int lb, mtiles, slabs, splits; int64_t tiles_total, tiles_per_split; size_t smem; };
bool plan_fused(const skv_problem& p, FusedPlan* o);
// The dz arguments are those of the dz kernel; `part` receives the [splits][h*L][r] partials of dC.
cudaError_t fused_launch(const FusedPlan& fp, int L, const DzParams& Z, float* part, cudaStream_t stream);

}  // namespace tc
}  // namespace skv
