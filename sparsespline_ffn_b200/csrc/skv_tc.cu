// Entry points of the tcgen05 kernel family as seen by the C ABI.
#include "skv_tc_prep.cuh"
#include "skv_tma.cuh"

namespace skv {
namespace tc {
bool fwd_eligible(const skv_problem& p);
bool bwd_eligible(const skv_problem& p);
size_t fwd_scratch_bytes(const skv_problem& p, bool rows_ok);
size_t bwd_scratch_bytes(const skv_problem& p, bool rows_ok);
int forward(const LaunchCtx& c, const void* z, int64_t zs, const void* C, void* act_out, int64_t as,
            void* delta_out, int64_t ds, void* scratch, bool rows_ok);
int backward(const LaunchCtx& c, const void* z, int64_t zs, const void* C, const void* g_act, int64_t gas,
             const void* g_delta, int64_t gds, void* dz, int64_t dzs, float* dC, void* dC_cast, void* scratch,
             bool rows_ok);

bool make_map_2d(CUtensorMap* m, const void* base, uint64_t rows, uint64_t cols, uint64_t pitch, uint32_t box_cols,
                 uint32_t box_rows, CUtensorMapSwizzle swizzle) {
  static const PFN_cuTensorMapEncodeTiled encode = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      p = nullptr;
    }
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled>(p);
  }();
  if (!encode) return false;
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {pitch * 2};
  const cuuint32_t box[2] = {box_cols, box_rows};
  const cuuint32_t es[2] = {1, 1};
  return encode(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, es,
                CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
}  // namespace tc

// A forward on these kernels is for a backward on them, but only the backward's count of tokens is limited: dz addresses the
// rows of a token tile by a 32-bit TMA coordinate (tiles are of 256 tokens at most).
bool tc_eligible(const skv_problem& p, int op) {
  return tc::bwd_eligible(p) && (op == SKV_OP_FORWARD || p.N < (1ll << 31) - 256);
}

// Split operands double the work, and half a tile of tokens or less leaves most of it to padding; the CUDA-core kernels
// are as fast there.
bool tc_worthwhile(const skv_problem& p) { return p.N > 64 || !tc::split_operands(p); }

size_t tc_scratch_bytes(const skv_problem& p, int op, bool rows_ok) {
  return op == SKV_OP_FORWARD ? tc::fwd_scratch_bytes(p, rows_ok) : tc::bwd_scratch_bytes(p, rows_ok);
}

int tc_forward(const LaunchCtx& c, const void* z, int64_t zs, const void* C, void* act_out, int64_t as,
               void* delta_out, int64_t ds, void* scratch, bool rows_ok) {
  return tc::forward(c, z, zs, C, act_out, as, delta_out, ds, scratch, rows_ok);
}

int tc_backward(const LaunchCtx& c, const void* z, int64_t zs, const void* C, const void* g_act, int64_t gas,
                const void* g_delta, int64_t gds, void* dz, int64_t dzs, float* dC, void* dC_cast, void* scratch,
                bool rows_ok) {
  return tc::backward(c, z, zs, C, g_act, gas, g_delta, gds, dz, dzs, dC, dC_cast, scratch, rows_ok);
}

}  // namespace skv
