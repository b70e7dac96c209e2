// Token-major rows ([N][h] bf16) through shared memory by tiled TMA.
//
// The contraction kernels have one thread per token, each of which wants 16 bytes (eight keys) of its own row
// at a time.  Read straight from global memory such a warp-wide access touches 32 lines, and the load/store
// unit takes it apart line by line, in front of everything else that is queued there.  A box of 128 tokens x 32
// keys moves as one TMA copy instead; with the 64-byte swizzle the 16-byte pieces of eight neighbouring rows
// lie in different banks, so a warp reads or writes its pieces at full width.
#pragma once

#include <cuda.h>
#include <cudaTypedefs.h>

#include "skv_tc_common.cuh"

namespace skv {
namespace tc {

constexpr int kBoxKeys = 32, kBoxRows = 128;
constexpr uint32_t kBoxBytes = kBoxRows * kBoxKeys * 2;

// Byte offset of 16-byte piece c (0..3) of a row in a box; the box starts on a 512-byte boundary.
__device__ __forceinline__ uint32_t box_piece(uint32_t row, uint32_t c) { return row * 64u + ((c ^ ((row >> 1) & 3u)) << 4); }

// One box of `map` at element coordinates (x, y) into this CTA's shared memory; x is a multiple of 8.
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}
// The reverse; elements past the array's bounds are not written.
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, const void* src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(x), "r"(y), "r"(smem_u32(src))
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// Until at most `Pending` of this thread's committed stores still read shared memory.
template <int Pending> __device__ __forceinline__ void bulk_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(Pending) : "memory");
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void lds64(uint32_t addr, uint32_t (&v)[2]) {
  asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(v[0]), "=r"(v[1]) : "r"(addr) : "memory");
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void sts64(uint32_t addr, uint32_t a, uint32_t b) {
  asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ void sts128(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// Map of a [rows][cols] bf16 matrix with row pitch `pitch` elements, zeros outside the matrix.
bool make_map_2d(CUtensorMap* m, const void* base, uint64_t rows, uint64_t cols, uint64_t pitch, uint32_t box_cols,
                 uint32_t box_rows, CUtensorMapSwizzle swizzle);
// The maps of this file's boxes.
inline bool make_box_map(CUtensorMap* m, const void* base, int64_t N, int h, int64_t pitch) {
  return make_map_2d(m, base, (uint64_t)N, (uint64_t)h, (uint64_t)pitch, kBoxKeys, kBoxRows, CU_TENSOR_MAP_SWIZZLE_64B);
}

}  // namespace tc
}  // namespace skv
