// Operand images of one call and the sums of its partial results, as the tensor-core kernels share them.
#pragma once

#include "skv_launch.cuh"
#include "skv_tc_common.cuh"

namespace skv {
namespace tc {

constexpr int kChunkKeys = 8;
constexpr int kPlanSMs = 148;                 // B200; only used to balance launch shapes
constexpr size_t kSmemLimit = 227 * 1024;
// The contraction kernels run one CTA per SM.  A kernel started while its predecessor still occupies the chip
// is placed unevenly, and a second CTA on an SM would only wait there for the first one's tensor memory while
// other SMs idle, so each asks for more than half of the shared memory.  65536 x 5120, r = 32: forward 0.818 ms without,
// 0.801 with; 2495 x 2048, L = 42, one step: 221 against 184 us with the kernels it was introduced for, 119 either way now.
constexpr size_t kSmemOnePerSM = 116 * 1024;

// Header at the start of a call's scratch: the final maxima (kAmaxG, kAmaxC), then the maxima of the blocks
// that scanned C and g_delta.
constexpr size_t kHeaderBytes = 4096;
constexpr int kBlockMax = 64;                 // first word of the block maxima
constexpr int kMaxBlocks = 444;               // scanning blocks per array

// The kernels work on whole chunks of keys and whole K = 16 steps of code channels; the images (and, when the
// rows of z cannot be read in 16-byte pieces, padded copies of the token-major arrays) carry the padding.
inline int padded_h(const skv_problem& p) { return (p.h + kChunkKeys - 1) / kChunkKeys * kChunkKeys; }
inline int padded_r(const skv_problem& p) { return (p.r + 15) / 16 * 16; }

// Operands as pairs of f16 (value and remainder), for results as accurate as float32 arithmetic on the same inputs.
// One f16 per weight is what this family has always given bf16 problems of the plain shapes below; every other problem had
// the CUDA-core kernels' float32 arithmetic and keeps its accuracy: twice the MMAs, still several times faster
// (linear spline, 4096 x 1024, r = 32, a training step).
inline bool split_operands(const skv_problem& p) {
  return p.spline_order == 1 || p.h % kChunkKeys != 0 || p.r % 16 != 0 || p.L > 49;
}

inline size_t align256(size_t x) { return (x + 255) / 256 * 256; }

// One [N][h] bf16 array copied to [N][hp] (pad columns zero); with act_out also phi of it at that pointer.
struct CopyJob {
  const __nv_bfloat16* src;
  int64_t ss;
  __nv_bfloat16* dst;        // null: no job
  __nv_bfloat16* act_out;
  int64_t as;
};

// Infinities and NaN in C and g_delta.  A (token, key) pair touches order + 1 knot rows, but the contractions multiply all rows by
// weights most of which are zero, and zero times an infinity is NaN: one such element of C would reach every token, one
// of g_delta every row of dC.  The problems with split operands are contained: their images hold zeros in such
// places, and where a scan has found any, the last kernels of a call add what the pairs that touch them contribute.
struct Contain {
  const __nv_bfloat16* z;    // null: not contained
  int64_t zs;
  const __nv_bfloat16* C;
  const __nv_bfloat16* g;
  int64_t gds, N;
  int h, L, r;
  GridParams grid;
  void* dz;                  // null: no dz wanted
  int64_t dzs;
  const void* dz_rows;       // padded rows that dz is in; null: it is in its place
  int64_t dz_rows_stride;
  float coef;                // lambda * scale, of dz
  bool dz_f32;
};

struct PrepParams {
  const __nv_bfloat16* C;
  int h, hp, L, r, rp;
  int lpc;                   // rows per key of the code-table image (4 per group of the forward's order), 0: none wanted
  __half* cimg;
  int lpt;                   // rows per key of the transformed-table image, 0: none wanted
  int tparts;                // f16 parts of its values: 1, or 2 (channels [0, rp) and the remainders in [rp, 2 rp))
  __half* timg;
  const __nv_bfloat16* g;    // null: no gradient image
  int64_t gds, N, tiles;     // tiles of 128 tokens in the image
  __half* gimg;
  CopyJob copy[2];
  bool contain;              // infinities and NaN become zeros in the images
  int act;
  uint32_t* hdr;
  int scan_c, scan_g;        // blocks that scan each array
  int blocks_c, blocks_t, blocks_g, blocks_copy;
};

// Maxima, then images and copies: two launches, and between them what the context has to be run beside the first.
int launch_prep(PrepParams& P, const LaunchCtx& c);

// Unsigned division by a constant: n / d for any 32-bit n (Granlund and Montgomery, "Division by invariant integers using
// multiplication", figure 4.1), for the places within the images.
struct FastDiv {
  uint32_t d, mul, s1, s2;
  explicit FastDiv(uint32_t divisor = 1) : d(divisor) {
    uint32_t l = 0;
    while ((1ull << l) < d) ++l;
    mul = (uint32_t)((((1ull << l) - d) << 32) / d + 1);
    s1 = l < 1 ? l : 1;
    s2 = l < 1 ? 0 : l - 1;
  }
  __device__ __forceinline__ uint32_t div(uint32_t n) const {
    const uint32_t t = __umulhi(mul, n);
    return (t + ((n - t) >> s1)) >> s2;
  }
};

// out[n][c] = lambda * 2^-k * sum over splits of partial[split][n][c], c < r of the rp partial columns.
int launch_finalize(const float* partial, int splits, int64_t N, int r, int rp, float lambda, const uint32_t* hdr,
                    void* out, int64_t ds, bool out_f32, const Contain& K, cudaStream_t stream);

// How many partials a knot row of dC has: `count`, or (count = 0) the number of runs of `run` places that touch the row's slab of
// `slab_rows` rows and `pitch` places.
struct DcParts {
  int count;
  uint32_t pitch, run, slab_rows;
  __host__ __device__ int of(uint32_t slab) const {
    return count ? count : (int)(((slab + 1) * pitch - 1) / run - slab * pitch / run) + 1;
  }
};

// dC = lambda * 2^-k * sum over the partials part[i][row][c] for `rows` knot rows.  Where K has dz in padded rows, its blocks
// bring it to its place too.
int launch_dc_reduce(const float* part, const DcParts& parts, int64_t rows, int64_t rows_padded, int r, int rp, float lambda,
                     const uint32_t* hdr, float* dC, void* dC_cast, const Contain& K, cudaStream_t stream);

// What infinities and NaN add to dz, for a call without dC (launch_dc_reduce does the same for the others).
int launch_dz_contain(const Contain& K, const uint32_t* hdr, cudaStream_t stream);

// dst[n][j] = src[n][j], j < h, from padded rows.
int launch_unpad(const void* src, int64_t ss, void* dst, int64_t ds, int64_t N, int h, bool f32, cudaStream_t stream);

}  // namespace tc
}  // namespace skv
