// What surrounds the tensor-core kernels of a call: range scales and f16 operand images before them, the
// sums over key or token splits after them.
//
// Each of these is a few microseconds of memory traffic, so launches, not bytes, are what they cost: the
// scans of C and g_delta share one launch, all images and copies another, and the maximum is combined by
// every warp of the second launch from the block maxima of the first, which needs neither atomics
// nor a cleared word.
#include "skv_tc_prep.cuh"

namespace skv {
namespace tc {
namespace {

constexpr uint32_t kInf = 0x7f800000u;                    // NaN patterns lie above it
constexpr uint32_t kBadBit = 0x80000000u;                 // of a block's word: it has seen an infinity or a NaN

// Largest |x| of packed bf16 as a float32 bit pattern: of all values, or (FINITE) of the finite ones.
template <bool FINITE>
__device__ __forceinline__ uint32_t absmax(uint32_t m, uint32_t w) {
  const uint32_t lo = (w << 16) & 0x7fff0000u, hi = w & 0x7fff0000u;
  if (!FINITE || lo < kInf) m = max(m, lo);
  if (!FINITE || hi < kInf) m = max(m, hi);
  return m;
}
template <bool FINITE>
__device__ __forceinline__ uint32_t absmax(uint32_t m, const uint4& v) {
  return absmax<FINITE>(absmax<FINITE>(absmax<FINITE>(absmax<FINITE>(m, v.x), v.y), v.z), v.w);
}

// Maximum over the block; valid in every thread.  `words` is shared scratch of 32 words.
__device__ __forceinline__ uint32_t block_max(uint32_t m, uint32_t* words) {
  m = __reduce_max_sync(0xffffffffu, m);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) words[threadIdx.x >> 5] = m;
  __syncthreads();
  const int nw = blockDim.x >> 5;
  m = (threadIdx.x & 31) < nw ? words[threadIdx.x & 31] : 0u;
  return __reduce_max_sync(0xffffffffu, m);
}

__device__ __forceinline__ uint4 ld8(const __nv_bfloat16* p, int n, bool vec) {   // n of 8 elements, the rest zero
  if (vec) return __ldg(reinterpret_cast<const uint4*>(p));
  const unsigned short* s = reinterpret_cast<const unsigned short*>(p);
  uint32_t v[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = i < n ? __ldg(s + i) : 0u;
  return make_uint4(v[0] | v[1] << 16, v[2] | v[3] << 16, v[4] | v[5] << 16, v[6] | v[7] << 16);
}

// This thread's share of the array that its block scans.
template <bool FINITE>
__device__ __forceinline__ uint32_t scan_share(const PrepParams& P, bool is_c, int64_t first, int64_t step) {
  uint32_t m = 0;
  if (is_c) {
    const int64_t total = (int64_t)P.h * P.L * P.r;
    const int64_t n8 = (reinterpret_cast<uintptr_t>(P.C) & 15) == 0 ? total / 8 : 0;
#pragma unroll 4
    for (int64_t i = first; i < n8; i += step) m = absmax<FINITE>(m, __ldg(reinterpret_cast<const uint4*>(P.C) + i));
    for (int64_t i = n8 * 8 + first; i < total; i += step)
      m = absmax<FINITE>(m, (uint32_t)__ldg(reinterpret_cast<const unsigned short*>(P.C) + i));
  } else {
    const bool vec = P.r % 8 == 0 && P.gds % 8 == 0 && (reinterpret_cast<uintptr_t>(P.g) & 15) == 0;
    const int cgs = (P.r + 7) / 8;
    const int64_t pieces = P.N * cgs;
#pragma unroll 4
    for (int64_t i = first; i < pieces; i += step) {
      const int64_t n = i / cgs;
      const int c = (int)(i - n * cgs) * 8;
      m = absmax<FINITE>(m, ld8(P.g + n * P.gds + c, P.r - c, vec));
    }
  }
  return m;
}

__global__ void __launch_bounds__(256) tc_scan_kernel(const __grid_constant__ PrepParams P) {
  __shared__ uint32_t words[32];
  pdl_wait();
  pdl_launch();                                         // only now: later kernels may read the call's inputs at once
  const bool is_c = (int)blockIdx.x < P.scan_c;
  const int blk = is_c ? blockIdx.x : blockIdx.x - P.scan_c, nblk = is_c ? P.scan_c : P.scan_g;
  const int64_t first = (int64_t)blk * blockDim.x + threadIdx.x, step = (int64_t)nblk * blockDim.x;
  uint32_t m = block_max(scan_share<false>(P, is_c, first, step), words);
  if (m >= kInf) m = block_max(scan_share<true>(P, is_c, first, step), words) | kBadBit;   // once more, without them
  if (threadIdx.x == 0) P.hdr[kBlockMax + (is_c ? 0 : kMaxBlocks) + blk] = m;
}

// Maximum of the block maxima, by every warp for itself: no barrier between the wait for the scan and the first image.
__device__ __forceinline__ uint32_t combine(const uint32_t* part, int n, bool& bad) {
  uint32_t m = 0, all = 0;
#pragma unroll 4
  for (int i = threadIdx.x & 31; i < n; i += 32) {
    const uint32_t v = part[i];
    m = max(m, v & ~kBadBit);
    all |= v;
  }
  bad = __any_sync(0xffffffffu, (all & kBadBit) != 0u);
  return __reduce_max_sync(0xffffffffu, m);
}

// Eight bf16 with zeros in the place of infinities and NaN.
__device__ __forceinline__ uint32_t finite2(uint32_t w) {
  return ((w & 0x7f80u) == 0x7f80u ? 0u : w & 0xffffu) | ((w & 0x7f800000u) == 0x7f800000u ? 0u : w & 0xffff0000u);
}
__device__ __forceinline__ uint4 finite8(const uint4& v, bool bad) {
  return bad ? make_uint4(finite2(v.x), finite2(v.y), finite2(v.z), finite2(v.w)) : v;
}

__device__ __forceinline__ uint4 scaled_h8(const uint4& v, float s) {
  return make_uint4(pack_h2(bf_lo(v.x) * s, bf_hi(v.x) * s), pack_h2(bf_lo(v.y) * s, bf_hi(v.y) * s),
                    pack_h2(bf_lo(v.z) * s, bf_hi(v.z) * s), pack_h2(bf_lo(v.w) * s, bf_hi(v.w) * s));
}

// Second difference of one bf16 column triple, scaled by a power of two (exact), as the dz table wants it.
__device__ __forceinline__ float diff2(float a, float b, float c, float s) { return (a - 2.0f * b + c) * s; }

// Division constants of the packing kernel: channel groups per row of the C image, the T image and g, rows per key of both.
struct PackDiv { FastDiv cgi_c, cgi_t, cgs, lpc, lpt; };

// Images.  Piece e (16 bytes) of an image is row e & 7 of the core matrix e >> 3; core matrices run over code
// channels first, then over groups of eight rows, so consecutive threads write consecutive bytes and
// the threads of a warp read whole rows.
//
// The sources of a thread's first pieces are requested before the wait for the scan, and rows are copied there (all are inputs of
// the call); what is left behind it is the maximum, arithmetic and stores.
constexpr int kPieces = 2;                              // pieces a thread works on at a time

template <bool IS_T>
__device__ __forceinline__ void pack_table(const PrepParams& P, const PackDiv& F, int blk) {
  const int cgs = P.rp / 8, cgi = IS_T ? cgs * P.tparts : cgs;             // channel groups of the image
  const int nblk = IS_T ? P.blocks_t : P.blocks_c, LP = IS_T ? P.lpt : P.lpc;
  const FastDiv &fc = IS_T ? F.cgi_t : F.cgi_c, &fl = IS_T ? F.lpt : F.lpc;
  const bool cvec = P.r % 8 == 0 && (reinterpret_cast<uintptr_t>(P.C) & 15) == 0;
  const int64_t pieces = (int64_t)P.hp * LP * cgi, step = (int64_t)nblk * blockDim.x;
  uint4* img = reinterpret_cast<uint4*>(IS_T ? P.timg : P.cimg);
  uint4 v[kPieces][IS_T ? 3 : 1];
  int bs[kPieces];                                      // row of the key, with kRest: of the remainders; -1: zeros
  constexpr int kRest = 1 << 16;
  auto request = [&](int64_t e0) {
#pragma unroll
    for (int x = 0; x < kPieces; ++x) {
      const int64_t e = e0 + x * step;
      bs[x] = -1;
      if (e >= pieces) continue;
      const uint32_t core = (uint32_t)(e >> 3), rg = fc.div(core);
      uint32_t cg = core - rg * (uint32_t)cgi;
      const bool rest = IS_T && cg >= (uint32_t)cgs;
      if (rest) cg -= cgs;
      const uint32_t row = rg * 8u + ((uint32_t)e & 7u), j = fl.div(row);
      const int b = (int)(row - j * LP), c = (int)cg * 8, left = P.r - c;
      if ((int)j >= P.h || left <= 0) continue;
      const __nv_bfloat16* base = P.C + (size_t)j * P.L * P.r + c;
      if constexpr (!IS_T) {
        // group f = b / 4 holds knot rows 2f, 2f + 1 and 2(f + F - 1), 2(f + F - 1) + 1, F = LP / 4 groups
        const int kr = 2 * (b >> 2) + (b & 1) + ((b & 2) ? LP / 2 - 2 : 0);
        if (kr >= P.L) continue;
        v[x][0] = ld8(base + (size_t)kr * P.r, left, cvec);
      } else {
        // b = 0: C[1] - C[0]; b > 0: C[b-1] - 2 C[b] + C[b+1]
        if (b >= P.L - 1) continue;
        v[x][0] = ld8(base + (size_t)(b > 0 ? b - 1 : 0) * P.r, left, cvec);
        v[x][1] = ld8(base + (size_t)(b > 0 ? b : 1) * P.r, left, cvec);
        v[x][2] = b > 0 ? ld8(base + (size_t)(b + 1) * P.r, left, cvec) : make_uint4(0, 0, 0, 0);
      }
      bs[x] = b + (rest ? kRest : 0);
    }
  };
  const int64_t first = (int64_t)blk * blockDim.x + threadIdx.x;
  request(first);
  pdl_wait();
  float scale, inv;
  bool bad;
  pow2_scales(combine(P.hdr + kBlockMax, P.scan_c, bad), scale, inv);
  bad = bad && P.contain;
  for (int64_t e0 = first; e0 < pieces; e0 += kPieces * step) {
    if (e0 != first) request(e0);
#pragma unroll
    for (int x = 0; x < kPieces; ++x) {
      if (e0 + x * step >= pieces) break;
      uint4 o = make_uint4(0, 0, 0, 0);
      if (bs[x] >= 0) {
        if constexpr (!IS_T) {
          o = scaled_h8(finite8(v[x][0], bad), scale);
        } else {
          const bool rest = bs[x] >= kRest, b0 = (bs[x] & (kRest - 1)) == 0;
          const uint4 v0 = finite8(v[x][0], bad), v1 = finite8(v[x][1], bad), v2 = finite8(v[x][2], bad);
          const uint32_t a0[4] = {v0.x, v0.y, v0.z, v0.w}, a1[4] = {v1.x, v1.y, v1.z, v1.w}, a2[4] = {v2.x, v2.y, v2.z, v2.w};
          uint32_t w[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float lo = b0 ? (bf_lo(a1[i]) - bf_lo(a0[i])) * scale : diff2(bf_lo(a0[i]), bf_lo(a1[i]), bf_lo(a2[i]), scale);
            float hi = b0 ? (bf_hi(a1[i]) - bf_hi(a0[i])) * scale : diff2(bf_hi(a0[i]), bf_hi(a1[i]), bf_hi(a2[i]), scale);
            if (rest) {
              lo -= __half2float(__float2half_rn(lo));
              hi -= __half2float(__float2half_rn(hi));
            }
            w[i] = pack_h2(lo, hi);
          }
          o = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
      img[e0 + x * step] = o;
    }
  }
}

__global__ void __launch_bounds__(256) tc_pack_kernel(const __grid_constant__ PrepParams P, const __grid_constant__ PackDiv F) {
  pdl_launch();
  int blk = blockIdx.x;
  if (blk < P.blocks_c + P.blocks_t) {
    if (blk < P.blocks_c) pack_table<false>(P, F, blk);
    else pack_table<true>(P, F, blk - P.blocks_c);
  } else if (blk < P.blocks_c + P.blocks_t + P.blocks_g) {
    const int cgs = P.rp / 8;
    const bool vec = P.r % 8 == 0 && P.gds % 8 == 0 && (reinterpret_cast<uintptr_t>(P.g) & 15) == 0;
    const int64_t pieces = P.tiles * 128 * cgs, step = (int64_t)P.blocks_g * blockDim.x;
    const int64_t first = (int64_t)(blk - P.blocks_c - P.blocks_t) * blockDim.x + threadIdx.x;
    uint4* img = reinterpret_cast<uint4*>(P.gimg);
    uint4 v[kPieces];
    auto request = [&](int64_t e0) {
#pragma unroll
      for (int x = 0; x < kPieces; ++x) {
        const int64_t e = e0 + x * step;
        const int64_t tc_ = e >> 7;                     // (tile, channel group)
        const int64_t tile = P.tiles < (1 << 27) ? (int64_t)F.cgs.div((uint32_t)tc_) : tc_ / cgs;
        const int c = (int)(tc_ - tile * cgs) * 8;
        const int64_t n = tile * 128 + (e & 127);
        v[x] = e < pieces && n < P.N && c < P.r ? ld8(P.g + n * P.gds + c, P.r - c, vec) : make_uint4(0, 0, 0, 0);
      }
    };
    request(first);
    pdl_wait();
    float scale, inv;
    bool bad;
    pow2_scales(combine(P.hdr + kBlockMax + kMaxBlocks, P.scan_g, bad), scale, inv);
    bad = bad && P.contain;
    for (int64_t e0 = first; e0 < pieces; e0 += kPieces * step) {
      if (e0 != first) request(e0);
#pragma unroll
      for (int x = 0; x < kPieces; ++x)
        if (e0 + x * step < pieces) img[e0 + x * step] = scaled_h8(finite8(v[x], bad), scale);
    }
  } else {
    blk -= P.blocks_c + P.blocks_t + P.blocks_g;
    for (int q = 0; q < 2; ++q) {
      const CopyJob& J = P.copy[q];
      if (!J.dst && !J.act_out) continue;
      const int w8 = P.hp / 8;
      const int64_t pieces = P.N * w8;
      for (int64_t i = (int64_t)blk * blockDim.x + threadIdx.x; i < pieces; i += (int64_t)P.blocks_copy * blockDim.x) {
        const int64_t n = i / w8;
        const int c = (int)(i - n * w8) * 8, left = min(8, P.h - c);
        const uint4 v = ld8(J.src + n * J.ss + c, left, false);
        if (J.dst) *reinterpret_cast<uint4*>(J.dst + n * P.hp + c) = v;
        if (J.act_out) {
          const uint32_t w[4] = {v.x, v.y, v.z, v.w};
          __nv_bfloat16* o = J.act_out + n * J.as + c;
#pragma unroll
          for (int k = 0; k < 8; ++k)
            if (k < left) o[k] = __float2bfloat16_rn(act_fwd((k & 1) ? bf_hi(w[k >> 1]) : bf_lo(w[k >> 1]), P.act));
        }
      }
    }
  }
  pdl_wait();                                           // whoever waits for this kernel has waited for the scan
  if (blockIdx.x == 0 && threadIdx.x < 32) {            // final maxima for the kernels that follow
    bool bad;
    if (P.scan_c) {
      const uint32_t m = combine(P.hdr + kBlockMax, P.scan_c, bad);
      if (threadIdx.x == 0) { P.hdr[kAmaxC] = m; P.hdr[kBadC] = bad; }
    }
    if (P.scan_g) {
      const uint32_t m = combine(P.hdr + kBlockMax + kMaxBlocks, P.scan_g, bad);
      if (threadIdx.x == 0) { P.hdr[kAmaxG] = m; P.hdr[kBadG] = bad; }
    }
  }
}

__device__ __forceinline__ bool is_bad(float x) { return (__float_as_uint(x) & 0x7f800000u) == 0x7f800000u; }

__device__ __forceinline__ float pair_weight(const Knot& k, int row, int order) {
  float B0, B1, B2;
  basis_weights(k, B0, B1, B2, order);
  return row == 0 ? B0 : row == 1 ? B1 : B2;
}

// delta: the contributions of infinities and NaN in C (a zero weight times one is NaN here too, as it is when the
// touched rows alone are added up).  A block takes the `outputs` groups of four columns that it has written.
template <typename TD>
__device__ __noinline__ void contain_delta(const Contain& K, int rp, float lambda, TD* out, int64_t ds, int outputs) {
  const int q4 = rp / 4;
  const int64_t total = K.N * q4;
  if ((int)threadIdx.x >= outputs) return;
  for (int64_t i = (int64_t)blockIdx.x * outputs + threadIdx.x; i < total; i += (int64_t)gridDim.x * outputs) {
    const int64_t n = i / q4;
    const int c = (int)(i - n * q4) * 4;
    float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    bool any[4] = {false, false, false, false};
    for (int j = 0; j < K.h; ++j) {
      const Knot k = knot_of(__bfloat162float(K.z[n * K.zs + j]), K.grid);
      for (int row = 0; row <= K.grid.order; ++row) {
        const __nv_bfloat16* src = K.C + ((size_t)j * K.L + k.bin + row) * K.r + c;
        for (int x = 0; x < 4 && c + x < K.r; ++x) {
          const float v = __bfloat162float(src[x]);
          if (is_bad(v)) {
            s[x] = fmaf(pair_weight(k, row, K.grid.order), v, s[x]);
            any[x] = true;
          }
        }
      }
    }
    for (int x = 0; x < 4; ++x)
      if (any[x]) st_f32<TD>(out + n * ds + c + x, lambda * s[x]);
  }
}

// dC: the same for infinities and NaN in g_delta.  A block lists the tokens that have any, 256 tokens at a time, and its
// threads, one per four columns of a knot row, walk the list.
__device__ __noinline__ void contain_dC(const Contain& K, int rp, float lambda, float* dC, __nv_bfloat16* dC_cast, int blocks) {
  __shared__ int list[256];
  __shared__ int count;
  const int q4 = rp / 4;
  const int64_t total = (int64_t)K.h * K.L * q4;
  for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < total; base += (int64_t)blocks * blockDim.x) {
    const int64_t i = base + threadIdx.x;
    const int64_t row = i / q4;
    const int c = (int)(i - row * q4) * 4, j = (int)(row / K.L), l = (int)(row - (int64_t)j * K.L);
    float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    bool any[4] = {false, false, false, false};
    for (int64_t n0 = 0; n0 < K.N; n0 += 256) {
      __syncthreads();
      if (threadIdx.x == 0) count = 0;
      __syncthreads();
      if (n0 + threadIdx.x < K.N) {
        const __nv_bfloat16* g = K.g + (n0 + threadIdx.x) * K.gds;
        bool bad = false;
        for (int e = 0; e < K.r; ++e) bad = bad || is_bad(__bfloat162float(g[e]));
        if (bad) list[atomicAdd(&count, 1)] = threadIdx.x;
      }
      __syncthreads();
      if (i < total) {
        for (int e = 0; e < count; ++e) {
          const int64_t n = n0 + list[e];
          const Knot k = knot_of(__bfloat162float(K.z[n * K.zs + j]), K.grid);
          if (!k.in_range || l < k.bin || l > k.bin + K.grid.order) continue;
          const float w = pair_weight(k, l - k.bin, K.grid.order);
          for (int x = 0; x < 4 && c + x < K.r; ++x) {
            const float v = __bfloat162float(K.g[n * K.gds + c + x]);
            if (is_bad(v)) {
              s[x] = fmaf(w, v, s[x]);
              any[x] = true;
            }
          }
        }
      }
    }
    for (int x = 0; x < 4; ++x) {
      if (!any[x]) continue;
      if (dC) dC[row * K.r + c + x] = lambda * s[x];
      if (dC_cast) dC_cast[row * K.r + c + x] = __float2bfloat16_rn(lambda * s[x]);
    }
  }
}

// dz: the channels of a pair in which g_delta or a touched row of C is infinite or NaN.  A block takes 256 tokens (one per
// thread) x 32 keys and first marks the knot rows of its keys and the tokens that have any.  Where dz is still in padded rows,
// all of it is brought to its place.
__device__ __noinline__ void contain_dz(const Contain& K, bool bad_g, bool bad_c, int64_t first, int64_t step) {
  __shared__ unsigned long long rows[32];
  const int key_groups = (K.h + 31) / 32;
  const int64_t tiles = (K.N + 255) / 256 * key_groups;
  for (int64_t t = first; t < tiles; t += step) {
    const int64_t n = t / key_groups * 256 + threadIdx.x;
    const int j0 = (int)(t % key_groups) * 32, keys = min(32, K.h - j0);
    __syncthreads();
    if (threadIdx.x < 32) rows[threadIdx.x] = 0ull;
    __syncthreads();
    if (bad_c)
      for (int e = threadIdx.x; e < keys * K.L; e += blockDim.x) {
        const __nv_bfloat16* src = K.C + ((size_t)j0 * K.L + e) * K.r;
        bool bad = false;
        for (int c = 0; c < K.r; ++c) bad = bad || is_bad(__bfloat162float(src[c]));
        if (bad) atomicOr(&rows[e / K.L], 1ull << (e % K.L));
      }
    const __nv_bfloat16* g = K.g + (n < K.N ? n : 0) * K.gds;
    bool token = false;
    if (bad_g && n < K.N)
      for (int c = 0; c < K.r; ++c) token = token || is_bad(__bfloat162float(g[c]));
    __syncthreads();
    for (int q = 0; q < keys && n < K.N; ++q) {
      const Knot k = knot_of(__bfloat162float(K.z[n * K.zs + j0 + q]), K.grid);
      const bool two = K.grid.order != 1;
      const __nv_bfloat16* src = K.C + ((size_t)(j0 + q) * K.L + k.bin) * K.r;
      float s = 0.0f;
      bool any = false;
      const bool touched = k.clamp_active && (token || ((rows[q] >> k.bin) & (two ? 7ull : 3ull)));
      for (int c = 0; touched && c < K.r; ++c) {
        const float gv = __bfloat162float(g[c]), c0 = __bfloat162float(src[c]), c1 = __bfloat162float(src[K.r + c]);
        const float c2 = two ? __bfloat162float(src[2 * K.r + c]) : 0.0f;
        if (!is_bad(gv) && !is_bad(c0) && !is_bad(c1) && !is_bad(c2)) continue;
        float d = c1 - c0;
        if (two) d = fmaf(k.tau, (c2 - c1) - d, d);
        s = fmaf(gv, d, s);
        any = true;
      }
      if (!any && !K.dz_rows) continue;
      const int64_t at = n * K.dzs + j0 + q, from = K.dz_rows ? n * K.dz_rows_stride + j0 + q : at;
      if (K.dz_f32) {
        float v = static_cast<const float*>(K.dz_rows ? K.dz_rows : K.dz)[from];
        if (any) v += K.coef * s;
        static_cast<float*>(K.dz)[at] = v;
      } else {
        __nv_bfloat16 v = static_cast<const __nv_bfloat16*>(K.dz_rows ? K.dz_rows : K.dz)[from];
        if (any) v = __float2bfloat16_rn(__bfloat162float(v) + K.coef * s);
        static_cast<__nv_bfloat16*>(K.dz)[at] = v;
      }
    }
  }
}

// Four consecutive columns per thread, SG lanes per output: each adds every SG-th split, eight loads in flight, and the
// SG sums are exchanged within the warp.  What one thread would add alone is a chain of round trips to L2:
// 1999 x 2560 (36 partials of 16 K outputs) 6.8 us behind the forward with SG = 1.
template <typename TD, bool CONTAIN, int SG>
__global__ void __launch_bounds__(256) tc_finalize_kernel(const float* partial, int splits, int64_t N, int r,
                                                          int rp, float lambda, const uint32_t* hdr,
                                                          TD* out, int64_t ds, const __grid_constant__ Contain K) {
  constexpr int kOut = 256 / SG;                        // outputs of a block
  pdl_wait();
  pdl_launch();
  float cscale, cinv;
  pow2_scales(hdr[kAmaxC], cscale, cinv);
  const float f = lambda * cinv;                        // undo the code-table image's range scaling
  const int q4 = rp / 4;
  const int64_t total = N * q4;
  const bool vec = ds % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0 && r == rp;
  constexpr int kPerWarp = 32 / SG;
  const int me = (int)(threadIdx.x / 32) * kPerWarp + (int)(threadIdx.x % kPerWarp), sg = (int)(threadIdx.x % 32) / kPerWarp;
  for (int64_t b = (int64_t)blockIdx.x * kOut; b < total; b += (int64_t)gridDim.x * kOut) {
    const int64_t i = b + me;
    float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (i < total) {
      const float4* src = reinterpret_cast<const float4*>(partial) + i;
#pragma unroll 8
      for (int k = sg; k < splits; k += SG) {
        const float4 v = src[(size_t)k * total];
        s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
      }
    }
#pragma unroll
    for (int x = kPerWarp; x < 32; x <<= 1) {
      s.x += __shfl_xor_sync(0xffffffffu, s.x, x);
      s.y += __shfl_xor_sync(0xffffffffu, s.y, x);
      s.z += __shfl_xor_sync(0xffffffffu, s.z, x);
      s.w += __shfl_xor_sync(0xffffffffu, s.w, x);
    }
    if (sg > 0) continue;
    if (i >= total) continue;
    const int64_t n = i / q4;
    const int c = (int)(i - n * q4) * 4;
    TD* o = out + n * ds + c;
    const float v[4] = {f * s.x, f * s.y, f * s.z, f * s.w};
    if (vec) {
      if constexpr (sizeof(TD) == 4) *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
      else *reinterpret_cast<uint2*>(o) = make_uint2(pack_bf2(v[0], v[1]), pack_bf2(v[2], v[3]));
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (c + k < r) st_f32<TD>(o + k, v[k]);
    }
  }
  if constexpr (CONTAIN) {
    if (hdr[kBadC] != 0u) {
      __syncthreads();                                  // the block's outputs are written: its threads take them in turn
      contain_delta(K, rp, lambda, out, ds, kOut);
    }
  }
}

// Rows of h elements from padded rows, a row per block at a time.
template <typename T>
__device__ __forceinline__ void unpad_rows(const void* src, int64_t ss, void* dst, int64_t ds, int64_t N, int h, int64_t first, int64_t step) {
  for (int64_t n = first; n < N; n += step) {
    const T* a = static_cast<const T*>(src) + n * ss;
    T* b = static_cast<T*>(dst) + n * ds;
#pragma unroll 4
    for (int j = threadIdx.x; j < h; j += blockDim.x) b[j] = a[j];
  }
}

// The first `blocks` blocks add; those behind them bring dz from padded rows to its place (a launch of its own for that took
// the GPU 5 us of a step of 2000 x 1001; the step waits for the host, and stayed at 77).  Where infinities or NaN were found
// contain_dz does both.
template <bool CONTAIN>
__global__ void __launch_bounds__(256) tc_dc_reduce_kernel(const float* part, const DcParts parts, int64_t rows,
                                                           int64_t rows_padded, int r, int rp, float lambda,
                                                           const uint32_t* hdr, float* dC,
                                                           __nv_bfloat16* dC_cast, const __grid_constant__ Contain K, int blocks) {
  pdl_wait();
  pdl_launch();
  if constexpr (CONTAIN) {
    if ((int)blockIdx.x >= blocks) {
      const bool bad_g = hdr[kBadG] != 0u, bad_c = hdr[kBadC] != 0u;
      const int64_t first = blockIdx.x - blocks, step = gridDim.x - blocks;
      if (bad_g || bad_c) contain_dz(K, bad_g, bad_c, first, step);
      else if (K.dz_f32) unpad_rows<float>(K.dz_rows, K.dz_rows_stride, K.dz, K.dzs, K.N, K.h, first, step);
      else unpad_rows<__nv_bfloat16>(K.dz_rows, K.dz_rows_stride, K.dz, K.dzs, K.N, K.h, first, step);
      return;
    }
  }
  float gscale, ginv;
  pow2_scales(hdr[kAmaxG], gscale, ginv);
  const float f = lambda * ginv;
  const int q4 = rp / 4;
  const int64_t total = rows * q4, pitch = rows_padded * q4;
  const bool vec = r == rp && ((reinterpret_cast<uintptr_t>(dC) | reinterpret_cast<uintptr_t>(dC_cast)) & 15) == 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)blocks * blockDim.x) {
    const float4* src = reinterpret_cast<const float4*>(part) + i;
    const int splits = parts.count ? parts.count : parts.of((uint32_t)(i / q4) / parts.slab_rows);
    float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 8
    for (int k = 0; k < splits; ++k) {
      const float4 v = __ldcs(src + (size_t)k * pitch);
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    s.x *= f; s.y *= f; s.z *= f; s.w *= f;
    if (vec) {
      if (dC) reinterpret_cast<float4*>(dC)[i] = s;
      if (dC_cast) reinterpret_cast<uint2*>(dC_cast)[i] = make_uint2(pack_bf2(s.x, s.y), pack_bf2(s.z, s.w));
    } else {
      const int64_t row = i / q4;
      const int c = (int)(i - row * q4) * 4;
      const float v[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (c + k >= r) break;
        if (dC) dC[row * r + c + k] = v[k];
        if (dC_cast) dC_cast[row * r + c + k] = __float2bfloat16_rn(v[k]);
      }
    }
  }
  if constexpr (CONTAIN) {
    const bool bad_g = hdr[kBadG] != 0u;
    if (bad_g) contain_dC(K, rp, lambda, dC, dC_cast, blocks);      // the elements of a thread are those it has written above
    if (K.dz && !K.dz_rows) {
      const bool bad_c = hdr[kBadC] != 0u;
      if (bad_g || bad_c) contain_dz(K, bad_g, bad_c, blockIdx.x, blocks);
    }
  }
}

__global__ void __launch_bounds__(256) tc_dz_contain_kernel(const uint32_t* hdr, const __grid_constant__ Contain K) {
  pdl_wait();
  pdl_launch();
  const bool bad_g = hdr[kBadG] != 0u, bad_c = hdr[kBadC] != 0u;
  if (bad_g || bad_c) contain_dz(K, bad_g, bad_c, blockIdx.x, gridDim.x);
}

template <typename T>
__global__ void __launch_bounds__(256) tc_unpad_kernel(const T* src, int64_t ss, T* dst, int64_t ds,
                                                       int64_t N, int h) {
  pdl_launch();
  pdl_wait();
  const int64_t total = N * h;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t n = i / h;
    const int j = (int)(i - n * h);
    dst[n * ds + j] = src[n * ss + j];
  }
}

int blocks_for(int64_t items, int64_t per_thread, int most) {
  const int64_t b = (items + 256 * per_thread - 1) / (256 * per_thread);
  return (int)(b < 1 ? 1 : (b > most ? most : b));
}

}  // namespace

int launch_prep(PrepParams& P, const LaunchCtx& ctx) {
  const cudaStream_t stream = ctx.stream;
  const int cgs = P.rp / 8;
  P.scan_c = P.lpc || P.lpt ? blocks_for((int64_t)P.h * P.L * P.r / 8, 2, kMaxBlocks) : 0;
  P.scan_g = P.g ? blocks_for(P.N * ((P.r + 7) / 8), 2, kMaxBlocks) : 0;
  P.blocks_c = P.lpc ? blocks_for((int64_t)P.hp * P.lpc * cgs, 2, kPlanSMs * 8) : 0;
  P.blocks_t = P.lpt ? blocks_for((int64_t)P.hp * P.lpt * cgs * P.tparts, 2, kPlanSMs * 8) : 0;
  P.blocks_g = P.g ? blocks_for(P.tiles * 128 * cgs, 2, kPlanSMs * 8) : 0;
  P.blocks_copy = 0;
  for (const CopyJob& J : P.copy)
    if (J.dst || J.act_out) P.blocks_copy = blocks_for(P.N * (P.hp / 8), 1, kPlanSMs * 16);
  // Not chained to what was on the stream: an SM that never runs empty keeps the split of shared memory and L1 that the last kernel
  // asked for, and behind a dC (all of it shared memory) the forward's strided rows of z find no L1 (65536 x 5120: 770 -> 977 us).
  tc_scan_kernel<<<(unsigned)(P.scan_c + P.scan_g), 256, 0, stream>>>(P);
  if (cudaGetLastError() != cudaSuccess) return SKV_ERR_LAUNCH;
  if (ctx.beside)
    if (int e = ctx.beside(ctx.beside_arg, false)) return e;
  const unsigned grid = (unsigned)(P.blocks_c + P.blocks_t + P.blocks_g + P.blocks_copy);
  const PackDiv F{FastDiv(cgs), FastDiv(cgs * (P.tparts ? P.tparts : 1)), FastDiv(cgs), FastDiv(P.lpc ? P.lpc : 1), FastDiv(P.lpt ? P.lpt : 1)};
  if (launch_chained<tc_pack_kernel>(dim3(grid), 256, 0, stream, P, F) != cudaSuccess) return SKV_ERR_LAUNCH;
  note_launches(2);
  return SKV_OK;
}

namespace {
template <typename TD, bool CONTAIN>
cudaError_t finalize(cudaStream_t stream, const float* partial, int splits, int64_t N, int r, int rp, float lambda,
                     const uint32_t* hdr, void* out, int64_t ds, const Contain& K) {
  // lanes per output: so many that a lane has two rounds of eight loads, where the outputs alone do not fill the chip
  // with four blocks per SM (9 splits, 8192 x 5120: 3.5 us with one lane, 4.7 with two)
  const int64_t outputs = N * (rp / 4);
  int sg = 1;
  while (sg < 8 && splits > 16 * sg && outputs * sg < (int64_t)kPlanSMs * 1024) sg *= 2;
  const dim3 grid((unsigned)blocks_for(outputs * sg, 1, kPlanSMs * 16));
  auto go = [&](auto n) {
    return launch_chained<tc_finalize_kernel<TD, CONTAIN, decltype(n)::value>>(grid, 256, 0, stream, partial, splits, N, r, rp, lambda,
                                                                               hdr, static_cast<TD*>(out), ds, K);
  };
  return sg == 1   ? go(std::integral_constant<int, 1>())
         : sg == 2 ? go(std::integral_constant<int, 2>())
         : sg == 4 ? go(std::integral_constant<int, 4>())
                   : go(std::integral_constant<int, 8>());
}
}  // namespace

int launch_finalize(const float* partial, int splits, int64_t N, int r, int rp, float lambda, const uint32_t* hdr,
                    void* out, int64_t ds, bool out_f32, const Contain& K, cudaStream_t stream) {
  auto* run = out_f32 ? (K.z ? finalize<float, true> : finalize<float, false>)
                      : (K.z ? finalize<__nv_bfloat16, true> : finalize<__nv_bfloat16, false>);
  const cudaError_t e = run(stream, partial, splits, N, r, rp, lambda, hdr, out, ds, K);
  note_launches(1);
  return e == cudaSuccess ? SKV_OK : SKV_ERR_LAUNCH;
}

int launch_dc_reduce(const float* part, const DcParts& parts, int64_t rows, int64_t rows_padded, int r, int rp, float lambda,
                     const uint32_t* hdr, float* dC, void* dC_cast, const Contain& K, cudaStream_t stream) {
  const int blocks = blocks_for(rows * (rp / 4), 1, kPlanSMs * 16);
  const dim3 grid((unsigned)(blocks + (K.z && K.dz_rows ? (K.N < kPlanSMs * 8 ? (int)K.N : kPlanSMs * 8) : 0)));
  const cudaError_t e =
      K.z ? launch_chained<tc_dc_reduce_kernel<true>>(grid, 256, 0, stream, part, parts, rows, rows_padded, r, rp, lambda, hdr,
                                                      dC, static_cast<__nv_bfloat16*>(dC_cast), K, blocks)
          : launch_chained<tc_dc_reduce_kernel<false>>(grid, 256, 0, stream, part, parts, rows, rows_padded, r, rp, lambda,
                                                       hdr, dC, static_cast<__nv_bfloat16*>(dC_cast), K, blocks);
  note_launches(1);
  return e == cudaSuccess ? SKV_OK : SKV_ERR_LAUNCH;
}

int launch_dz_contain(const Contain& K, const uint32_t* hdr, cudaStream_t stream) {
  const dim3 grid((unsigned)blocks_for(K.N * ((K.h + 31) / 32), 1, kPlanSMs * 4));
  const cudaError_t e = launch_chained<tc_dz_contain_kernel>(grid, 256, 0, stream, hdr, K);
  note_launches(1);
  return e == cudaSuccess ? SKV_OK : SKV_ERR_LAUNCH;
}

int launch_unpad(const void* src, int64_t ss, void* dst, int64_t ds, int64_t N, int h, bool f32, cudaStream_t stream) {
  const dim3 grid((unsigned)blocks_for(N * h, 4, kPlanSMs * 16));
  const cudaError_t e =
      f32 ? launch_chained<tc_unpad_kernel<float>>(grid, 256, 0, stream, static_cast<const float*>(src), ss,
                                                   static_cast<float*>(dst), ds, N, h)
          : launch_chained<tc_unpad_kernel<__nv_bfloat16>>(grid, 256, 0, stream, static_cast<const __nv_bfloat16*>(src), ss,
                                                           static_cast<__nv_bfloat16*>(dst), ds, N, h);
  note_launches(1);
  return e == cudaSuccess ? SKV_OK : SKV_ERR_LAUNCH;
}

}  // namespace tc
}  // namespace skv
