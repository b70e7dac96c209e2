// What surrounds the tensor-core kernels of a call: range scales and f16 operand images before them, the
// sums over key or token splits after them.
//
// Each of these is a few microseconds of memory traffic, so launches, not bytes, are what they cost: the
// scans of C and g_delta share one launch, all images and copies another, and the maximum is combined by
// every block of the second launch from the block maxima of the first, which needs neither atomics
// nor a cleared word.
#include "skv_tc_prep.cuh"

namespace skv {
namespace tc {
namespace {

__device__ __forceinline__ uint32_t absmax_bf2(uint32_t m, uint32_t w) {
  // |x| of a bf16 as a float32 bit pattern; NaN patterns lie above infinity and are skipped
  const uint32_t lo = (w << 16) & 0x7fff0000u, hi = w & 0x7fff0000u;
  if (lo <= 0x7f800000u) m = max(m, lo);
  if (hi <= 0x7f800000u) m = max(m, hi);
  return m;
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

__global__ void __launch_bounds__(256) tc_scan_kernel(const PrepParams P) {
  __shared__ uint32_t words[32];
  pdl_launch();
  uint32_t m = 0;
  const bool is_c = (int)blockIdx.x < P.scan_c;
  const int blk = is_c ? blockIdx.x : blockIdx.x - P.scan_c, nblk = is_c ? P.scan_c : P.scan_g;
  const int64_t first = (int64_t)blk * blockDim.x + threadIdx.x, step = (int64_t)nblk * blockDim.x;
  if (is_c) {
    const int64_t total = (int64_t)P.h * P.L * P.r;
    const int64_t n8 = (reinterpret_cast<uintptr_t>(P.C) & 15) == 0 ? total / 8 : 0;
#pragma unroll 4
    for (int64_t i = first; i < n8; i += step) {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(P.C) + i);
      m = absmax_bf2(absmax_bf2(absmax_bf2(absmax_bf2(m, v.x), v.y), v.z), v.w);
    }
    for (int64_t i = n8 * 8 + first; i < total; i += step)
      m = absmax_bf2(m, __ldg(reinterpret_cast<const unsigned short*>(P.C) + i));
  } else {
    const bool vec = P.r % 8 == 0 && P.gds % 8 == 0 && (reinterpret_cast<uintptr_t>(P.g) & 15) == 0;
    const int cgs = (P.r + 7) / 8;
    const int64_t pieces = P.N * cgs;
#pragma unroll 4
    for (int64_t i = first; i < pieces; i += step) {
      const int64_t n = i / cgs;
      const int c = (int)(i - n * cgs) * 8;
      const uint4 v = ld8(P.g + n * P.gds + c, P.r - c, vec);
      m = absmax_bf2(absmax_bf2(absmax_bf2(absmax_bf2(m, v.x), v.y), v.z), v.w);
    }
  }
  m = block_max(m, words);
  if (threadIdx.x == 0) P.hdr[kBlockMax + (is_c ? 0 : kMaxBlocks) + blk] = m;
}

__device__ __forceinline__ uint32_t combine(const uint32_t* part, int n, uint32_t* words) {
  uint32_t m = 0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) m = max(m, part[i]);
  return block_max(m, words);
}

__device__ __forceinline__ uint4 scaled_h8(const uint4& v, float s) {
  return make_uint4(pack_h2(bf_lo(v.x) * s, bf_hi(v.x) * s), pack_h2(bf_lo(v.y) * s, bf_hi(v.y) * s),
                    pack_h2(bf_lo(v.z) * s, bf_hi(v.z) * s), pack_h2(bf_lo(v.w) * s, bf_hi(v.w) * s));
}

// Second difference of one bf16 column triple, scaled by a power of two (exact), as the dz table wants it.
__device__ __forceinline__ float diff2(float a, float b, float c, float s) { return (a - 2.0f * b + c) * s; }

// Images.  Piece e (16 bytes) of an image is row e & 7 of the core matrix e >> 3; core matrices run over code
// channels first, then over groups of eight rows, so consecutive threads write consecutive bytes and
// the threads of a warp read whole rows.
__global__ void __launch_bounds__(256) tc_pack_kernel(const PrepParams P) {
  __shared__ uint32_t words[32];
  pdl_launch();
  pdl_wait();
  int blk = blockIdx.x;
  const int cgs = P.rp / 8;
  const bool cvec = P.r % 8 == 0 && (reinterpret_cast<uintptr_t>(P.C) & 15) == 0;
  if (blk == 0) {                                       // final maxima for the kernels that follow
    if (P.scan_c) {
      const uint32_t m = combine(P.hdr + kBlockMax, P.scan_c, words);
      if (threadIdx.x == 0) P.hdr[kAmaxC] = m;
    }
    if (P.scan_g) {
      const uint32_t m = combine(P.hdr + kBlockMax + kMaxBlocks, P.scan_g, words);
      if (threadIdx.x == 0) P.hdr[kAmaxG] = m;
    }
  }
  if (blk < P.blocks_c + P.blocks_t) {
    const bool is_t = blk >= P.blocks_c;
    const int nblk = is_t ? P.blocks_t : P.blocks_c;
    if (is_t) blk -= P.blocks_c;
    float scale, inv;
    pow2_scales(combine(P.hdr + kBlockMax, P.scan_c, words), scale, inv);
    const int LP = is_t ? P.lpt : P.lpc;
    const int cgi = is_t ? cgs * P.tparts : cgs;        // channel groups of the image
    const int64_t pieces = (int64_t)P.hp * LP * cgi;
    uint4* img = reinterpret_cast<uint4*>(is_t ? P.timg : P.cimg);
#pragma unroll 2
    for (int64_t e = (int64_t)blk * blockDim.x + threadIdx.x; e < pieces; e += (int64_t)nblk * blockDim.x) {
      const uint32_t core = (uint32_t)(e >> 3);
      const uint32_t rg = core / (uint32_t)cgi;
      uint32_t cg = core - rg * cgi;
      const bool rest = cg >= (uint32_t)cgs;            // remainders
      if (rest) cg -= cgs;
      const uint32_t row = rg * 8u + ((uint32_t)e & 7u);
      const uint32_t j = row / (uint32_t)LP;
      const int b = (int)(row - j * LP), c = (int)cg * 8, left = P.r - c;
      uint4 o = make_uint4(0, 0, 0, 0);
      if ((int)j < P.h && left > 0) {
        const __nv_bfloat16* base = P.C + (size_t)j * P.L * P.r + c;
        if (!is_t) {
          // group f = b / 4 holds knot rows 2f, 2f + 1 and 2(f + F - 1), 2(f + F - 1) + 1, F = LP / 4 groups
          const int kr = 2 * (b >> 2) + (b & 1) + ((b & 2) ? LP / 2 - 2 : 0);
          if (kr < P.L) o = scaled_h8(ld8(base + (size_t)kr * P.r, left, cvec), scale);
        } else if (b < P.L - 1) {
          // b = 0: C[1] - C[0]; b > 0: C[b-1] - 2 C[b] + C[b+1]
          const uint4 v0 = ld8(base + (size_t)(b > 0 ? b - 1 : 0) * P.r, left, cvec);
          const uint4 v1 = ld8(base + (size_t)(b > 0 ? b : 1) * P.r, left, cvec);
          const uint4 v2 = b > 0 ? ld8(base + (size_t)(b + 1) * P.r, left, cvec) : make_uint4(0, 0, 0, 0);
          const uint32_t a0[4] = {v0.x, v0.y, v0.z, v0.w}, a1[4] = {v1.x, v1.y, v1.z, v1.w}, a2[4] = {v2.x, v2.y, v2.z, v2.w};
          uint32_t w[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float lo = b > 0 ? diff2(bf_lo(a0[i]), bf_lo(a1[i]), bf_lo(a2[i]), scale) : (bf_lo(a1[i]) - bf_lo(a0[i])) * scale;
            float hi = b > 0 ? diff2(bf_hi(a0[i]), bf_hi(a1[i]), bf_hi(a2[i]), scale) : (bf_hi(a1[i]) - bf_hi(a0[i])) * scale;
            if (rest) {
              lo -= __half2float(__float2half_rn(lo));
              hi -= __half2float(__float2half_rn(hi));
            }
            w[i] = pack_h2(lo, hi);
          }
          o = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
      img[e] = o;
    }
    return;
  }
  blk -= P.blocks_c + P.blocks_t;
  if (blk < P.blocks_g) {
    float scale, inv;
    pow2_scales(combine(P.hdr + kBlockMax + kMaxBlocks, P.scan_g, words), scale, inv);
    const bool vec = P.r % 8 == 0 && P.gds % 8 == 0 && (reinterpret_cast<uintptr_t>(P.g) & 15) == 0;
    const int64_t pieces = P.tiles * 128 * cgs;
    uint4* img = reinterpret_cast<uint4*>(P.gimg);
#pragma unroll 2
    for (int64_t e = (int64_t)blk * blockDim.x + threadIdx.x; e < pieces; e += (int64_t)P.blocks_g * blockDim.x) {
      const int64_t tc_ = e >> 7;                       // (tile, channel group)
      const int64_t tile = tc_ / cgs;
      const int c = (int)(tc_ - tile * cgs) * 8;
      const int64_t n = tile * 128 + (e & 127);
      img[e] = n < P.N && c < P.r ? scaled_h8(ld8(P.g + n * P.gds + c, P.r - c, vec), scale) : make_uint4(0, 0, 0, 0);
    }
    return;
  }
  blk -= P.blocks_g;
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

// Four consecutive columns per thread; the splits of an element are added in order, four loads in flight.
template <typename TD>
__global__ void __launch_bounds__(256) tc_finalize_kernel(const float* partial, int splits, int64_t N, int r,
                                                          int rp, float lambda, const uint32_t* hdr,
                                                          TD* out, int64_t ds) {
  pdl_launch();
  pdl_wait();
  float cscale, cinv;
  pow2_scales(hdr[kAmaxC], cscale, cinv);
  lambda *= cinv;                                       // undo the code-table image's range scaling
  const int q4 = rp / 4;
  const int64_t total = N * q4;
  const bool vec = ds % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0 && r == rp;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const float4* src = reinterpret_cast<const float4*>(partial) + i;
    float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 8
    for (int k = 0; k < splits; ++k) {
      const float4 v = src[(size_t)k * total];
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    const int64_t n = i / q4;
    const int c = (int)(i - n * q4) * 4;
    TD* o = out + n * ds + c;
    const float v[4] = {lambda * s.x, lambda * s.y, lambda * s.z, lambda * s.w};
    if (vec) {
      if constexpr (sizeof(TD) == 4) *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
      else *reinterpret_cast<uint2*>(o) = make_uint2(pack_bf2(v[0], v[1]), pack_bf2(v[2], v[3]));
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (c + k < r) st_f32<TD>(o + k, v[k]);
    }
  }
}

__global__ void __launch_bounds__(256) tc_dc_reduce_kernel(const float* part, const DcParts parts, int64_t rows,
                                                           int64_t rows_padded, int r, int rp, float lambda,
                                                           const uint32_t* hdr, float* dC,
                                                           __nv_bfloat16* dC_cast) {
  pdl_wait();
  float gscale, ginv;
  pow2_scales(hdr[kAmaxG], gscale, ginv);
  const float f = lambda * ginv;
  const int q4 = rp / 4;
  const int64_t total = rows * q4, pitch = rows_padded * q4;
  const bool vec = r == rp && ((reinterpret_cast<uintptr_t>(dC) | reinterpret_cast<uintptr_t>(dC_cast)) & 15) == 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
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

int launch_prep(PrepParams& P, cudaStream_t stream) {
  const int cgs = P.rp / 8;
  P.scan_c = P.lpc || P.lpt ? blocks_for((int64_t)P.h * P.L * P.r / 8, 2, kPlanSMs * 2) : 0;
  P.scan_g = P.g ? blocks_for(P.N * ((P.r + 7) / 8), 2, kPlanSMs * 2) : 0;
  P.blocks_c = P.lpc ? blocks_for((int64_t)P.hp * P.lpc * cgs, 2, kPlanSMs * 8) : 0;
  P.blocks_t = P.lpt ? blocks_for((int64_t)P.hp * P.lpt * cgs * P.tparts, 2, kPlanSMs * 8) : 0;
  P.blocks_g = P.g ? blocks_for(P.tiles * 128 * cgs, 2, kPlanSMs * 8) : 0;
  P.blocks_copy = 0;
  for (const CopyJob& J : P.copy)
    if (J.dst || J.act_out) P.blocks_copy = blocks_for(P.N * (P.hp / 8), 1, kPlanSMs * 16);
  tc_scan_kernel<<<(unsigned)(P.scan_c + P.scan_g), 256, 0, stream>>>(P);
  if (cudaGetLastError() != cudaSuccess) return SKV_ERR_LAUNCH;
  const unsigned grid = (unsigned)(P.blocks_c + P.blocks_t + P.blocks_g + P.blocks_copy);
  if (launch_chained<tc_pack_kernel>(dim3(grid), 256, 0, stream, P) != cudaSuccess) return SKV_ERR_LAUNCH;
  note_launches(2);
  return SKV_OK;
}

int launch_finalize(const float* partial, int splits, int64_t N, int r, int rp, float lambda, const uint32_t* hdr,
                    void* out, int64_t ds, bool out_f32, cudaStream_t stream) {
  const dim3 grid((unsigned)blocks_for(N * (rp / 4), 1, kPlanSMs * 16));
  const cudaError_t e =
      out_f32 ? launch_chained<tc_finalize_kernel<float>>(grid, 256, 0, stream, partial, splits, N, r, rp, lambda, hdr,
                                                          static_cast<float*>(out), ds)
              : launch_chained<tc_finalize_kernel<__nv_bfloat16>>(grid, 256, 0, stream, partial, splits, N, r, rp, lambda,
                                                                  hdr, static_cast<__nv_bfloat16*>(out), ds);
  note_launches(1);
  return e == cudaSuccess ? SKV_OK : SKV_ERR_LAUNCH;
}

int launch_dc_reduce(const float* part, const DcParts& parts, int64_t rows, int64_t rows_padded, int r, int rp, float lambda,
                     const uint32_t* hdr, float* dC, void* dC_cast, cudaStream_t stream) {
  const dim3 grid((unsigned)blocks_for(rows * (rp / 4), 1, kPlanSMs * 16));
  const cudaError_t e =
      launch_chained<tc_dc_reduce_kernel>(grid, 256, 0, stream, part, parts, rows, rows_padded, r, rp, lambda, hdr, dC,
                                          static_cast<__nv_bfloat16*>(dC_cast));
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
