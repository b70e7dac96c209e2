// CUDA-core kernels of the spline-KV feature operator: any N, h, L and r <= 256, bf16 or float32
// I/O, float32 arithmetic, quadratic or linear spline.  They are the float32 tier of the library, the
// path for shapes the tcgen05 kernels do not cover, and the path of the smallest forwards.
//
// They use the sparsity the tensor-core kernels cannot: a (token, key) pair touches order + 1 knot
// rows of r channels, nothing else.  A row is read with 16-byte loads by LPT neighbouring lanes, so
// a warp works on 32 / LPT tokens of one key at a time; knot interval and weights of a pair are
// computed once by one lane and handed to the LPT lanes through shared memory (a 16-byte broadcast).
//
// Every kernel of a forward or backward is chained to what was on the stream in front of it and may be resident while its inputs
// are written, so it reads them through plain pointers (skv_launch.cuh).
#include "skv_common.cuh"
#include "skv_launch.cuh"

namespace skv {
namespace {

constexpr int kWarp = 32;
constexpr unsigned kFull = 0xffffffffu;
constexpr int kWarps = 8;             // warps per CTA of the kernels below, but for staged_warps
constexpr int kGroups = 4;            // token groups a warp of the staged forward keeps accumulators for

// Warps per CTA of the kernels over a staged table, two CTAs per SM.  What a lane waits for is a chain of two shared-memory reads per
// key (weights, then rows), so warps are what hides it: sixteen where a lane's registers allow it (64 of them: float32 rows
// of up to 128 channels, and four to sixteen lanes per token, so that their staging buffers leave room for the table).
__host__ __device__ constexpr int staged_warps(int lpt, int cv, int element_bytes) {
  return element_bytes == 4 && cv == 1 && lpt >= 4 ? 16 : 8;
}

__host__ __device__ inline int64_t cdiv64(int64_t a, int64_t b) { return (a + b - 1) / b; }

// 16 bytes of a table row as float32.
template <typename T> struct Vec;
template <> struct Vec<float> {
  static constexpr int n = 4;
  static __device__ __forceinline__ void cvt(const uint4& v, float* f) {
    f[0] = __uint_as_float(v.x); f[1] = __uint_as_float(v.y); f[2] = __uint_as_float(v.z); f[3] = __uint_as_float(v.w);
  }
};
template <> struct Vec<__nv_bfloat16> {
  static constexpr int n = 8;
  static __device__ __forceinline__ void cvt(const uint4& v, float* f) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      f[2 * i] = __uint_as_float(w[i] << 16);
      f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  }
};

// Rows [0, rows) of r elements, contiguous in global memory, into shared rows of `pitch` elements.
// The pad columns are not written (the caller zeroes the buffer once).
template <typename T>
__device__ __forceinline__ void stage_rows(T* dst, const T* src, int rows, int r, int pitch) {
  if (r == pitch && (reinterpret_cast<uintptr_t>(src) & 15) == 0) {
    const int n16 = (int)((size_t)rows * r * sizeof(T) / 16);
#pragma unroll 8
    for (int i = threadIdx.x; i < n16; i += blockDim.x)
      reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(src)[i];
  } else {
    // `per` threads copy one row (the largest power of two not above r, at most a warp)
    int per = 32;
    while (per > r) per >>= 1;
    const int c0 = threadIdx.x & (per - 1);
#pragma unroll 4
    for (int row = threadIdx.x / per; row < rows; row += blockDim.x / per)
      for (int c = c0; c < r; c += per) dst[(size_t)row * pitch + c] = src[(size_t)row * r + c];
  }
}

__device__ __forceinline__ void zero16(void* p, size_t bytes) {
  for (size_t i = threadIdx.x; i < bytes / 16; i += blockDim.x) reinterpret_cast<uint4*>(p)[i] = make_uint4(0, 0, 0, 0);
}

struct FwdArgs {
  const void* z;
  int64_t zs;
  const void* C;
  void* act_out;
  int64_t as;
  void* delta_out;
  int64_t ds;
  float* partial;            // [splits][N][r], or null when one CTA covers all keys of its tokens
  int64_t N;
  int h, L, r;
  GridParams g;
  float lambda;
  int act;
  int kch;                   // staged: keys per slab; small: keys of a warp at a time, at most 32
  int keys_per_split;
  int groups;                // staged: token groups per warp (1..kGroups); small: CTAs per token
};

// Weights of one pair for the gather loop: B_0..B_2 and the element offset of row `bin`.
__device__ __forceinline__ float4 pair_weights(float zz, const GridParams& g, int key_row, int pitch) {
  const Knot k = knot_of(zz, g);
  float B0, B1, B2;
  basis_weights(k, B0, B1, B2, g.order);
  return make_float4(B0, B1, B2, __int_as_float((key_row + k.bin) * pitch));
}

// ---------------------------------------------------------------------------------------------
// Forward over a staged table: grid = (token tiles, key splits).  A CTA walks the keys of its split in
// slabs whose table rows it copies to shared memory; a warp owns `groups` groups of 32 / LPT tokens and
// keeps their residuals in registers over all slabs.
//
// Bound: shared-memory bandwidth (three rows of r channels per pair, 128 bytes a clock; 81 % of it at 4096 x 1024, r = 32, float32, 80 us;
// 58 % and 103 us with half the warps), which is why a
// bf16 table stays bf16 there.
// ---------------------------------------------------------------------------------------------
template <typename T, typename TD, int LPT, int CV>
__global__ void __launch_bounds__(staged_warps(LPT, CV, sizeof(T)) * kWarp, 2) simt_forward_kernel(const FwdArgs P) {
  constexpr int V = Vec<T>::n, W = staged_warps(LPT, CV, sizeof(T));
  constexpr int TPW = kWarp / LPT;
  constexpr int pitch = LPT * V * CV;
  constexpr int kPre = TPW < 8 ? TPW : 8;                                 // tokens of a group loaded ahead
  constexpr int kAhead = TPW * kGroups <= 8 ? kGroups : 1;                // groups loaded ahead: all where that is eight values
  extern __shared__ __align__(16) uint8_t smem_raw[];
  float4* wbuf = reinterpret_cast<float4*>(smem_raw);                     // [warp][TPW][32]
  T* Cs = reinterpret_cast<T*>(wbuf + W * TPW * kWarp);               // [kch][L][pitch]
  const int warp = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
  const int sub = lane / LPT, sl = lane % LPT;
  float4* my = wbuf + warp * TPW * kWarp;
  const T* z = static_cast<const T*>(P.z);
  T* act_out = static_cast<T*>(P.act_out);
  pdl_wait();
  pdl_launch();
  const int64_t tile0 = (int64_t)blockIdx.x * (W * TPW * P.groups);
  const int kbeg = blockIdx.y * P.keys_per_split, kend = min(P.h, kbeg + P.keys_per_split);
  const int rowstep = pitch;
  const bool three = P.g.order != 1;

  if (pitch != P.r) zero16(Cs, (size_t)P.kch * P.L * pitch * sizeof(T));
  float acc[kGroups][CV][V];
#pragma unroll
  for (int m = 0; m < kGroups; ++m)
#pragma unroll
    for (int c = 0; c < CV; ++c)
#pragma unroll
      for (int i = 0; i < V; ++i) acc[m][c][i] = 0.0f;

  for (int j0 = kbeg; j0 < kend; j0 += P.kch) {
    const int kc = min(P.kch, kend - j0);
    // rows of the first token of the group whose pre-activations are loaded next, and of the group that is worked on
    // (running pointers: as offsets of the group number the compiler would keep every group's in registers)
    const int64_t first = tile0 + (int64_t)warp * TPW;
    const T* zp = z + first * P.zs + j0 + lane;
    T* ap = act_out ? act_out + first * P.as + j0 + lane : nullptr;
    float zn[kAhead][kPre];
    auto load_z = [&](int m) {
      asm volatile("" : "+l"(zp));
      const int64_t n0 = first + (int64_t)m * (W * TPW);
#pragma unroll
      for (int t = 0; t < kPre; ++t)
        zn[m % kAhead][t] = m < P.groups && lane < kc && n0 + t < P.N ? ld_f32<T>(zp + t * P.zs) : 0.0f;
      if (kPre == TPW) zp += (int64_t)(W * TPW) * P.zs;
    };
#pragma unroll
    for (int m = 0; m < kAhead; ++m) load_z(m);
    __syncthreads();
    stage_rows(Cs, static_cast<const T*>(P.C) + (size_t)j0 * P.L * P.r, kc * P.L, P.r, pitch);
    __syncthreads();
#pragma unroll
    for (int m = 0; m < kGroups; ++m) {
      if (m >= P.groups) break;
      const int64_t n0 = first + (int64_t)m * (W * TPW);
      if (n0 >= P.N) break;
      asm volatile("" : "+l"(ap));
      __syncwarp();
#pragma unroll
      for (int t = 0; t < TPW; ++t) {
        float4 w = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (lane < kc && n0 + t < P.N) {
          const float zz = t < kPre ? zn[m % kAhead][t < kPre ? t : 0] : ld_f32<T>(zp + t * P.zs);
          w = pair_weights(zz, P.g, lane * P.L, pitch);
          if (act_out) st_f32<T>(ap + t * P.as, act_fwd(zz, P.act));
        }
        my[t * kWarp + lane] = w;
      }
      if (kPre < TPW) zp += (int64_t)(W * TPW) * P.zs;
      if (act_out) ap += (int64_t)(W * TPW) * P.as;
      if (kAhead < kGroups) load_z(m + kAhead);       // the next group's pre-activations are requested now
      __syncwarp();
#pragma unroll 2
      for (int q = 0; q < kc; ++q) {
        const float4 w = my[sub * kWarp + q];
        const T* row = Cs + __float_as_int(w.w) + sl * V;
#pragma unroll
        for (int c = 0; c < CV; ++c) {
          const T* rc = row + c * (LPT * V);
          float f0[V], f1[V], f2[V];
          Vec<T>::cvt(*reinterpret_cast<const uint4*>(rc), f0);
          Vec<T>::cvt(*reinterpret_cast<const uint4*>(rc + rowstep), f1);
#pragma unroll
          for (int i = 0; i < V; ++i) acc[m][c][i] = fmaf(w.y, f1[i], fmaf(w.x, f0[i], acc[m][c][i]));
          if (three) {
            Vec<T>::cvt(*reinterpret_cast<const uint4*>(rc + 2 * rowstep), f2);
#pragma unroll
            for (int i = 0; i < V; ++i) acc[m][c][i] = fmaf(w.z, f2[i], acc[m][c][i]);
          }
        }
      }
    }
  }
#pragma unroll
  for (int m = 0; m < kGroups; ++m) {
    if (m >= P.groups) break;
    const int64_t n = tile0 + (int64_t)(m * W + warp) * TPW + sub;
    if (n >= P.N) continue;
#pragma unroll
    for (int c = 0; c < CV; ++c)
#pragma unroll
      for (int i = 0; i < V; ++i) {
        const int col = c * (LPT * V) + sl * V + i;
        if (col < P.r) {
          if (P.partial) P.partial[((size_t)blockIdx.y * P.N + n) * P.r + col] = acc[m][c][i];
          else st_f32<TD>(static_cast<TD*>(P.delta_out) + n * P.ds + col, P.lambda * acc[m][c][i]);
        }
      }
  }
}

// ---------------------------------------------------------------------------------------------
// Forward that reads the table rows where they are: a cluster of CTAs takes a token, each CTA a share of its keys, a warp up
// to 32 of them at a time.  For few tokens most of the table is never touched, so nothing is copied or packed first.
// 32 / LPT keys of a warp are worked on at once; the lane groups', the warps' and the CTAs' sums are added in a fixed order,
// the last of them through the shared memory of the cluster's first CTA.  Also the path of a table too large per key
// for shared memory.
//
// Bound: the latency of one dependent chain (z -> knot -> row -> sums), so the keys of a token are spread over as many
// warps as the chip holds and four rows' loads are in flight per lane; then, from about 64 tokens at h = 5120 on, by what
// L2 delivers (three rows per pair).
// ---------------------------------------------------------------------------------------------
// 16 bytes of a row at element `col`, as one load or (BYTES 8) two, where rows start on such boundaries; 0: element by element.
template <typename T, int BYTES>
__device__ __forceinline__ void load_row(const T* row, int col, int r, float (&f)[Vec<T>::n]) {
  if constexpr (BYTES == 16) {
    Vec<T>::cvt(*reinterpret_cast<const uint4*>(row + col), f);
  } else if constexpr (BYTES == 8) {
    const uint2 a = *reinterpret_cast<const uint2*>(row + col);
    const uint2 b = col + Vec<T>::n / 2 < r ? reinterpret_cast<const uint2*>(row + col)[1] : make_uint2(0, 0);
    Vec<T>::cvt(make_uint4(a.x, a.y, b.x, b.y), f);
  } else {
#pragma unroll
    for (int i = 0; i < Vec<T>::n; ++i) f[i] = col + i < r ? ld_f32<T>(row + col + i) : 0.0f;
  }
}

constexpr int kSmallWarps = 32;       // most warps of a CTA
constexpr int kSmallCluster = 8;      // most CTAs of a token

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// One float32 into the shared memory of the cluster's first CTA, at the place `p` has in this one's.
__device__ __forceinline__ void store_first_cta(float* p, float v) {
  uint32_t a = (uint32_t)__cvta_generic_to_shared(p), b;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(b) : "r"(a));
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(b), "f"(v) : "memory");
}

template <typename T, typename TD, int LPT, int CV, int BYTES>
__global__ void __launch_bounds__(kSmallWarps * kWarp, 1) simt_forward_small_kernel(const FwdArgs P) {
  constexpr int V = Vec<T>::n;
  constexpr int TPW = kWarp / LPT;
  constexpr int pitch = LPT * V * CV;
  extern __shared__ __align__(16) uint8_t smem_raw[];
  const int W = blockDim.x / kWarp, cs = P.groups;
  float* parts = reinterpret_cast<float*>(smem_raw);                       // [kSmallCluster][pitch], of the first CTA
  float* red = parts + kSmallCluster * pitch;                              // [warp][pitch], in the place of
  float4* wbuf = reinterpret_cast<float4*>(red);                           // [warp][32]
  const int warp = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
  const int sub = lane / LPT, sl = lane % LPT, rank = blockIdx.x % cs;
  const T* z = static_cast<const T*>(P.z);
  const T* C = static_cast<const T*>(P.C);
  T* act_out = static_cast<T*>(P.act_out);
  const int kbeg = rank * P.keys_per_split, kend = min(P.h, kbeg + P.keys_per_split);
  const bool three = P.g.order != 1;
  float4* my = wbuf + warp * kWarp;
  pdl_wait();
  pdl_launch();
  if (cs > 1) cluster_arrive();                       // the first CTA has started before anything is sent to it

  for (int64_t n = blockIdx.x / cs; n < P.N; n += gridDim.x / cs) {
    float acc[CV][V];
#pragma unroll
    for (int c = 0; c < CV; ++c)
#pragma unroll
      for (int i = 0; i < V; ++i) acc[c][i] = 0.0f;
    const T* zr = z + n * P.zs;
    float znext = 0.0f;
    const int kw = P.kch;
    int j0 = kbeg + warp * kw;
    if (lane < kw && j0 + lane < kend) znext = ld_f32<T>(zr + j0 + lane);
    for (; j0 < kend; j0 += W * kw) {
      const int kc = min(kw, kend - j0);
      const float zz = znext;
      if (lane < kw && j0 + W * kw + lane < kend) znext = ld_f32<T>(zr + j0 + W * kw + lane);
      __syncwarp();
      if (lane < kc) {
        my[lane] = pair_weights(zz, P.g, lane * P.L, P.r);
        if (act_out) st_f32<T>(act_out + n * P.as + j0 + lane, act_fwd(zz, P.act));
      }
      __syncwarp();
      const T* base = C + (size_t)j0 * P.L * P.r;
#pragma unroll 4
      for (int q = sub; q < kc; q += TPW) {
        const float4 w = my[q];
        const T* row = base + __float_as_int(w.w);
#pragma unroll
        for (int c = 0; c < CV; ++c) {
          const int col = c * (LPT * V) + sl * V;
          if (col < P.r) {
            float f0[V], f1[V], f2[V];
            load_row<T, BYTES>(row, col, P.r, f0);
            load_row<T, BYTES>(row + P.r, col, P.r, f1);
            if (three) load_row<T, BYTES>(row + 2 * P.r, col, P.r, f2);
#pragma unroll
            for (int i = 0; i < V; ++i) {
              acc[c][i] = fmaf(w.y, f1[i], fmaf(w.x, f0[i], acc[c][i]));
              if (three) acc[c][i] = fmaf(w.z, f2[i], acc[c][i]);
            }
          }
        }
      }
    }
#pragma unroll
    for (int s = LPT; s < kWarp; s <<= 1) {
#pragma unroll
      for (int c = 0; c < CV; ++c)
#pragma unroll
        for (int i = 0; i < V; ++i) acc[c][i] += __shfl_xor_sync(kFull, acc[c][i], s);
    }
    __syncthreads();
    if (sub == 0) {
#pragma unroll
      for (int c = 0; c < CV; ++c)
#pragma unroll
        for (int i = 0; i < V; ++i) red[(size_t)warp * pitch + c * (LPT * V) + sl * V + i] = acc[c][i];
    }
    __syncthreads();
    if (cs > 1) cluster_wait();                       // the first CTA is there and has read what it was sent last
    for (int col = threadIdx.x; col < P.r; col += blockDim.x) {
      float s = 0.0f;
#pragma unroll 8
      for (int w = 0; w < W; ++w) s += red[(size_t)w * pitch + col];
      if (cs > 1) store_first_cta(parts + rank * pitch + col, s);
      else st_f32<TD>(static_cast<TD*>(P.delta_out) + n * P.ds + col, P.lambda * s);
    }
    if (cs > 1) {
      __syncwarp();
      cluster_arrive();
      cluster_wait();
      if (rank == 0) {
        for (int col = threadIdx.x; col < P.r; col += blockDim.x) {
          float s = 0.0f;
          for (int k = 0; k < cs; ++k) s += parts[k * pitch + col];
          st_f32<TD>(static_cast<TD*>(P.delta_out) + n * P.ds + col, P.lambda * s);
        }
      }
      __syncwarp();
      cluster_arrive();
    }
    __syncthreads();                                  // the sums have been read
  }
  if (cs > 1) cluster_wait();
}

// Sum of the key splits' partial residuals in a fixed order, lambda, cast.  A CTA takes 32 times Q neighbouring elements;
// its eight warps each add every eighth split, so that a sum over many splits is not one serial chain.  Q = 4 where r allows it
// (4096 x 32 elements, 18 splits: 8.3 us element by element; a step of 4096 x 1024 takes 2.5 us less with fours).
template <typename TD, int Q>
__global__ void __launch_bounds__(256) simt_finalize_kernel(const float* partial, int splits, int64_t N, int r, float lambda, TD* out,
                                                            int64_t ds) {
  __shared__ float part[8][kWarp][Q];
  pdl_wait();
  pdl_launch();
  const int warp = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
  const int64_t total = N * r;
  for (int64_t b = (int64_t)blockIdx.x * (kWarp * Q); b < total; b += (int64_t)gridDim.x * (kWarp * Q)) {
    const int64_t i = b + lane * Q;
    float s[Q] = {};
    if (i < total) {
#pragma unroll 4
      for (int k = warp; k < splits; k += 8) {
        const float* src = partial + (size_t)k * total + i;
        if constexpr (Q == 4) {
          const float4 v = *reinterpret_cast<const float4*>(src);
          s[0] += v.x; s[1] += v.y; s[2] += v.z; s[3] += v.w;
        } else {
          s[0] += *src;
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < Q; ++q) part[warp][lane][q] = s[q];
    __syncthreads();
    // element `warp` of a lane's (of its only one the first warp takes care)
    if (warp < Q && i < total) {
      float sum = 0.0f;
#pragma unroll
      for (int w = 0; w < 8; ++w) sum += part[w][lane][warp];
      const int64_t e = i + warp;
      st_f32<TD>(out + (e / r) * ds + (e % r), lambda * sum);
    }
  }
}

// ---------------------------------------------------------------------------------------------
// dz: grid = (token tiles, key slabs).  The derivative of the quadratic spline is linear between the knots,
//     sum_k B_k' C[bin + k] = (1 - tau) D[bin] + tau D[bin + 1],   D[b] = C[b + 1] - C[b]
// (the linear spline: D[bin] alone), so the slab is staged as its differences D in float32 and a pair
// reads two rows instead of three.  The lanes of a token hold partial sums of eight keys and one
// transpose-reduce turns them into one key's sum per lane; 32 keys' results go through shared memory so
// that z, g_act and dz are read and written by whole rows of 32 keys.
//
// Bound: shared-memory latency and bandwidth, two float32 rows of r channels per pair (52 % of it with 27 warps per SM; 4096 x 1024, r = 32:
// 84 us, 103 with half the warps).
// ---------------------------------------------------------------------------------------------
struct DzArgs {
  const void* z;
  int64_t zs;
  const void* C;
  const void* g_act;
  int64_t gas;
  const void* g_delta;
  int64_t gds;
  void* dz;
  int64_t dzs;
  int64_t N;
  int h, L, r;
  GridParams g;
  float coef;                // lambda * scale
  int act;
  int kch;                   // keys per slab, at most 32
  int groups;                // token groups per warp
};

// STAGED = false: a key's differences do not fit shared memory; they are formed from the table itself.
template <typename T, int LPT, int CV, bool STAGED>
__global__ void __launch_bounds__(staged_warps(LPT, CV, 4) * kWarp, 2) simt_dz_kernel(const DzArgs P) {
  constexpr int V = 4, W = staged_warps(LPT, CV, 4);
  constexpr int Q = LPT < 8 ? LPT : 8;                                     // keys of a transpose
  constexpr int TPW = kWarp / LPT;
  constexpr int pitch = LPT * V * CV;
  constexpr int kPre = TPW < 8 ? TPW : 8;                                  // tokens of the next group loaded ahead
  constexpr int kRes = kWarp + 4;                                          // pitch of the result rows
  extern __shared__ __align__(16) uint8_t smem_raw[];
  float2* wbuf = reinterpret_cast<float2*>(smem_raw);                     // [warp][TPW][32]  (tau, row offset)
  float* rbuf = reinterpret_cast<float*>(wbuf + W * TPW * kWarp);     // [warp][TPW][kRes]
  float* Ds = rbuf + W * TPW * kRes;                                  // [kch][rows][pitch]
  const int warp = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
  const int sub = lane / LPT, sl = lane % LPT;
  float2* my = wbuf + warp * TPW * kWarp;
  float* res = rbuf + warp * TPW * kRes;
  const T* z = static_cast<const T*>(P.z);
  const T* C = static_cast<const T*>(P.C);
  const T* g_act = static_cast<const T*>(P.g_act);
  const T* g_delta = static_cast<const T*>(P.g_delta);
  T* dz = static_cast<T*>(P.dz);
  const bool two = P.g.order != 1;
  const int R = P.L - 1;                                                   // difference rows per key
  pdl_wait();
  pdl_launch();
  const int64_t tile0 = (int64_t)blockIdx.x * (W * TPW * P.groups);
  const int j0 = blockIdx.y * P.kch, kc = min(P.kch, P.h - j0);

  if constexpr (STAGED) {
    int per = 32;
    while (per > P.r) per >>= 1;
    const int c0 = threadIdx.x & (per - 1);
#pragma unroll 4
    for (int row = threadIdx.x / per; row < kc * R; row += blockDim.x / per) {
      const T* src = C + ((size_t)(j0 + row / R) * P.L + row % R) * P.r;
      for (int c = c0; c < pitch; c += per)
        Ds[(size_t)row * pitch + c] = c < P.r ? ld_f32<T>(src + P.r + c) - ld_f32<T>(src + c) : 0.0f;
    }
  }
  __syncthreads();

  // rows of z, g_delta and g_act of the next group are requested while this one is worked on
  float zn[kPre], an[kPre], gn[CV][V];
  auto load_group = [&](int m) {
    const int64_t n0 = tile0 + (int64_t)(m * W + warp) * TPW;
    const bool on = m < P.groups && lane < kc;
#pragma unroll
    for (int t = 0; t < kPre; ++t) {
      zn[t] = on && n0 + t < P.N ? ld_f32<T>(z + (n0 + t) * P.zs + j0 + lane) : 0.0f;
      an[t] = on && g_act && n0 + t < P.N ? ld_f32<T>(g_act + (n0 + t) * P.gas + j0 + lane) : 0.0f;
    }
#pragma unroll
    for (int c = 0; c < CV; ++c)
#pragma unroll
      for (int i = 0; i < V; ++i) {
        const int col = c * (LPT * V) + sl * V + i;
        gn[c][i] = m < P.groups && n0 + sub < P.N && col < P.r ? ld_f32<T>(g_delta + (n0 + sub) * P.gds + col) : 0.0f;
      }
  };
  load_group(0);
  for (int m = 0; m < P.groups; ++m) {
    const int64_t n0 = tile0 + (int64_t)(m * W + warp) * TPW;
    if (n0 >= P.N) break;
    float zz[TPW], ga[kPre];
    float gd[CV][V];
#pragma unroll
    for (int t = 0; t < TPW; ++t)
      zz[t] = t < kPre ? zn[t < kPre ? t : 0]
                       : (lane < kc && n0 + t < P.N ? ld_f32<T>(z + (n0 + t) * P.zs + j0 + lane) : 0.0f);
#pragma unroll
    for (int t = 0; t < kPre; ++t) ga[t] = an[t];
#pragma unroll
    for (int c = 0; c < CV; ++c)
#pragma unroll
      for (int i = 0; i < V; ++i) gd[c][i] = gn[c][i];
    load_group(m + 1);
    uint32_t live = 0u;                                                    // bit t: 0 <= u <= G-1 for (t, lane)
#pragma unroll
    for (int t = 0; t < TPW; ++t) {
      float2 w = make_float2(0.0f, 0.0f);
      if (lane < kc && n0 + t < P.N) {
        const Knot k = knot_of(zz[t], P.g);
        w = make_float2(k.tau, __int_as_float(STAGED ? (lane * R + k.bin) * pitch : (lane * P.L + k.bin) * P.r));
        if (k.clamp_active) live |= 1u << t;
      }
      my[t * kWarp + lane] = w;
    }
    __syncwarp();
#pragma unroll 1
    for (int q0 = 0; q0 < kc; q0 += Q) {
      float v[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const float2 w = my[sub * kWarp + q0 + q];                          // keys past kc: row 0, result unused
        float s = 0.0f;
#pragma unroll
        for (int c = 0; c < CV; ++c) {
          float d[V], e[V];
          if constexpr (STAGED) {
            const float* row = Ds + __float_as_int(w.y) + sl * V + c * (LPT * V);
            const float4 a = *reinterpret_cast<const float4*>(row);
            d[0] = a.x; d[1] = a.y; d[2] = a.z; d[3] = a.w;
            if (two) {
              const float4 b = *reinterpret_cast<const float4*>(row + pitch);
              e[0] = b.x; e[1] = b.y; e[2] = b.z; e[3] = b.w;
            }
          } else {
            const T* row = C + (size_t)j0 * P.L * P.r + __float_as_int(w.y);
#pragma unroll
            for (int i = 0; i < V; ++i) {
              const int col = c * (LPT * V) + sl * V + i;
              const float c1 = col < P.r ? ld_f32<T>(row + P.r + col) : 0.0f;
              d[i] = col < P.r ? c1 - ld_f32<T>(row + col) : 0.0f;
              e[i] = two && col < P.r ? ld_f32<T>(row + 2 * P.r + col) - c1 : 0.0f;
            }
          }
          // (interpolated before the product: adjacent differences cancel, and the two products' roundings would not)
          if (two) {
#pragma unroll
            for (int i = 0; i < V; ++i) d[i] = fmaf(w.x, e[i] - d[i], d[i]);
          }
#pragma unroll
          for (int i = 0; i < V; ++i) s = fmaf(gd[c][i], d[i], s);
        }
        v[q] = s;
      }
      // afterwards v[0] of lane sl is the sum over the token's lanes of v[sl % Q]
#pragma unroll
      for (int s = Q / 2; s >= 1; s >>= 1) {
#pragma unroll
        for (int i = 0; i < s; ++i) {
          const bool up = (sl & s) != 0;
          const float send = up ? v[i] : v[i + s];
          const float keep = up ? v[i + s] : v[i];
          v[i] = keep + __shfl_xor_sync(kFull, send, s);
        }
      }
#pragma unroll
      for (int s = Q; s < LPT; s <<= 1) v[0] += __shfl_xor_sync(kFull, v[0], s);
      if (sl < Q) res[sub * kRes + q0 + sl] = v[0];
    }
    __syncwarp();
#pragma unroll
    for (int t = 0; t < TPW; ++t) {
      if (lane < kc && n0 + t < P.N) {
        float o = (live >> t) & 1u ? P.coef * res[t * kRes + lane] : 0.0f;
        if (g_act)
          o = fmaf(t < kPre ? ga[t < kPre ? t : 0] : ld_f32<T>(g_act + (n0 + t) * P.gas + j0 + lane), act_grad(zz[t], P.act), o);
        st_f32<T>(dz + (n0 + t) * P.dzs + j0 + lane, o);
      }
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------------------------
// dC: grid = (key groups, token splits), one warp per key.  A tile of up to 256 tokens is staged (g rows in
// float32 and the CTA's columns of z); the warp sorts the tile's tokens by knot interval (a counting sort
// over warp votes, so the order, and with it the result, is always the same) and walks the intervals: the
// rows of an interval are summed in registers over all of its tokens, in a window that slides from interval to
// interval and adds one finished row to the key's accumulator each time, where adding every token to its rows would
// read and write three rows of shared memory for each.  Tokens outside the grid have no weight and leave the lists.
//
// Bound: latencies and instruction issue (66 % of the slots with 21 warps per SM): at 4096 x 1024, r = 32, the products of the rows
// take 49 us of 104, the walk over the intervals and the finished rows 28, staging and the sort 27.  With eight warps per CTA, two
// CTAs per SM, no request ahead and a full reduction per finished row it took 173.
// ---------------------------------------------------------------------------------------------
struct DcArgs {
  const void* z;
  int64_t zs;
  const void* g_delta;
  int64_t gds;
  float* part;               // [splits][h][L][r]; null: the sums are final and go to dC / dC_cast
  float* dC;
  void* dC_cast;
  int64_t N;
  int h, L, r;
  GridParams g;
  float lambda;
  int TT;                    // tokens per tile, a multiple of 32
  int64_t tokens_per_split;
  bool first;                // the first kernel of a call; else it runs beside dz, which it has nothing to wait for
};

constexpr int kMaxTile = 256;
constexpr int kDcMaxWarps = 24;
constexpr int kDcAhead = 4;                // pieces of four gradients that a thread requests before a tile is worked on

// Four neighbouring elements, aligned.
template <typename T> struct Quad;
template <> struct Quad<float> {
  float4 v;
  __device__ __forceinline__ void load(const float* p) { v = *reinterpret_cast<const float4*>(p); }
  __device__ __forceinline__ float4 get() const { return v; }
};
template <> struct Quad<__nv_bfloat16> {
  uint2 v;
  __device__ __forceinline__ void load(const __nv_bfloat16* p) { v = *reinterpret_cast<const uint2*>(p); }
  __device__ __forceinline__ float4 get() const {
    return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16),
                       __uint_as_float(v.y & 0xffff0000u));
  }
};

// GACC = true: a key's accumulator does not fit shared memory and lives in the partial buffer.
template <typename T, int LPT, int CV, bool GACC>
__global__ void __launch_bounds__(kDcMaxWarps * kWarp, 1) simt_dc_kernel(const DcArgs P) {
  constexpr int V = 4;
  constexpr int S = kWarp / LPT;
  constexpr int pitch = LPT * V * CV;
  constexpr int kPer = kMaxTile / kWarp;                                   // tokens of a tile per lane, at most
  extern __shared__ __align__(16) uint8_t smem_raw[];
  const int W = blockDim.x / kWarp, TT = P.TT, nb = P.L - P.g.order, r = P.r;
  const int zp = W | 1;                                                    // odd: a column of z has no bank conflicts
  float* gs = reinterpret_cast<float*>(smem_raw);                          // [TT][pitch]
  float4* ent_all = reinterpret_cast<float4*>(gs + (size_t)TT * pitch);    // [W][TT]  (w0, w1, w2, offset of the token's row)
  float* acc_all = reinterpret_cast<float*>(ent_all + (size_t)W * TT);     // [W][L][pitch] unless GACC
  float* zt = acc_all + (GACC ? 0 : (size_t)W * P.L * pitch);              // [TT][zp]
  int* off_all = reinterpret_cast<int*>(zt + (size_t)TT * zp);             // [W][nb + 1]
  const int warp = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
  const int sub = lane / LPT, sl = lane % LPT;
  const int j0 = blockIdx.x * W, kd = min(W, P.h - j0);
  const int64_t nbeg = (int64_t)blockIdx.y * P.tokens_per_split, nend = min(P.N, nbeg + P.tokens_per_split);
  const T* z = static_cast<const T*>(P.z);
  const T* g_delta = static_cast<const T*>(P.g_delta);
  const bool three = P.g.order != 1;
  const bool mine = warp < kd;
  float4* ent = ent_all + (size_t)warp * TT;
  int* off = off_all + warp * (nb + 1);
  float* acc = GACC ? P.part + (((size_t)blockIdx.y * P.h + j0 + (mine ? warp : 0)) * P.L) * r
                    : acc_all + (size_t)warp * P.L * pitch;
  const int ap = GACC ? r : pitch;

  if (P.first) pdl_wait();
  pdl_launch();
  if constexpr (GACC) {
    if (mine)
      for (int i = lane; i < P.L * r; i += kWarp) acc[i] = 0.0f;
  } else {
    zero16(acc_all, (size_t)W * P.L * pitch * sizeof(float));
  }
  if (r != pitch) zero16(gs, (size_t)TT * pitch * sizeof(float));

  // A tile's gradients and pre-activations are requested before the tile in front of it is worked on: the first
  // kDcAhead pieces of four gradients of every thread, and one column of z per thread.
  const bool quads = r % 4 == 0 && P.gds % 4 == 0 && (reinterpret_cast<uintptr_t>(g_delta) & (4 * sizeof(T) - 1)) == 0;
  const int rq = r / 4, zk = threadIdx.x % W, zt0 = threadIdx.x / W;       // a thread's key and first token of z: every 32nd
  Quad<T> gn[kDcAhead];
  float zn[kPer];
  auto request = [&](int64_t t0) {
    const int tt = (int)min((int64_t)TT, nend - t0);
    if (quads) {
#pragma unroll
      for (int i = 0; i < kDcAhead; ++i) {
        const int e = threadIdx.x + i * blockDim.x, t = e / rq;
        if (t < tt) gn[i].load(g_delta + (t0 + t) * P.gds + (e - t * rq) * 4);
      }
    }
    const T* src = z + (t0 + zt0) * P.zs + j0 + zk;
#pragma unroll
    for (int i = 0; i < kPer; ++i)
      zn[i] = zt0 + i * kWarp < tt && zk < kd ? ld_f32<T>(src + (int64_t)(i * kWarp) * P.zs) : 0.0f;
  };
  request(nbeg);

  for (int64_t t0 = nbeg; t0 < nend; t0 += TT) {
    const int tt = (int)min((int64_t)TT, nend - t0);
    __syncthreads();
    if (quads) {
#pragma unroll
      for (int i = 0; i < kDcAhead; ++i) {
        const int e = threadIdx.x + i * blockDim.x, t = e / rq;
        if (t < tt) *reinterpret_cast<float4*>(gs + (size_t)t * pitch + (e - t * rq) * 4) = gn[i].get();
      }
      for (int e = threadIdx.x + kDcAhead * blockDim.x; e < tt * rq; e += blockDim.x) {
        const int t = e / rq;
        Quad<T> q;
        q.load(g_delta + (t0 + t) * P.gds + (e - t * rq) * 4);
        *reinterpret_cast<float4*>(gs + (size_t)t * pitch + (e - t * rq) * 4) = q.get();
      }
    } else {
      for (int e = threadIdx.x; e < tt * r; e += blockDim.x) {
        const int t = e / r, c = e - t * r;
        gs[(size_t)t * pitch + c] = ld_f32<T>(g_delta + (t0 + t) * P.gds + c);
      }
    }
#pragma unroll
    for (int i = 0; i < kPer; ++i)
      if (zt0 + i * kWarp < tt) zt[(zt0 + i * kWarp) * zp + zk] = zn[i];
    for (int i = lane; i <= nb; i += kWarp) off[i] = 0;
    __syncthreads();
    if (t0 + TT < nend) request(t0 + TT);
    if (!mine) continue;

    // ---- rank of every token within its interval, counts per interval
    int bins[kPer], pos[kPer];
    float tau[kPer];
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      bins[i] = -1;
      if (i * kWarp < tt) {
        const int t = i * kWarp + lane;
        if (t < tt) {
          const Knot k = knot_of(zt[t * zp + warp], P.g);
          tau[i] = k.tau;
          if (k.in_range) bins[i] = k.bin;
        }
        const unsigned same = __match_any_sync(kFull, bins[i]);
        const int rank = __popc(same & ((1u << lane) - 1u));
        const int base = bins[i] >= 0 ? off[bins[i]] : 0;
        __syncwarp();
        if (bins[i] >= 0 && rank == 0) off[bins[i]] = base + __popc(same);
        __syncwarp();
        pos[i] = base + rank;
      }
    }
    // ---- counts -> first entry of each interval (off[nb] = number of entries)
    int carry = 0;
    for (int b0 = 0; b0 <= nb; b0 += kWarp) {
      const int b = b0 + lane;
      const int c = b < nb ? off[b] : 0;
      int x = c;
#pragma unroll
      for (int s = 1; s < kWarp; s <<= 1) {
        const int y = __shfl_up_sync(kFull, x, s);
        if (lane >= s) x += y;
      }
      if (b <= nb) off[b] = carry + x - c;
      carry += __shfl_sync(kFull, x, kWarp - 1);
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      if (bins[i] >= 0) {
        Knot k;
        k.tau = tau[i];
        k.in_range = true;
        float B0, B1, B2;
        basis_weights(k, B0, B1, B2, P.g.order);
        ent[off[bins[i]] + pos[i]] = make_float4(B0, B1, B2, __int_as_float((i * kWarp + lane) * pitch));
      }
    }
    __syncwarp();
    // ---- one interval at a time; the window of rows b, b + 1, b + 2 slides along, so each interval finishes one row.  The
    // three sums take the three places in turn (the loop is unrolled by three) instead of moving.
    float a[3][CV][V];
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int c = 0; c < CV; ++c)
#pragma unroll
        for (int i = 0; i < V; ++i) a[k][c][i] = 0.0f;
    auto finish_row = [&](float (&w)[CV][V], int row) {  // a finished sum goes to the key's accumulator, its place is free
#pragma unroll
      for (int c = 0; c < CV; ++c) {
        // the lane groups' sums are added while the channels are shared out among them: V -> V / 2 -> 1 per lane
        int col = sl * V + c * (LPT * V), n = V;
        bool write = true;
#pragma unroll
        for (int s = S / 2; s >= 1; s >>= 1) {
          const bool up = (sub & s) != 0;
          if (n > 1) {
            n /= 2;
#pragma unroll
            for (int i = 0; i < V / 2; ++i) {
              if (i >= n) continue;
              const float send = up ? w[c][i] : w[c][i + n], keep = up ? w[c][i + n] : w[c][i];
              w[c][i] = keep + __shfl_xor_sync(kFull, send, s * LPT);
            }
            if (up) col += n;
          } else {
            w[c][0] += __shfl_xor_sync(kFull, w[c][0], s * LPT);
            write = write && !up;
          }
        }
        float* dst = acc + (size_t)row * ap + col;
        if (write) {
          if constexpr (S == 1 && !GACC) {
            float4 d = *reinterpret_cast<float4*>(dst);
            d.x += w[c][0]; d.y += w[c][1]; d.z += w[c][2]; d.w += w[c][3];
            *reinterpret_cast<float4*>(dst) = d;
          } else {
#pragma unroll
            for (int i = 0; i < V; ++i)
              if (i < n && (!GACC || col + i < r)) dst[i] += w[c][i];
          }
        }
#pragma unroll
        for (int i = 0; i < V; ++i) w[c][i] = 0.0f;
      }
    };
    int end = off[0], dirty = 0;                      // rows of the window that hold something
    auto interval = [&](int b, float (&w0)[CV][V], float (&w1)[CV][V], float (&w2)[CV][V]) {
      const int beg = end;
      end = off[b + 1];
      if (beg != end) {
        dirty = 3;
#pragma unroll 2
        for (int p = beg + sub; p < end; p += S) {
          const float4 e = ent[p];
          const float* gr = gs + __float_as_int(e.w) + sl * V;
#pragma unroll
          for (int c = 0; c < CV; ++c) {
            const float4 g4 = *reinterpret_cast<const float4*>(gr + c * (LPT * V));
            const float gv[V] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
            for (int i = 0; i < V; ++i) {
              w0[c][i] = fmaf(e.x, gv[i], w0[c][i]);
              w1[c][i] = fmaf(e.y, gv[i], w1[c][i]);
            }
            if (three) {                               // (a third weight of zero times an infinity is not zero)
#pragma unroll
              for (int i = 0; i < V; ++i) w2[c][i] = fmaf(e.z, gv[i], w2[c][i]);
            }
          }
        }
      }
      if (dirty > 0) { finish_row(w0, b); --dirty; }
    };
    int b = 0;
    for (; b + 3 <= nb; b += 3) {
      interval(b, a[0], a[1], a[2]);
      interval(b + 1, a[1], a[2], a[0]);
      interval(b + 2, a[2], a[0], a[1]);
    }
    if (nb - b == 1) {
      interval(b, a[0], a[1], a[2]);
      if (dirty > 0) finish_row(a[1], nb);
      if (three && dirty > 1) finish_row(a[2], nb + 1);
    } else if (nb - b == 2) {
      interval(b, a[0], a[1], a[2]);
      interval(b + 1, a[1], a[2], a[0]);
      if (dirty > 0) finish_row(a[2], nb);
      if (three && dirty > 1) finish_row(a[0], nb + 1);
    } else {
      if (dirty > 0) finish_row(a[0], nb);
      if (three && dirty > 1) finish_row(a[1], nb + 1);
    }
    __syncwarp();
  }
  if (!P.first) pdl_wait();                            // whoever waits for this kernel has waited for dz
  __syncthreads();
  if (!mine) return;
  const size_t row0 = (size_t)(j0 + warp) * P.L;
  if (P.part) {
    if constexpr (!GACC) {
      float* dst = P.part + ((size_t)blockIdx.y * P.h * P.L + row0) * r;
      for (int i = lane; i < P.L * r; i += kWarp) dst[i] = acc[(size_t)(i / r) * pitch + i % r];
    }
  } else {
    for (int i = lane; i < P.L * r; i += kWarp) {
      const float v = P.lambda * acc[(size_t)(i / r) * pitch + i % r];
      if (P.dC) P.dC[row0 * r + i] = v;
      if (P.dC_cast) st_f32<T>(static_cast<T*>(P.dC_cast) + row0 * r + i, v);
    }
  }
}

template <typename T>
__global__ void simt_dc_reduce_kernel(const float* part, int splits, size_t elems, float lambda, float* dC, T* dC_cast) {
  pdl_wait();
  pdl_launch();
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < elems; i += (size_t)gridDim.x * blockDim.x) {
    float s = 0.0f;
#pragma unroll 4
    for (int k = 0; k < splits; ++k) s += part[(size_t)k * elems + i];
    s *= lambda;
    if (dC) dC[i] = s;
    if (dC_cast) st_f32<T>(dC_cast + i, s);
  }
}

template <typename T>
__global__ void simt_knot_index_kernel(const T* __restrict__ z, int64_t zs, int64_t N, int h, GridParams g,
                                       int32_t* __restrict__ bins) {
  const int64_t total = N * (int64_t)h;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t n = i / h;
    const int j = (int)(i % h);
    bins[i] = knot_of(ld_f32<T>(z + n * zs + j), g).bin;
  }
}

// =================================================================================================
// plans and launches
// =================================================================================================
constexpr int kPlanSMs = 148;                            // B200; only used to balance launch shapes
constexpr size_t kSmemHalf = 110 * 1024;                 // two CTAs per SM
constexpr size_t kSmemFull = 216 * 1024;
constexpr size_t kSmemMost = 226 * 1024;
constexpr size_t kFwdScratchCap = SKV_NOALLOC_SCRATCH_BYTES;   // the key splits' partials stay below this

// Lanes per token (a power of two from 2 to 32) and 16-byte pieces per lane for rows of r elements.
void lanes_for(int r, int v, int* lpt, int* cv) {
  int l = 2;
  while (l < 32 && l * v < r) l <<= 1;
  *lpt = l;
  *cv = l * v < r ? 2 : 1;
}

struct FwdPlan { bool small; int lpt, cv, warps, kch, groups, splits, keys_per_split; int64_t tiles; size_t smem; };

FwdPlan make_forward_plan(const skv_problem& p) {
  FwdPlan f;
  const int size = p.dtype == SKV_BF16 ? 2 : 4, v = 16 / size;
  lanes_for(p.r, v, &f.lpt, &f.cv);
  const int tpw = kWarp / f.lpt, pitch = f.lpt * v * f.cv;
  const int64_t N = p.N > 0 ? p.N : 1;
  const int warps = staged_warps(f.lpt, f.cv, size);
  const size_t wb = (size_t)warps * tpw * kWarp * 16, per_key = (size_t)p.L * pitch * size;
  size_t most_keys = kSmemHalf > wb ? (kSmemHalf - wb) / per_key : 0;
  if (most_keys < 8) most_keys = (kSmemFull - wb) / per_key;
  if (most_keys > 32) most_keys = 32;
  f.kch = (int)most_keys;
  f.warps = warps;
  f.small = f.kch < 1 || N <= small_forward_tokens(p);
  const size_t part_bytes = (size_t)N * p.r * sizeof(float);
  f.splits = 1;
  if (f.small) {
    // CTAs of a token, warps of a CTA and keys of a warp's pass.  Microseconds: a pass is a chain of latencies, one more for
    // every 32 / LPT keys, or what an SM takes from L2 (60 KB; it holds 32 of these warps); launch, sums, and the
    // cluster's exchange.  A cluster lives within a GPC, so large ones do not fill the chip.
    double best = 0.0;
    for (int cs = kSmallCluster; cs >= 1; cs >>= 1) {
      const int64_t keys = cdiv64(p.h, cs), ctas = N * cs;
      for (int most : {32, 24, 16, 10, 8}) {
        const int64_t passes = cdiv64(keys, (int64_t)most * kWarp), w = cdiv64(keys, passes * kWarp) < 4 ? cdiv64(keys, passes * kWarp) : most;
        const int64_t kw = cdiv64(cdiv64(keys, passes * w), tpw) * tpw < kWarp ? cdiv64(cdiv64(keys, passes * w), tpw) * tpw : kWarp;
        const int64_t per_sm = kSmallWarps / w, sms = cs == 8 ? (per_sm > 1 ? 128 : 120) : cs == 4 ? (per_sm > 1 ? 138 : 132) : kPlanSMs;
        const int64_t waves = cdiv64(ctas, sms * per_sm);
        const int64_t resident = cdiv64(ctas, sms) < per_sm ? cdiv64(ctas, sms) : per_sm;
        const double lat = 0.7 + 0.45 * cdiv64(kw, tpw), load = (double)(resident * w * kw) * 3 * p.r * size / 60000.0;
        const double t = waves * (passes * (lat > load ? lat : load) + (cs > 1 ? 2.0 : 1.2));
        if (best == 0.0 || t < best) {
          best = t;
          f.groups = cs;
          f.warps = (int)w;
          f.kch = (int)kw;
          f.keys_per_split = (int)keys;
        }
      }
    }
    f.tiles = N < 1 << 20 ? N : 1 << 20;                 // clusters; each goes on to further tokens
    const size_t row = (size_t)pitch * 4;
    f.smem = kSmallCluster * row + f.warps * (row > kWarp * 16 ? row : kWarp * 16);
    return f;
  }
  const int slots = kPlanSMs * (wb + most_keys * per_key <= kSmemHalf + 1024 ? 2 : 1);
  double best = 0.0;
  for (int groups = kGroups; groups >= 1; groups >>= 1) {
    const int64_t tiles = cdiv64(N, (int64_t)warps * tpw * groups);
    int last = 0;
    for (int s = 1; s <= 64; ++s) {
      // the keys of a split in equal slabs, and a whole number of them
      const int64_t share = cdiv64(p.h, s);
      const int slabs = (int)cdiv64(share, (int64_t)most_keys), kch = (int)cdiv64(share, slabs);
      const int per = slabs * kch, splits = (int)cdiv64(p.h, per);
      if (splits > 1 && splits * part_bytes > kFwdScratchCap) break;
      if (splits == last) continue;
      last = splits;
      // clocks: a slab's copy, the work of one token group on it (rows of every pair, weights of every token), and the
      // partials' round trip
      const double copy = 1000.0 + (double)kch * per_key / 32.0;
      const double work = (double)warps * tpw * (kch * (pitch * size / 64.0 + 0.5) + 12.0);
      const double t = (double)cdiv64(tiles * splits, slots) * slabs * (copy + groups * work) +
                       (splits > 1 ? 4000.0 + (double)splits * part_bytes / 1500.0 : 0.0);
      if (best == 0.0 || t < best) {
        best = t;
        f.groups = groups;
        f.tiles = tiles;
        f.splits = splits;
        f.kch = kch;
        f.keys_per_split = per;
      }
    }
  }
  f.smem = wb + (size_t)f.kch * per_key;
  return f;
}

struct DzPlan { bool staged; int lpt, cv, warps, kch, groups; int64_t tiles; size_t smem; };
DzPlan make_dz_plan(const skv_problem& p) {
  DzPlan d;
  lanes_for(p.r, 4, &d.lpt, &d.cv);
  const int tpw = kWarp / d.lpt, pitch = d.lpt * 4 * d.cv;
  d.warps = staged_warps(d.lpt, d.cv, 4);
  const size_t bufs = (size_t)d.warps * tpw * (kWarp * 8 + (kWarp + 4) * 4), per_key = (size_t)(p.L - 1) * pitch * 4;
  size_t most_keys = (kSmemHalf - bufs) / per_key;
  if (most_keys < 8) most_keys = (kSmemFull - bufs) / per_key;
  d.staged = most_keys >= 1;
  if (most_keys > 32 || !d.staged) most_keys = 32;
  const int slots = kPlanSMs * (bufs + (d.staged ? most_keys * per_key : 0) <= kSmemHalf + 1024 ? 2 : 1);
  const int64_t N = p.N > 0 ? p.N : 1, unit = (int64_t)d.warps * tpw;
  double best = 0.0;
  for (int64_t kch = (int64_t)most_keys; kch >= 1; --kch) {
    if (kch > 8 && kch % 8) continue;                    // whole transposes, and aligned pieces of z and dz
    const int64_t slabs = cdiv64(p.h, kch);
    const double copy = 1000.0 + (d.staged ? (double)kch * per_key / 24.0 : 0.0);
    const double work = (double)unit * (cdiv64(kch, 8) * 8 * (pitch / 16.0 + 0.5) + 16.0);
    for (int64_t groups = 1; groups <= 64; groups <<= 1) {
      const int64_t tiles = cdiv64(N, unit * groups);
      const double t = (double)cdiv64(tiles * slabs, slots) * (copy + groups * work);
      if (best == 0.0 || t < best) { best = t; d.groups = (int)groups; d.tiles = tiles; d.kch = (int)kch; }
      if (tiles == 1) break;
    }
  }
  d.smem = bufs + (d.staged ? d.kch * per_key : 0);
  return d;
}

struct DcPlan { bool gacc; int lpt, cv, W, TT, splits; int64_t tokens_per_split; size_t smem; };
DcPlan make_dc_plan(const skv_problem& p) {
  DcPlan d;
  lanes_for(p.r, 4, &d.lpt, &d.cv);
  const int pitch = d.lpt * 4 * d.cv, nb = p.L - 1, S = kWarp / d.lpt;
  const size_t per_acc = (size_t)p.L * pitch * 4;
  auto bytes = [&](int W, int TT, bool gacc) {
    return (size_t)TT * pitch * 4 + (size_t)W * TT * 16 + (gacc ? 0 : W * per_acc) + (size_t)TT * (W | 1) * 4 +
           (size_t)W * (nb + 2) * 4;
  };
  const int64_t N = p.N > 0 ? p.N : 1;
  const double elems = (double)p.h * p.L * p.r;
  double best = 0.0;
  auto consider = [&](int W, int TT, bool gacc) {
    const int64_t groups = cdiv64(p.h, W), tiles = cdiv64(N, TT);
    // warp instructions of a tile and key: the sort, S pairs at a time, a finished row per interval; issued by a chip that
    // needs about twenty warps per SM to be busy
    const double tile = (double)W * (TT * 1.5 + TT * (6.0 + 14.0 * d.cv) / S + p.L * (14.0 + 12.0 * d.cv)) / (W < 20 ? W / 20.0 : 1.0);
    int64_t last = 0;
    for (int64_t s = 1; s <= 16 && s <= tiles; ++s) {
      const int64_t per = cdiv64(tiles, s), splits = cdiv64(tiles, per);
      if (splits == last) continue;
      last = splits;
      // clocks, with a CTA's prologue and epilogue, and the partials' round trip
      const double t = (double)cdiv64(groups * splits, kPlanSMs) * (per * (tile / 3.0 + 500.0) + 3000.0) +
                       (splits > 1 ? 3000.0 + splits * elems * 8 / 1500.0 : 0.0);
      if (best != 0.0 && t >= best) continue;
      best = t;
      d.gacc = gacc;
      d.W = W;
      d.TT = TT;
      d.smem = bytes(W, TT, gacc);
      d.splits = (int)splits;
      d.tokens_per_split = per * TT;
    }
  };
  for (int TT = kMaxTile; TT >= 64; TT >>= 1)
    for (int W : {24, 20, 16, 12, 8, 6, 4, 2, 1})
      if (bytes(W, TT, false) <= kSmemMost) consider(W, TT, false);
  if (best == 0.0) consider(kWarps, 64, true);
  return d;
}

// The plan of the last problem this thread asked about: a call asks for its scratch and again for its launch.
template <typename Plan, Plan (*Make)(const skv_problem&)>
const Plan& last_plan(const skv_problem& p) {
  static thread_local struct { int64_t N; int h, L, r, dtype, order; Plan plan; } last{-1, 0, 0, 0, 0, 0, {}};
  if (last.N != p.N || last.h != p.h || last.L != p.L || last.r != p.r || last.dtype != p.dtype || last.order != p.spline_order)
    last = {p.N, p.h, p.L, p.r, p.dtype, p.spline_order, Make(p)};
  return last.plan;
}
const FwdPlan& plan_forward(const skv_problem& p) { return last_plan<FwdPlan, make_forward_plan>(p); }
const DzPlan& plan_dz(const skv_problem& p) { return last_plan<DzPlan, make_dz_plan>(p); }
const DcPlan& plan_dc(const skv_problem& p) { return last_plan<DcPlan, make_dc_plan>(p); }

template <auto Kernel, typename... Args>
int launch(dim3 grid, int warps, size_t smem, cudaStream_t stream, const Args&... args) {
  if (launch_chained<Kernel>(grid, (unsigned)(warps * kWarp), smem, stream, args...) == cudaSuccess) return SKV_OK;
  cudaGetLastError();
  return SKV_ERR_LAUNCH;
}

// The CTAs of a token as a cluster.
template <typename K>
int launch_small(K kernel, const FwdPlan& f, const FwdArgs& a, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(f.tiles * f.groups));
  cfg.blockDim = dim3((unsigned)(f.warps * kWarp));
  cfg.dynamicSmemBytes = f.smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)f.groups;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  if (cudaLaunchKernelEx(&cfg, kernel, a) == cudaSuccess) return SKV_OK;
  cudaGetLastError();
  return SKV_ERR_LAUNCH;
}

// One case per (lanes per token, pieces per lane) that rows of up to 256 elements need.
#define SKV_LANES(LPT_, CV_, CALL)                                    \
  if (CV_ == 2) CALL(32, 2)                                           \
  else if (LPT_ == 2) CALL(2, 1)                                      \
  else if (LPT_ == 4) CALL(4, 1)                                      \
  else if (LPT_ == 8) CALL(8, 1)                                      \
  else if (LPT_ == 16) CALL(16, 1)                                    \
  else CALL(32, 1)

template <typename T, typename TD>
int forward_t(const LaunchCtx& c, const void* z, int64_t zs, const void* C, void* act_out, int64_t as,
              void* delta_out, int64_t ds, void* scratch, size_t scratch_bytes) {
  const skv_problem& p = c.p;
  FwdPlan f = plan_forward(p);
  if (f.splits > 1 && (!scratch || scratch_bytes < (size_t)f.splits * p.N * p.r * sizeof(float))) {
    f.splits = 1;                                        // no room for partials: a CTA covers all keys
    f.keys_per_split = p.h;
  }
  FwdArgs a;
  a.z = z; a.zs = zs; a.C = C; a.act_out = act_out; a.as = as; a.delta_out = delta_out; a.ds = ds;
  a.partial = f.splits > 1 ? static_cast<float*>(scratch) : nullptr;
  a.N = p.N; a.h = p.h; a.L = p.L; a.r = p.r; a.g = c.g; a.lambda = p.lambda_scale; a.act = p.activation;
  a.kch = f.kch; a.keys_per_split = f.keys_per_split; a.groups = f.groups;
  const dim3 grid((unsigned)f.tiles, (unsigned)f.splits);
  constexpr int n = Vec<T>::n;
  const uintptr_t at = reinterpret_cast<uintptr_t>(C);
  const int bytes = p.r % n == 0 && at % 16 == 0 ? 16 : p.r % (n / 2) == 0 && at % 8 == 0 ? 8 : 0;
  int e = SKV_OK;
  // (32 lanes take 256 bf16 in one piece: two pieces per lane are for float32)
#define SKV_CALL(LPT_, CV_)                                                                                     \
  {                                                                                                             \
    if constexpr (CV_ == 1 || n == 4) {                                                                         \
      if (f.small && bytes == 16) e = launch_small(simt_forward_small_kernel<T, TD, LPT_, CV_, 16>, f, a, c.stream);    \
      else if (f.small && bytes == 8) e = launch_small(simt_forward_small_kernel<T, TD, LPT_, CV_, 8>, f, a, c.stream);  \
      else if (f.small) e = launch_small(simt_forward_small_kernel<T, TD, LPT_, CV_, 0>, f, a, c.stream);     \
      else e = launch<simt_forward_kernel<T, TD, LPT_, CV_>>(grid, f.warps, f.smem, c.stream, a);                 \
    }                                                                                                           \
  }
  SKV_LANES(f.lpt, f.cv, SKV_CALL)
#undef SKV_CALL
  if (e) return e;
  note_launches(1);
  if (f.splits > 1) {
    const bool fours = p.r % 4 == 0 && reinterpret_cast<uintptr_t>(a.partial) % 16 == 0;
    const int64_t blocks = cdiv64(p.N * p.r, fours ? 4 * kWarp : kWarp);
    const dim3 fgrid((unsigned)(blocks < 4096 ? blocks : 4096));
    e = fours ? launch<simt_finalize_kernel<TD, 4>>(fgrid, 8, 0, c.stream, (const float*)a.partial, f.splits, p.N, p.r, p.lambda_scale,
                                                    static_cast<TD*>(delta_out), ds)
              : launch<simt_finalize_kernel<TD, 1>>(fgrid, 8, 0, c.stream, (const float*)a.partial, f.splits, p.N, p.r, p.lambda_scale,
                                                    static_cast<TD*>(delta_out), ds);
    note_launches(1);
  }
  return e;
}

template <typename T>
int backward_t(const LaunchCtx& c, const void* z, int64_t zs, const void* C, const void* g_act, int64_t gas,
               const void* g_delta, int64_t gds, void* dz, int64_t dzs, float* dC, void* dC_cast,
               void* scratch, size_t scratch_bytes) {
  const skv_problem& p = c.p;
  if (dz) {
    const DzPlan d = plan_dz(p);
    DzArgs a;
    a.z = z; a.zs = zs; a.C = C; a.g_act = g_act; a.gas = gas; a.g_delta = g_delta; a.gds = gds; a.dz = dz; a.dzs = dzs;
    a.N = p.N; a.h = p.h; a.L = p.L; a.r = p.r; a.g = c.g; a.coef = p.lambda_scale * c.g.scale; a.act = p.activation;
    a.kch = d.kch; a.groups = d.groups;
    const dim3 grid((unsigned)d.tiles, (unsigned)cdiv64(p.h, d.kch));
    int e = SKV_OK;
#define SKV_CALL(LPT_, CV_)                                                                              \
  {                                                                                                      \
    e = d.staged ? launch<simt_dz_kernel<T, LPT_, CV_, true>>(grid, d.warps, d.smem, c.stream, a)        \
                 : launch<simt_dz_kernel<T, LPT_, CV_, false>>(grid, d.warps, d.smem, c.stream, a);      \
  }
    SKV_LANES(d.lpt, d.cv, SKV_CALL)
#undef SKV_CALL
    if (e) return e;
    note_launches(1);
  }
  if (dC || dC_cast) {
    DcPlan d = plan_dc(p);
    const size_t elems = (size_t)p.h * p.L * p.r;
    const int64_t room = scratch ? (int64_t)(scratch_bytes / (elems * sizeof(float))) : 0;
    if (d.gacc && room < 1) return SKV_ERR_SCRATCH;
    if (d.splits > room) {                               // fewer splits where there is less room for partials
      d.splits = room > 1 ? (int)room : 1;
      d.tokens_per_split = cdiv64(cdiv64(p.N, d.splits), d.TT) * d.TT;
      d.splits = (int)cdiv64(p.N, d.tokens_per_split);
    }
    const bool parts = d.splits > 1 || d.gacc;
    DcArgs a;
    a.z = z; a.zs = zs; a.g_delta = g_delta; a.gds = gds;
    a.part = parts ? static_cast<float*>(scratch) : nullptr;
    a.dC = dC; a.dC_cast = dC_cast;
    a.N = p.N; a.h = p.h; a.L = p.L; a.r = p.r; a.g = c.g; a.lambda = p.lambda_scale;
    a.TT = d.TT; a.tokens_per_split = d.tokens_per_split;
    a.first = !dz;
    const dim3 grid((unsigned)cdiv64(p.h, d.W), (unsigned)d.splits);
    int e = SKV_OK;
#define SKV_CALL(LPT_, CV_)                                                                              \
  {                                                                                                      \
    e = d.gacc ? launch<simt_dc_kernel<T, LPT_, CV_, true>>(grid, d.W, d.smem, c.stream, a)              \
               : launch<simt_dc_kernel<T, LPT_, CV_, false>>(grid, d.W, d.smem, c.stream, a);            \
  }
    SKV_LANES(d.lpt, d.cv, SKV_CALL)
#undef SKV_CALL
    if (e) return e;
    note_launches(1);
    if (parts) {
      const unsigned rgrid = (unsigned)((elems + 255) / 256 < 4096 ? (elems + 255) / 256 : 4096);
      if (int e2 = launch<simt_dc_reduce_kernel<T>>(dim3(rgrid), 8, 0, c.stream, (const float*)a.part, d.splits, elems, p.lambda_scale,
                                                    dC, static_cast<T*>(dC_cast)))
        return e2;
      note_launches(1);
    }
  }
  return SKV_OK;
}

}  // namespace

size_t simt_scratch_bytes(const skv_problem& p, int op) {
  if (op == SKV_OP_BACKWARD) {
    const DcPlan d = plan_dc(p);
    return d.splits > 1 || d.gacc ? (size_t)d.splits * p.h * p.L * p.r * sizeof(float) : 0;
  }
  const FwdPlan f = plan_forward(p);
  return f.splits > 1 ? (size_t)f.splits * (p.N > 0 ? p.N : 1) * p.r * sizeof(float) : 0;
}

// Tokens up to which the forward reads table rows in place.  The line was fitted to earlier forms of both sides (in place: 8 us and one
// for every 1.05 M of N h r; the tensor-core chain: 15 us and one for every 0.26 M table elements).  In place against the
// tensor-core chain as they are, on the GPU, L = 22: h = 5120, r = 32 (line at 132): 132 tokens 17.2 and 18.1 us, 160 tokens 26.3 and 17.9;
// h = 5120, r = 128 (99): 100 tokens 48.9 and 48.8.  Elsewhere it is off: h = 2560, r = 32 (177): 200 tokens 14.9 and 15.6; h = 1024, r = 32
// (310): 250 tokens 8.3 and 12.3, 300 tokens 13.8 and 12.4.  Float32 has no tensor-core side; its 64 is not measured against the staged kernel.
int64_t small_forward_tokens(const skv_problem& p) {
  if (p.dtype != SKV_BF16) return 64;
  const int64_t n = 4 * (int64_t)p.L + 7300000 / ((int64_t)p.h * p.r);
  return n > 512 ? 512 : n;
}

int simt_forward(const LaunchCtx& c, const void* z, int64_t zs, const void* C, void* act_out, int64_t as,
                 void* delta_out, int64_t ds, void* scratch, size_t scratch_bytes) {
  if (c.p.dtype == SKV_F32)
    return forward_t<float, float>(c, z, zs, C, act_out, as, delta_out, ds, scratch, scratch_bytes);
  return c.p.delta_f32
             ? forward_t<__nv_bfloat16, float>(c, z, zs, C, act_out, as, delta_out, ds, scratch, scratch_bytes)
             : forward_t<__nv_bfloat16, __nv_bfloat16>(c, z, zs, C, act_out, as, delta_out, ds, scratch, scratch_bytes);
}

int simt_backward(const LaunchCtx& c, const void* z, int64_t zs, const void* C, const void* g_act, int64_t gas,
                  const void* g_delta, int64_t gds, void* dz, int64_t dzs, float* dC, void* dC_cast,
                  void* scratch, size_t scratch_bytes) {
  return c.p.dtype == SKV_BF16
             ? backward_t<__nv_bfloat16>(c, z, zs, C, g_act, gas, g_delta, gds, dz, dzs, dC, dC_cast, scratch,
                                         scratch_bytes)
             : backward_t<float>(c, z, zs, C, g_act, gas, g_delta, gds, dz, dzs, dC, dC_cast, scratch,
                                 scratch_bytes);
}

int simt_knot_index(const LaunchCtx& c, const void* z, int64_t zs, int32_t* bins) {
  const int64_t total = c.p.N * (int64_t)c.p.h;
  const unsigned grid = (unsigned)(cdiv64(total, 256) < 8192 ? cdiv64(total, 256) : 8192);
  if (c.p.dtype == SKV_BF16)
    simt_knot_index_kernel<__nv_bfloat16><<<grid, 256, 0, c.stream>>>((const __nv_bfloat16*)z, zs, c.p.N, c.p.h,
                                                                       c.g, bins);
  else
    simt_knot_index_kernel<float><<<grid, 256, 0, c.stream>>>((const float*)z, zs, c.p.N, c.p.h, c.g, bins);
  note_launches(1);
  return cudaGetLastError() == cudaSuccess ? SKV_OK : SKV_ERR_LAUNCH;
}

}  // namespace skv
