// Readout of the feature without materialising it:
//
//   y[N, D] = act(z)[N, h] * W[:, :h]^T  +  (lambda * delta)[N, r] * W[:, h:h+r]^T        (bf16, float32 accumulate)
//
// which is what spline_kv_fwd_fused_cuda of the reference returns
// (src/sparsespline_ffn/cuda_ext/spline_kv_fwd.cu:307-417: activation buffer, delta, two library GEMMs and
// an add).  Here it is one tcgen05 GEMM over the virtual operand [act(z) | lambda*delta] of K = h + r
// columns: the activation is applied to the z tile on its way from global to shared memory, so neither
// act(z) nor the concatenated feature is ever written to HBM; delta (bf16, lambda applied) comes from the
// feature kernel run in its delta-only mode just before.
//
// One persistent CTA per SM walks output tiles of 256 or 128 tokens x 256 outputs (with 256 two 128-row MMAs share
// each B tile, which halves the L2 traffic per flop of a 128 x 256 tile; with 128 the two accumulators in tensor
// memory are of successive tiles), or K slices of them:
//   warp  9    loader (lane 0): per stage one tiled TMA load of the 256 x 64 z (or delta) tile, 128-byte
//              swizzle, zero fill past N and h, and one 32 KB bulk copy from the pre-tiled image of W
//   warps 0-7  ReLU^2 in place on the landed z tile (elementwise, so the swizzled layout does not matter);
//              nothing to do for the identity activation.  After a tile's last stage the same warps are
//              its epilogue (accumulator -> bf16 -> y)
//   warp  8    MMA issue (lane 0): 128 x 256 x 16 per instruction
// Three stages of (A 32 KB + B 32 KB), or four of (16 + 32).  Tiles that share their 256 tokens are adjacent in the walk, so the
// z tile is read from HBM once and from L2 by the other D/256 - 1 CTAs.
// (Loading the z tile with ordinary 16-byte loads into registers instead cost 37 L1 wavefronts per
// load instruction and left the kernel bound by the load/store unit at 1.23 ms for the d20 shape,
// against 0.66 ms with the TMA load.  Six stages of 32 columns with the 64-byte swizzle were no faster
// than three of 64 and doubled the L2 traffic; squaring one K step (16 columns) at a time, with a barrier
// per step so that its MMAs start early, was slower: 0.71 against 0.68 ms.  So was a ReLU^2 variant with
// the squared tile in tensor memory (128-token tiles, accumulator in 256 columns, A ring in the rest; no
// stores back to shared memory and no A reads from it): 0.72 ms, because a 128 x 256 tile needs 48 KB
// from L2 per 4.2 MFLOP against 64 KB per 8.4 MFLOP here, and both kernels take in about 90 GB/s per
// SM, which looks like the limit of the L2-to-SM path.)
#include "skv_tc_prep.cuh"
#include "skv_tma.cuh"

namespace skv {
namespace tc {

constexpr int32_t kStatusTimeoutReadout = 0x10;

namespace {

constexpr int kRoK = 64;                         // K columns per stage: 64 (128-byte swizzle) or 32 (64-byte swizzle)
// Tiles of MT * 128 tokens x 256 outputs, MT = 2 or 1 (see readout_plan).
__host__ __device__ constexpr uint32_t ro_a_bytes(int mt) { return (uint32_t)mt * 128 * kRoK * 2; }
__host__ __device__ constexpr int ro_stages(int mt) { return mt == 2 ? 3 : 4; }      // 192 KB of stages
constexpr uint32_t kRoBBytes = 256 * kRoK * 2;   // one B stage: 256 outputs x kRoK
constexpr int kRoThreads = 320;

struct RoParams {
  const uint8_t* wimg;           // [n_tiles][ks][kRoBBytes]
  __nv_bfloat16* y;
  int64_t ys;
  int64_t N;
  int h, r, D;
  int ks_z;                      // stages that read z: ceil(h / kRoK)
  int ks;                        // all stages: ks_z + ceil(r / kRoK)
  int n_tiles;                   // ceil(D / 256)
  int64_t tiles;                 // m_tiles * n_tiles
  int64_t whole;                 // the first tiles are worked on in one piece, the others in K slices
  int slices, ks_per;            // of each of the others, and stages per slice
  float* partial;                // [slices][tiles - whole][128 * MT][256]
  int32_t* status;
  long long wait_cycles;
  int skip_copy;                 // test hook: the loader leaves out its first stage
};

// What a CTA works on at a time: a whole tile, or a K slice of one.
struct RoItem { int64_t tile; int slice, s_beg, s_end; };      // slice < 0: whole
__device__ __forceinline__ RoItem ro_item(const RoParams& P, int64_t t) {
  if (t < P.whole) return {t, -1, 0, P.ks};
  const int64_t rest = P.tiles - P.whole, i = t - P.whole;
  const int slice = (int)(i / rest);
  return {P.whole + i % rest, slice, slice * P.ks_per, min(P.ks, (slice + 1) * P.ks_per)};
}

// W[D][ws] (the layout of torch.nn.Linear.weight, columns [0,h) for act(z) and [h,h+r) for delta) ->
// per (output tile, stage) a 256 x kRoK K-major tile of 8 x 16-byte core matrices, [k core][n core][8 rows],
// zero where the tile reaches past D, h or r.
// `first`: the first kernel of a call; else it runs beside the one that is (and writes what the call in front of this one may
// still read only because that one has waited).
__global__ void tc_pack_w_kernel(const __nv_bfloat16* W, int64_t ws, int D, int h, int r, int ks_z, int ks,
                                 int64_t chunks, uint4* img, int first) {
  if (first) pdl_wait();
  pdl_launch();
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < chunks; idx += (int64_t)gridDim.x * blockDim.x) {
    constexpr int kPer = (int)(kRoBBytes / 16);
    const int c = (int)(idx % kPer);
    const int64_t ts = idx / kPer;
    const int s = (int)(ts % ks);
    const int64_t nt = ts / ks;
    const int kc = c >> 8, nc = (c >> 3) & 31, row = c & 7;
    const int64_t n = nt * 256 + nc * 8 + row;
    bool ok = n < D;
    int64_t k;
    if (s < ks_z) {
      k = (int64_t)s * kRoK + kc * 8;
      ok = ok && k < h;
    } else {
      const int kd = (s - ks_z) * kRoK + kc * 8;
      ok = ok && kd < r;
      k = (int64_t)h + kd;
    }
    img[idx] = ok ? ld16(W + n * ws + k) : make_uint4(0, 0, 0, 0);
  }
  if (!first) pdl_wait();                            // whoever waits for this kernel has waited for the one in front of it
}

template <bool RELU, int MT>
__global__ void __launch_bounds__(kRoThreads, 1)
    tc_readout_kernel(const RoParams P, const __grid_constant__ CUtensorMap map_z, const __grid_constant__ CUtensorMap map_d) {
  extern __shared__ uint8_t smem_raw[];
  constexpr int kRoStages = ro_stages(MT);
  constexpr uint32_t kRoABytes = ro_a_bytes(MT);
  constexpr uint32_t NB = MT == 1 ? 2u : 1u;     // accumulators in flight: all 512 tensor-memory columns either way
  // the swizzled A stages need 512-byte alignment (1024 keeps room for the 128-byte mode)
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* a_base = smem;
  uint8_t* b_base = smem + kRoStages * kRoABytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(b_base + kRoStages * kRoBBytes);
  uint64_t* full = bars;                         // [stages] TMA + bulk copy landed
  uint64_t* ready = full + kRoStages;            // [stages] activation applied (one arrival per warp); RELU only
  uint64_t* empty = ready + kRoStages;           // [stages] MMA -> loader
  uint64_t* acc_full = empty + kRoStages;        // [NB] MMA -> epilogue
  uint64_t* acc_empty = acc_full + NB;           // [NB] epilogue -> MMA (one arrival per warp)
  uint64_t* done = acc_empty + NB;               // [1]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const WaitCtx wc{abort_flag, P.status, kStatusTimeoutReadout, P.wait_cycles};

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int i = 0; i < kRoStages; ++i) { mbar_init(full + i, 1); mbar_init(ready + i, 8); mbar_init(empty + i, 1); }
    for (uint32_t i = 0; i < NB; ++i) { mbar_init(acc_full + i, 1); mbar_init(acc_empty + i, 8); }
    mbar_init(done, 1);
    *abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == 8) tmem_alloc(tmem_slot, 512);
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int64_t step = gridDim.x, items = P.whole + (P.tiles - P.whole) * P.slices;
  pdl_wait();
  pdl_launch();

  if (warp < 8) {
    // ------------------------------------------------------------------ activation in place, then epilogue
    uint32_t it = 0, ti = 0;
    bool drain = false;
    for (int64_t t = blockIdx.x; t < items && !drain; t += step, ++ti) {
      const RoItem item = ro_item(P, t);
      const int64_t tile = item.tile;
      if (RELU) {
        for (int s = item.s_beg; s < item.s_end && !drain; ++s, ++it) {
          const uint32_t st = it % kRoStages;
          if (mbar_wait(full + st, (it / kRoStages) & 1u, wc)) { drain = true; break; }
          if (s < P.ks_z) {
            // elementwise, so the swizzled layout does not matter: 16-byte chunk j * 256 + tid of the stage
            constexpr int kPerThread = (int)(kRoABytes / 4096);
            const uint32_t src = smem_u32(a_base + st * kRoABytes) + (uint32_t)tid * 16u;
            uint4 v[kPerThread];
#pragma unroll
            for (int j = 0; j < kPerThread; ++j) v[j] = lds128(src + (uint32_t)j * 4096u);
#pragma unroll
            for (int j = 0; j < kPerThread; ++j) {
              v[j].x = relu_sq_bf2(v[j].x); v[j].y = relu_sq_bf2(v[j].y);
              v[j].z = relu_sq_bf2(v[j].z); v[j].w = relu_sq_bf2(v[j].w);
              sts128(src + (uint32_t)j * 4096u, v[j].x, v[j].y, v[j].z, v[j].w);
            }
            fence_async_smem();
          }
          mbar_arrive_warp(ready + st);
        }
        if (drain) break;
      }
      // ---- epilogue of this item: accumulator rows of this warp -> bf16 -> y, or float32 -> partial
      const uint32_t ab = ti % NB;
      if (mbar_wait(acc_full + ab, (ti / NB) & 1u, wc)) break;
      tc_fence_after();
      // MT = 2: warps 0-3 and 4-7 take a token half each; MT = 1: an output half each
      const int64_t n = (tile / P.n_tiles) * (128 * MT) + (MT == 2 ? warp * 32 : (warp & 3) * 32) + lane;
      const int col0 = MT == 2 ? 0 : (warp >> 2) * 128;
      const int n0 = (int)(tile % P.n_tiles) * 256 + col0;
      const uint32_t taddr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (MT == 2 ? (uint32_t)(warp >> 2) * 256u : ab * 256u + (uint32_t)col0);
      const int64_t nn = n < P.N ? n : 0;
      float* part = P.partial;
      if (item.slice >= 0)
        part += (((size_t)item.slice * (P.tiles - P.whole) + (tile - P.whole)) * (128 * MT) + (MT == 2 ? warp * 32 : (warp & 3) * 32) + lane) * 256 + col0;
#pragma unroll 1
      for (int c = 0; c < 4 * MT; ++c) {
        float v[32];
        tmem_ld16(taddr + (uint32_t)(c * 32), v);
        tmem_ld16(taddr + (uint32_t)(c * 32 + 16), v + 16);
        if (n < P.N) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int col = n0 + c * 32 + q * 8;
            if (col >= P.D) continue;
            if (item.slice >= 0) {
              float4* o = reinterpret_cast<float4*>(part + c * 32 + q * 8);
              o[0] = make_float4(v[q * 8], v[q * 8 + 1], v[q * 8 + 2], v[q * 8 + 3]);
              o[1] = make_float4(v[q * 8 + 4], v[q * 8 + 5], v[q * 8 + 6], v[q * 8 + 7]);
            } else {
              *reinterpret_cast<uint4*>(P.y + nn * P.ys + col) =
                  make_uint4(pack_bf2(v[q * 8], v[q * 8 + 1]), pack_bf2(v[q * 8 + 2], v[q * 8 + 3]),
                             pack_bf2(v[q * 8 + 4], v[q * 8 + 5]), pack_bf2(v[q * 8 + 6], v[q * 8 + 7]));
            }
          }
        }
      }
      tc_fence_before();
      mbar_arrive_warp(acc_empty + ab);
    }
  } else if (warp == 8) {
    // ------------------------------------------------------------------ MMA issue
    if (elect_one()) {
      // A: K-major tile whose rows are one swizzle span (128 or 64 bytes) long, 8-row groups 8 rows apart;
      // a K step of 16 elements advances the start address by 32 bytes inside the swizzled row.
      constexpr uint32_t kRowBytes = kRoK * 2;
      const uint32_t a_hi = ((8u * kRowBytes) >> 4) | (1u << 14) | ((kRoK == 64 ? 2u : 4u) << 29);
      const uint32_t b_hi = desc_hi(128u);
      constexpr uint32_t idesc = instr_desc(1, 1, 0, 0, 128, 256);
      uint32_t it = 0, ti = 0;
      bool drain = false;
      for (int64_t t = blockIdx.x; t < items && !drain; t += step, ++ti) {
        const uint32_t ab = ti % NB;
        if (ti >= NB) drain = mbar_wait(acc_empty + ab, (ti / NB - 1u) & 1u, wc);
        if (drain) break;
        tc_fence_after();
        const RoItem item = ro_item(P, t);
        const int s_beg = item.s_beg, s_end = item.s_end;
        const uint32_t d_addr = tmem_base + (MT == 1 ? ab * 256u : 0u);
        for (int s = s_beg; s < s_end; ++s, ++it) {
          const uint32_t st = it % kRoStages, ph = (it / kRoStages) & 1u;
          drain = mbar_wait((RELU ? ready : full) + st, ph, wc);
          if (drain) break;
          tc_fence_after();
          int nk = kRoK / 16;
          if (s >= P.ks_z) nk = min(kRoK / 16, (P.r - (s - P.ks_z) * kRoK + 15) / 16);
          uint32_t a_lo = ((smem_u32(a_base + st * kRoABytes) >> 4) & 0x3FFFu) | (1u << 16);
          uint32_t b_lo = desc_lo(smem_u32(b_base + st * kRoBBytes), 4096u);
          for (int k = 0; k < nk; ++k) {
            const uint32_t accf = (s > s_beg || k > 0) ? 1u : 0u;
            umma_f16_split(d_addr, a_lo, a_hi, b_lo, b_hi, idesc, accf);                             // tokens 0-127
            if constexpr (MT == 2)
              umma_f16_split(d_addr + 256u, a_lo + ((128u * kRowBytes) >> 4), a_hi, b_lo, b_hi, idesc, accf);  // tokens 128-255
            a_lo += 32u >> 4;
            b_lo += 8192u >> 4;
          }
          umma_commit(empty + st);
        }
        if (!drain) umma_commit(acc_full + ab);
      }
      umma_commit(done);
    }
  } else {
    // ------------------------------------------------------------------ loader
    if (elect_one()) {
      uint32_t it = 0;
      bool stop = false;
      for (int64_t t = blockIdx.x; t < items && !stop; t += step) {
        const RoItem item = ro_item(P, t);
        const uint8_t* src = P.wimg + (size_t)(item.tile % P.n_tiles) * P.ks * kRoBBytes;
        const int m0 = (int)((item.tile / P.n_tiles) * (128 * MT));
        const int s_beg = item.s_beg, s_end = item.s_end;
        for (int s = s_beg; s < s_end; ++s, ++it) {
          const uint32_t st = it % kRoStages;
          if (it == 0 && P.skip_copy) continue;      // test hook: nothing ever completes full[0]
          if (it >= kRoStages && mbar_wait(empty + st, ((it / kRoStages) - 1u) & 1u, wc)) { stop = true; break; }
          mbar_arrive_expect_tx(full + st, kRoABytes + kRoBBytes);
          if (s < P.ks_z) tma_load_2d(a_base + st * kRoABytes, &map_z, s * kRoK, m0, full + st);
          else tma_load_2d(a_base + st * kRoABytes, &map_d, (s - P.ks_z) * kRoK, m0, full + st);
          bulk_g2s(b_base + st * kRoBBytes, src + (size_t)s * kRoBBytes, kRoBBytes, full + st);
        }
      }
      if (*abort_flag) {              // let copies in flight land before the CTA's shared memory goes away
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) {}
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 8) {
    mbar_wait_drain(done, 0, P.wait_cycles);
    tc_fence_after();
    tmem_free(tmem_base, 512);
  }
}

// Boxes of 128 * mt rows x kRoK columns, the swizzle span of one row.
bool make_map(CUtensorMap* m, const void* base, uint64_t rows, uint64_t cols, uint64_t pitch, int mt) {
  return make_map_2d(m, base, rows, cols, pitch, kRoK, 128 * mt, CU_TENSOR_MAP_SWIZZLE_128B);
}

// y = bf16 of the sum of the K slices' partials, in order, for the tiles that were sliced; four outputs per thread.
__global__ void __launch_bounds__(256) tc_readout_sum_kernel(const float* partial, int slices, int64_t whole, int64_t rest, int rows,
                                                             int n_tiles, int64_t N, int D, __nv_bfloat16* y, int64_t ys) {
  pdl_wait();
  pdl_launch();
  const int64_t total = rest * rows * 64;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t b = i / (rows * 64), tile = whole + b;
    const int e = (int)(i - b * (rows * 64));
    const int64_t n = tile / n_tiles * rows + e / 64;
    const int col = (int)(tile % n_tiles) * 256 + e % 64 * 4;
    if (n >= N || col >= D) continue;
    const float4* src = reinterpret_cast<const float4*>(partial) + i;
    float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 8
    for (int k = 0; k < slices; ++k) {
      const float4 v = src[(size_t)k * total];
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    *reinterpret_cast<uint2*>(y + n * ys + col) = make_uint2(pack_bf2(s.x, s.y), pack_bf2(s.z, s.w));
  }
}

// Tile height, how many tiles are worked on whole, and K slices of the others.  Microseconds: a stage of 256 tokens costs 0.91 with
// ReLU^2 (0.70 without), one of 128 tokens more than half of that (it reads as much of W); an item's fill and epilogue; a launch more and
// partials through L2.  256 tokens give the best rate; whole rounds of tiles need no partials; slices spread a last round that
// is not full, or few tokens, over the chip.  8192 x 5120 -> 1280 (320 tiles of 128 tokens on 148 SMs): in three rounds 127 us,
// in two rounds and six slices 105 with the sum; these constants take five slices (the whole call 252 us in three rounds, 233 so).
struct RoPlan { int mt, slices, ks_per; int64_t whole; };
RoPlan readout_plan(const skv_problem& p, int64_t D) {
  const int ks = (p.h + kRoK - 1) / kRoK + (p.r + kRoK - 1) / kRoK;
  const bool relu = p.activation == SKV_ACT_RELU_SQ;
  RoPlan best{2, 1, ks, 0};
  double best_t = 0.0;
  for (int mt = 2; mt >= 1; --mt) {
    const int64_t tiles = ((p.N > 0 ? p.N : 1) + 128 * mt - 1) / (128 * mt) * ((D + 255) / 256), rounds = tiles / kPlanSMs;
    const double stage = mt == 2 ? (relu ? 0.91 : 0.70) : (relu ? 0.50 : 0.37), fix = 3.0 * mt;
    auto take = [&](double t, int slices, int per, int64_t whole) {
      if (best_t == 0.0 || t < best_t) { best_t = t; best = {mt, slices, per, whole}; }
    };
    take((double)((tiles + kPlanSMs - 1) / kPlanSMs) * (ks * stage + fix), 1, ks, tiles);
    for (int64_t full = rounds; full >= 0 && full >= rounds - 1; --full) {
      const int64_t whole = full * kPlanSMs, rest = tiles - whole;
      int last = 1;
      for (int s = 2; s <= 16 && s <= (ks + 3) / 4 && rest > 0; ++s) {
        const int per = (ks + s - 1) / s, slices = (ks + per - 1) / per;
        if (slices == last) continue;
        last = slices;
        take(full * (ks * stage + fix) + (double)((rest * slices + kPlanSMs - 1) / kPlanSMs) * (per * stage + fix) + 8.0 +
                 (double)slices * rest * mt * 128 * 256 * 8.0 / 4.0e6,
             slices, per, whole);
      }
    }
  }
  return best;
}

size_t wimg_bytes(const skv_problem& p, int64_t D) {
  const size_t ks = (size_t)(p.h + kRoK - 1) / kRoK + (size_t)(p.r + kRoK - 1) / kRoK;
  return (size_t)((D + 255) / 256) * ks * kRoBBytes;
}

}  // namespace

bool readout_eligible(const skv_problem& p, int64_t D) {
  return p.N < ((int64_t)1 << 31) - 256 && p.dtype == SKV_BF16 && (p.activation == SKV_ACT_RELU_SQ || p.activation == SKV_ACT_IDENTITY) && p.h % 8 == 0 &&
         p.r % 8 == 0 && D >= 8 && D % 8 == 0 && D <= (1 << 24);
}

int64_t readout_tiles(const skv_problem& p, int64_t D, int mt) {
  return ((p.N > 0 ? p.N : 1) + 128 * mt - 1) / (128 * mt) * ((D + 255) / 256);
}

void describe_readout_plan(const skv_problem& p, int64_t D, int64_t* out) {
  const RoPlan f = readout_plan(p, D);
  out[0] = 128 * f.mt;
  out[1] = readout_tiles(p, D, f.mt);
  out[2] = f.whole;
  out[3] = f.slices;
}

// Image of W, then the K slices' partials.
size_t readout_image_bytes(const skv_problem& p, int64_t D) {
  const RoPlan f = readout_plan(p, D);
  return wimg_bytes(p, D) + (size_t)(f.slices > 1 ? f.slices * (readout_tiles(p, D, f.mt) - f.whole) : 0) * f.mt * 128 * 256 * sizeof(float);
}

// Row pitch (elements) of the delta buffer the GEMM reads: whole stages of kRoK columns.
int64_t readout_delta_pitch(const skv_problem& p) { return (int64_t)((p.r + kRoK - 1) / kRoK) * kRoK; }

// Tiled image of W, in front of the feature kernels or beside their first, so that the GEMM can be chained to them.
int readout_pack(const LaunchCtx& c, const void* W, int64_t ws, int64_t D, void* wimg, bool first) {
  const skv_problem& p = c.p;
  const int ks_z = (p.h + kRoK - 1) / kRoK, ks = ks_z + (p.r + kRoK - 1) / kRoK;
  const int64_t chunks = (D + 255) / 256 * ks * (kRoBBytes / 16);
  const int pgrid = (int)((chunks + 255) / 256 < 4096 ? (chunks + 255) / 256 : 4096);
  const cudaError_t e = launch_chained<tc_pack_w_kernel>(dim3((unsigned)pgrid), 256, 0, c.stream, static_cast<const __nv_bfloat16*>(W),
                                                         ws, (int)D, p.h, p.r, ks_z, ks, chunks, static_cast<uint4*>(wimg),
                                                         first ? 1 : 0);
  note_launches(1);
  return e == cudaSuccess ? SKV_OK : SKV_ERR_LAUNCH;
}

// y = [act(z) | delta] * W^T; `delta` is [N][readout_delta_pitch()] bf16 (its map ends at column r: what lies behind reads as
// zeros), `wimg`
// has readout_image_bytes().
int readout(const LaunchCtx& c, const void* z, int64_t zs, const void* delta, int64_t D, void* y, int64_t ys, void* wimg) {
  const skv_problem& p = c.p;
  const RoPlan f = readout_plan(p, D);
  RoParams P;
  P.wimg = static_cast<const uint8_t*>(wimg);
  P.y = static_cast<__nv_bfloat16*>(y);
  P.ys = ys;
  P.N = p.N;
  P.h = (int)p.h;
  P.r = (int)p.r;
  P.D = (int)D;
  P.ks_z = (int)((p.h + kRoK - 1) / kRoK);
  P.ks = P.ks_z + (int)((p.r + kRoK - 1) / kRoK);
  P.n_tiles = (int)((D + 255) / 256);
  P.tiles = readout_tiles(p, D, f.mt);
  P.whole = f.whole;
  P.slices = f.slices;
  P.ks_per = f.ks_per;
  P.partial = reinterpret_cast<float*>(static_cast<uint8_t*>(wimg) + wimg_bytes(p, D));
  P.status = c.status;
  P.wait_cycles = wait_cycle_limit();
  P.skip_copy = debug_skip_copy() == 2;
  CUtensorMap map_z, map_d;
  if (!make_map(&map_z, z, (uint64_t)p.N, (uint64_t)p.h, (uint64_t)zs, f.mt) ||
      !make_map(&map_d, delta, (uint64_t)p.N, (uint64_t)p.r, (uint64_t)readout_delta_pitch(p), f.mt))
    return SKV_ERR_LAUNCH;
  const size_t smem = (size_t)ro_stages(f.mt) * (ro_a_bytes(f.mt) + kRoBBytes) + 1024 + 256;
  const int64_t items = P.whole + (P.tiles - P.whole) * P.slices;
  const dim3 grid((unsigned)(items < c.num_sms ? items : c.num_sms));
  const bool relu = p.activation == SKV_ACT_RELU_SQ;
  const cudaError_t err =
      f.mt == 2 ? (relu ? launch_chained<tc_readout_kernel<true, 2>>(grid, kRoThreads, smem, c.stream, P, map_z, map_d)
                        : launch_chained<tc_readout_kernel<false, 2>>(grid, kRoThreads, smem, c.stream, P, map_z, map_d))
                : (relu ? launch_chained<tc_readout_kernel<true, 1>>(grid, kRoThreads, smem, c.stream, P, map_z, map_d)
                        : launch_chained<tc_readout_kernel<false, 1>>(grid, kRoThreads, smem, c.stream, P, map_z, map_d));
  note_launches(1);
  if (err != cudaSuccess) { cudaGetLastError(); return SKV_ERR_LAUNCH; }
  if (P.slices > 1) {
    const int rows = 128 * f.mt;
    const int64_t rest = P.tiles - P.whole, blocks = (rest * rows * 64 + 255) / 256;
    const dim3 sgrid((unsigned)(blocks < kPlanSMs * 16 ? blocks : kPlanSMs * 16));
    if (launch_chained<tc_readout_sum_kernel>(sgrid, 256, 0, c.stream, (const float*)P.partial, P.slices, P.whole, rest, rows, P.n_tiles,
                                              P.N, P.D, P.y, P.ys) != cudaSuccess) {
      cudaGetLastError();
      return SKV_ERR_LAUNCH;
    }
    note_launches(1);
  }
  return SKV_OK;
}

}  // namespace tc
}  // namespace skv
