// tcgen05 forward kernel of the spline-KV feature operator and its launch over the template cases; one
// translation unit per (spline order, base path) instantiates it.
//
//   delta[n, c] = sum_j sum_b Phi[n, (j,b)] * C[j, b, c]
//
// is computed as a dense GEMM on the 5th-generation tensor cores: the expanded basis Phi (order + 1
// non-zero weights per key, at knot rows bin, bin + 1, ...) is built per token as f16 in tensor memory, the
// code table is staged by TMA bulk copies from a range-scaled f16 image in the canonical operand layout, and
// tcgen05.mma accumulates 128-token x r tiles in tensor memory in float32.
#pragma once

#include "skv_tc_prep.cuh"

namespace skv {
namespace tc {

constexpr int kMaxTaCStages = 8;

struct FwdParams {
  const __nv_bfloat16* z;
  int64_t zs;
  __nv_bfloat16* act_out;
  int64_t as;
  const __half* cimg;       // [h/8][8*LP/8][r/8][8][8] f16 image of C, LP rows per key
  float* partial;           // [splits][N][r]
  int64_t N;
  int r;                    // code channels, padded to a multiple of 16
  GridParams g;
  int act;
  int chunks_total, chunks_per_split;
  int32_t* status;
  uint32_t b_lbo, b_sbo;
  int cstages;              // depth of the code-table ring (2..8)
  long long wait_cycles;    // limit of every bounded wait, in clock cycles
  int skip_copy;            // test hook: the loader leaves out the copy of its first chunk
};

// Knot rows per key in units of two (f16x2 words) the kernel is instantiated for: the common knot counts
// (L = 15..16, 21..22, 23..24, 31..32, 41..42) as they are, every other one rounded up (zero rows).
inline int fwd_words(int L) {
  const int hl = (L + 1) / 2;
  for (int v : {4, 6, 8, 11, 12, 16, 21, 22, 32})
    if (hl <= v) return v;
  return 0;
}

// Token groups (of 128) a CTA can hold: 8 * words columns of Phi and r of accumulator each.
inline int fwd_max_groups(int words, int r) {
  const int hlp = (words + 1) & ~1;
  const int g = 512 / (kChunkKeys * hlp + r);
  return g > 4 ? 4 : g;
}

// ---------------------------------------------------------------------------------------------
// Launch shape: grid = (token tiles of 128*GROUPS tokens, key splits).  Each producer thread owns a token: it
// builds the complete Phi row segment of a key (HL = L/2 f16x2 words, two of them non-zero) in
// registers and writes it with tcgen05.st into its own tensor-memory lane; the MMA takes A from
// tensor memory and only the code-table chunk (B) from shared memory.  Nothing has to be
// cleared: a row segment is overwritten completely every chunk.
//
// Tensor-memory columns per token group: 8*HL for A (single-buffered) followed by r for the
// accumulator; with four groups (512 tokens per CTA, 16 producer warps) the other groups keep the
// SM busy while one group waits for its MMAs.
// ---------------------------------------------------------------------------------------------
// Keys of each half chunk (of four) that are placed through the staging row (load/store pipe); the
// others are placed by multiplying with 0/1 masks in packed f16 arithmetic (FMA pipe).  With the mask
// arithmetic the d20 shape takes 0.917 / 0.890 / 0.903 ms for 0 / 1 / 2 of four.  (The linear spline
// stages none: the word behind its last interval's weight would lie past the row.)
constexpr int kStagedPerHalf = 1;

template <int GROUPS, int HL, int ACT, bool LIN>
__global__ void __launch_bounds__(160 * GROUPS + 32, 1) tc_forward_ta_kernel(const FwdParams P) {
  extern __shared__ __align__(128) uint8_t smem[];
  // Keys are padded to HLP words (an even count), so that half a chunk (4 keys) is a whole number
  // of K = 16 steps; the code-table image has 2*HLP rows per key, the padding rows are zero.
  constexpr int HLP = (HL + 1) & ~1;
  constexpr int NSTH = LIN ? 0 : kStagedPerHalf;
  constexpr int kHalfKeys = kChunkKeys / 2;
  constexpr int kHalfSteps = kHalfKeys * HLP / 8;                  // K = 16 steps per half chunk
  const int r = P.r;
  const uint32_t c_bytes = (uint32_t)(kChunkKeys * 2 * HLP * r * 2);
  const int CS = P.cstages;
  uint8_t* c_base = smem;                                          // [cstage][c_bytes]
  // One private staging row of HLP words per producer thread.  Placing the two non-zero words of
  // a row segment costs about thirty compare/select instructions on the half-rate ALU pipe; for
  // NSTH of the four keys of every half chunk the thread instead stores the two words into its
  // (zeroed) staging row at the dynamic position, reads the row back and zeroes the two words
  // again, which moves that work to the load/store pipe.  The rows of a warp are interleaved by
  // lane (word w of lane l at (w * 32 + l) * 4 bytes of the warp's region), so the bank of every
  // access is the lane and neither the scattered stores nor the loads conflict, whatever the knot
  // intervals of the 32 tokens are.
  constexpr int SW = HLP;
  uint8_t* stage_base = c_base + (size_t)CS * c_bytes;             // [128*GROUPS][SW words]
  uint64_t* bars = reinterpret_cast<uint64_t*>(stage_base + (size_t)128 * GROUPS * SW * 4);
  uint64_t* full = bars;                          // [group][half]  producers -> MMA
  uint64_t* empty = full + 2 * GROUPS;            // [group][half]  MMA -> producers
  uint64_t* cfull = empty + 2 * GROUPS;           // [cstage]       TMA -> MMA
  uint64_t* cempty = cfull + kMaxTaCStages;       // [cstage]       MMA -> TMA
  uint64_t* done = cempty + kMaxTaCStages;        // [group]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + GROUPS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const WaitCtx wc{abort_flag, P.status, kStatusTimeoutFwd, P.wait_cycles};

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int chunk_begin = blockIdx.y * P.chunks_per_split;
  const int nch = min(P.chunks_per_split, P.chunks_total - chunk_begin);
  const int64_t tile_base = (int64_t)blockIdx.x * (128 * GROUPS);
  const uint32_t grp_cols = (uint32_t)(kChunkKeys * HLP + r);
  uint32_t tmem_cols = 32;
  while (tmem_cols < GROUPS * grp_cols) tmem_cols <<= 1;

  if (tid == 0) {
    for (int i = 0; i < 2 * GROUPS; ++i) { mbar_init(full + i, 4); mbar_init(empty + i, 1); }
    for (int i = 0; i < GROUPS; ++i) mbar_init(done + i, 1);
    for (int i = 0; i < kMaxTaCStages; ++i) { mbar_init(cfull + i, 1); mbar_init(cempty + i, GROUPS); }
    *abort_flag = 0;
    mbar_init_fence();
  }
  if (NSTH > 0)
    for (uint32_t i = tid; i < (uint32_t)(128 * GROUPS * SW / 4); i += blockDim.x)
      reinterpret_cast<uint4*>(stage_base)[i] = make_uint4(0, 0, 0, 0);
  if (warp == 5 * GROUPS) tmem_alloc(tmem_slot, tmem_cols);
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch();
  pdl_wait();

  if (warp < 4 * GROUPS) {
    // ------------------------------------------------------------------ producers / epilogue
    const int grp = warp >> 2;
    const int t = tid & 127;
    const int64_t n = tile_base + grp * 128 + t;
    const bool valid = n < P.N;
    const __nv_bfloat16* zrow = P.z + (valid ? n : 0) * P.zs + (int64_t)chunk_begin * kChunkKeys;
    __nv_bfloat16* arow = P.act_out ? P.act_out + (valid ? n : 0) * P.as + (int64_t)chunk_begin * kChunkKeys : nullptr;
    const uint32_t lane_addr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)grp * grp_cols;
    uint4 znext = valid && nch > 0 ? ld16(zrow) : make_uint4(0, 0, 0, 0);
    // word w of this thread's staging row lives at (warp * HLP + w) * 128 + lane * 4: its bank is the
    // lane, whatever w is, so neither the scattered stores nor the loads conflict
    const uint32_t srow = smem_u32(stage_base) + (uint32_t)(warp * HLP * 128 + lane * 4);
    const uint32_t srow_biased = srow - (kWordBias << 7);          // wp carries the bias kWordBias
    for (int ci = 0; ci < nch; ++ci) {
      const uint4 zc = znext;
      if (ci + 1 < nch && valid) znext = ld16(zrow + (ci + 1) * kChunkKeys);
      const uint32_t zw[4] = {zc.x, zc.y, zc.z, zc.w};
      // phi(z) of the chunk's eight keys in packed bf16 arithmetic: the product of two bf16 values is
      // exact in float32, so one rounding to bf16 gives the same result as float32 arithmetic and a cast
      uint32_t aw[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if constexpr (ACT == SKV_ACT_RELU_SQ) aw[i] = relu_sq_bf2(zw[i]);
        else aw[i] = P.act == SKV_ACT_GELU ? pack_bf2(gelu_fwd(bf_lo(zw[i])), gelu_fwd(bf_hi(zw[i]))) : zw[i];
      }
      // The group's A columns are written and consumed in two halves of 4 keys: the MMAs of one
      // half run while the other half is being built, so the producers do not wait for them.
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        if (ci > 0) {
          mbar_wait(empty + grp * 2 + half, (uint32_t)(ci - 1) & 1u, wc);
          tc_fence_after();
        }
        // The first NSTH keys of the half go through the staging row: their stores and loads are
        // issued first, the select chains of the other keys run while those loads are in flight,
        // and the staged rows are written to tensor memory last.
        // The words of two neighbouring keys are stored to tensor memory together (2 * HLP columns:
        // one 16- and one 8-column store at HLP = 12 instead of two of each).
        uint32_t WP[kHalfKeys / 2][2 * HLP];
        // knot interval and weights of the half's four keys, two keys (one packed z word) at a time
        uint32_t kx0[kHalfKeys], kx1[kHalfKeys], kwp[kHalfKeys];
#pragma unroll
        for (int pq = 0; pq < kHalfKeys / 2; ++pq) {
          uint32_t a0[2], a1[2], aw2[2];
          phi_pair_words2<LIN>(zw[half * (kHalfKeys / 2) + pq], P.g, a0, a1, aw2);   // rows past N read z = 0; their accumulator rows are never stored
          kx0[2 * pq] = a0[0]; kx1[2 * pq] = a1[0]; kwp[2 * pq] = aw2[0];
          kx0[2 * pq + 1] = a0[1]; kx1[2 * pq + 1] = a1[1]; kwp[2 * pq + 1] = aw2[1];
        }
#pragma unroll
        for (int qq = 0; qq < NSTH; ++qq) {
          const uint32_t x0 = kx0[qq], x1 = kx1[qq], wp = kwp[qq];
          const uint32_t pos = srow_biased + (wp << 7);
          sts32(pos, x0);
          sts32(pos + 128u, x1);
#pragma unroll
          for (int i = 0; i < HLP; ++i)
            asm volatile("ld.shared.b32 %0, [%1];" : "=r"(WP[qq >> 1][(qq & 1) * HLP + i]) : "r"(srow + (uint32_t)i * 128u) : "memory");
          sts32(pos, 0u);
          sts32(pos + 128u, 0u);
        }
#pragma unroll
        for (int qq = NSTH; qq < kHalfKeys; ++qq) {
          const uint32_t x0 = kx0[qq], x1 = kx1[qq], wp = kwp[qq];
          // Placement at word-pair granularity: wp = 2 * qd + s.  The two words land in pair qd as
          // (x0, x1) when s = 0, or as (0, x0) there and (x1, 0) in pair qd + 1 when s = 1.
          uint32_t* W = &WP[qq >> 1][(qq & 1) * HLP];
          const bool odd = (wp & 1u) != 0u;
          const uint32_t y0 = odd ? 0u : x0, y1 = odd ? x0 : x1, y2 = odd ? x1 : 0u;
          constexpr int kLastPair = (HL - (LIN ? 1 : 2)) >> 1;   // largest qd: bin <= L - 3 (linear: L - 2)
          // Each word is its value times a 0/1 mask in packed f16 arithmetic (x * 1 and x * 0 are exact
          // for the non-negative finite weights, and at most one term of a sum is non-zero), so the
          // placement runs on the FMA pipe instead of compare/select chains on the busier ALU pipe.
          // wp >> 1 is (kKnotBias >> 2) + qd with qd < 64; times 0x10001 that is the f16 pair with bit
          // patterns qd (low: a subnormal, or zero) and (kKnotBias >> 18) + qd (high): distinct per qd.
          // f16 comparisons do not flush subnormals (this file is not built with a flush-to-zero flag).
          const uint32_t q2 = (wp >> 1) * 0x00010001u;
          const __half2 qh = *reinterpret_cast<const __half2*>(&q2);
          const __half2 h0 = *reinterpret_cast<const __half2*>(&y0), h1 = *reinterpret_cast<const __half2*>(&y1),
                        h2 = *reinterpret_cast<const __half2*>(&y2);
          __half2 m[HLP / 2];
#pragma unroll
          for (int i = 0; i < HLP / 2; ++i) {
            const uint32_t ci2 = (((kKnotBias >> 18) + (uint32_t)i) << 16) | (uint32_t)i;
            m[i] = i <= kLastPair ? __heq2(qh, *reinterpret_cast<const __half2*>(&ci2)) : __float2half2_rn(0.0f);
          }
#pragma unroll
          for (int i = 0; i < HLP / 2; ++i) {
            __half2 e = __hmul2(m[i], h0);
            if (i > 0) e = __hfma2(m[i - 1], h2, e);
            const __half2 o = __hmul2(m[i], h1);
            W[2 * i] = *reinterpret_cast<const uint32_t*>(&e);
            W[2 * i + 1] = *reinterpret_cast<const uint32_t*>(&o);
          }
          if ((qq & 1) && (qq & ~1) >= NSTH)            // a pair of mask-placed keys is complete
            tmem_st_words<2 * HLP>(lane_addr + (uint32_t)((half * kHalfKeys + (qq & ~1)) * HLP), WP[qq >> 1]);
        }
        // (All four keys in one 32- and one 16-column store was slower: 0.909 against 0.890 ms.)
#pragma unroll
        for (int pp = 0; 2 * pp < NSTH; ++pp)            // pairs with a staged key: their loads have landed by now
          tmem_st_words<2 * HLP>(lane_addr + (uint32_t)((half * kHalfKeys + 2 * pp) * HLP), WP[pp]);
        tmem_wait_st();
        tc_fence_before();
        mbar_arrive_warp(full + grp * 2 + half);
      }
      if (arow && valid) *reinterpret_cast<uint4*>(arow + ci * kChunkKeys) = make_uint4(aw[0], aw[1], aw[2], aw[3]);
    }
    // epilogue: accumulator -> float32 partial of this key split
    mbar_wait(done + grp, 0, wc);
    tc_fence_after();
    float* prow = P.partial + ((size_t)blockIdx.y * P.N + (valid ? n : 0)) * r;
    const uint32_t daddr = lane_addr + (uint32_t)(kChunkKeys * HLP);
    for (int c0 = 0; c0 < r; c0 += 16) {
      float v[16];
      tmem_ld16(daddr + c0, v);
      if (valid) {
#pragma unroll
        for (int i = 0; i < 16; i += 4)
          *reinterpret_cast<float4*>(prow + c0 + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
      }
    }
    tc_fence_before();
  } else if (warp < 5 * GROUPS) {
    // ------------------------------------------------------------------ MMA issue, one warp per token group
    // (one thread cannot issue N = r MMAs faster than about one per 45 cycles)
    if (elect_one()) {
      const int grp = warp - 4 * GROUPS;
      const uint32_t idesc = instr_desc(0, 0, 0, 1, 128, r);
      const uint32_t b_hi = desc_hi(P.b_sbo);
      const uint32_t b_step = (2u * (uint32_t)(r / 8) * 128u) >> 4;          // per K=16 step
      const uint32_t a_addr0 = tmem_base + (uint32_t)grp * grp_cols;
      const uint32_t d_addr = a_addr0 + (uint32_t)(kChunkKeys * HLP);
      for (int ci = 0; ci < nch; ++ci) {
        const int cs = ci % CS;
        bool drain = mbar_wait(cfull + cs, (uint32_t)(ci / CS) & 1u, wc);
        uint32_t b_lo = desc_lo(smem_u32(c_base + (size_t)cs * c_bytes), P.b_lbo);
        uint32_t a_addr = a_addr0;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          drain = drain || mbar_wait(full + grp * 2 + half, (uint32_t)ci & 1u, wc);
          if (drain) break;                          // draining: issue nothing more
          tc_fence_after();
#pragma unroll
          for (int ks = 0; ks < kHalfSteps; ++ks) {     // 8 columns of A (16 K elements) per step
            umma_f16_ta(d_addr, a_addr, b_lo, b_hi, idesc, (ci > 0 || half > 0 || ks > 0) ? 1u : 0u);
            a_addr += 8u;
            b_lo += b_step;
          }
          umma_commit(empty + grp * 2 + half);
        }
        if (drain) break;
        umma_commit(cempty + cs);
      }
      umma_commit(done + grp);
    }
  } else {
    // ------------------------------------------------------------------ code-table loader
    if (elect_one()) {
      const uint8_t* src = reinterpret_cast<const uint8_t*>(P.cimg) + (size_t)chunk_begin * c_bytes;
      for (int ci = 0; ci < nch; ++ci) {
        const int s = ci % CS;
        if (ci >= CS)
          mbar_wait(cempty + s, (uint32_t)((ci / CS) - 1) & 1u, wc);
        if (*abort_flag) break;
        if (ci == 0 && P.skip_copy) continue;      // test hook: nothing ever completes cfull[0]
        mbar_arrive_expect_tx(cfull + s, c_bytes);
        bulk_g2s(c_base + (size_t)s * c_bytes, src + (size_t)ci * c_bytes, c_bytes, cfull + s);
      }
      if (*abort_flag) {
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) {}
      }
    }
  }
  __syncthreads();
  if (warp == 5 * GROUPS) {
    for (int i = 0; i < GROUPS; ++i) mbar_wait_drain(done + i, 0, P.wait_cycles);
    tc_fence_after();
    tmem_free(tmem_base, tmem_cols);
  }
}

template <int G, int HL, int ACT, bool LIN>
cudaError_t fwd_launch_one(const FwdParams& P, dim3 grid, size_t smem, cudaStream_t stream) {
  constexpr int hlp = (HL + 1) & ~1;
  if constexpr (G * (kChunkKeys * hlp + 16) <= 512)
    return launch_chained<tc_forward_ta_kernel<G, HL, ACT, LIN>>(grid, 160 * G + 32, smem, stream, P);
  else
    return cudaErrorInvalidValue;
}

template <int ACT, bool LIN>
cudaError_t fwd_launch(int groups, int words, const FwdParams& P, dim3 grid, size_t smem, cudaStream_t stream) {
#define SKV_FWD_WORDS(HL_)                                                              \
  if (words == HL_) {                                                                   \
    if (groups == 4) return fwd_launch_one<4, HL_, ACT, LIN>(P, grid, smem, stream);    \
    if (groups == 3) return fwd_launch_one<3, HL_, ACT, LIN>(P, grid, smem, stream);    \
    if (groups == 2) return fwd_launch_one<2, HL_, ACT, LIN>(P, grid, smem, stream);    \
    return fwd_launch_one<1, HL_, ACT, LIN>(P, grid, smem, stream);                     \
  }
  SKV_FWD_WORDS(4) SKV_FWD_WORDS(6) SKV_FWD_WORDS(8) SKV_FWD_WORDS(11) SKV_FWD_WORDS(12)
  SKV_FWD_WORDS(16) SKV_FWD_WORDS(21) SKV_FWD_WORDS(22) SKV_FWD_WORDS(32)
#undef SKV_FWD_WORDS
  return cudaErrorInvalidValue;
}

}  // namespace tc
}  // namespace skv
