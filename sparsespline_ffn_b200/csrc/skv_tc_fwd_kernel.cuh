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
#include "skv_tma.cuh"

namespace skv {
namespace tc {

constexpr int kMaxCStages = 8;

struct FwdParams {
  const __nv_bfloat16* z;
  int64_t zs;
  __nv_bfloat16* act_out;
  int64_t as;
  const __half* cimg;       // [h/8][8*LP/8][r/8][8][8] f16 image of C, LP = 4 F rows per key
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

// Groups of four knot rows per key (see the kernel) the kernel is instantiated for: enough for 2 F - 1 words.
inline int fwd_fold(int L) {
  const int hl = (L + 1) / 2;
  for (int v : {4, 6, 8, 10, 12, 18})
    if (hl <= 2 * v - 1) return v;
  return 0;
}
// Tensor-memory columns of a token group: Phi of 8 keys, its metadata in two halves, the accumulator.
__host__ __device__ constexpr int fwd_meta_cols(int F) { return (F / 2 + 1) & ~1; }
inline int fwd_max_groups(int F, int r, bool split) {
  const int g = 512 / (kChunkKeys * F * (split ? 2 : 1) + 2 * fwd_meta_cols(F) + r);
  return g > 4 ? 4 : g;
}

// ---------------------------------------------------------------------------------------------
// Launch shape: grid = (token tiles of 128*GROUPS tokens, key splits).  Each producer thread owns a token: it
// builds the Phi row segment of a key in registers and writes it with tcgen05.st into its own tensor-memory
// lane; the MMA takes A from tensor memory and only the code-table chunk (B) from shared memory.  Nothing has
// to be cleared: a row segment is overwritten completely every chunk.
//
// Sparse A.  Of a key's L knot rows a token has weights on three consecutive ones, which always lie in two
// neighbouring f16x2 words w, w + 1 (rows 2w, 2w + 1).  The table image orders a key's rows in F groups of four, group f
// = words f and f + F - 1, so that the two words fall into neighbouring groups whichever they are: groups w, w + 1 as
// their first halves, or (from w = F - 1 on) groups w - F + 1, w - F + 2 as their second.  That is the 2:4 pattern of
// the sparse MMA: a key is F words of A instead of 2 F (tensor-memory writes, words to place and MMAs all halve), and its
// metadata is one bit per key, "first or second halves": nibbles 0x4 (elements 0, 1) or 0xE (elements 2, 3).
// Metadata layout for 16-bit types: the 32-bit word of lane l, K step of 32: lanes with bit 3 clear hold elements 0..15 of
// rows l and l + 8 (low, high half), lanes with bit 3 set elements 16..31 of rows l - 8 and l; hence one shuffle.
//
// Bound: instruction issue of the producers and the load/store data path, which also carries the tensor-memory stores.
// Tensor-memory columns per token group: 8*F for A, written and consumed in two halves of 4 keys so that the MMAs of
// one run while the other is built, the metadata of the halves, r for the accumulator.
// ---------------------------------------------------------------------------------------------
// Keys of each half chunk (of four) whose words are placed through a staging row in shared memory: two stores at the
// dynamic position, F loads, two clearing stores.  The rows of a warp are interleaved by lane, so the bank of
// every access is the lane and nothing conflicts, whatever the knot intervals are.  The other keys are placed by 0/1 masks in
// packed f16 arithmetic.  0 / 1 / 2 / 4 staged keys: 0.823 / 0.801 / 0.824 / 0.925 ms at the d20 shape (0.876 with a dense
// A); with all four the load/store data path is 87 % busy.
constexpr int kStagedPerHalf = 1;

// Chunks whose MMAs follow one another in an accumulator of the SPLIT cases; what they gave is then added to the partial in
// float32.  The tensor core cuts a sum off at the accumulator's last bit, always towards zero, so the error grows with the
// number of MMAs and does not average out: 65536 x 5113, r = 32, error of delta against 64 bits with every chunk
// in one accumulator 1.8e-5 (2.6e-5 where all summands are positive), with 16 chunks 2.3e-6, with 8 1.2e-6 (1.4e-6); the call 1.41,
// 1.43 and 1.47 ms.  (Single f16 operands are off by 2e-4 already.)
constexpr int kSplitChain = 8;

// SPLIT: the weights' remainders follow the weights, in columns of their own and with the same metadata.
template <int GROUPS, int F, int ACT, bool LIN, bool SPLIT>
__global__ void __launch_bounds__(160 * GROUPS + 32, 1) tc_forward_kernel(const FwdParams P) {
  extern __shared__ __align__(128) uint8_t smem[];
  constexpr int kHalfKeys = kChunkKeys / 2;
  constexpr int kHalfWords = kHalfKeys * F;                        // words of A per half chunk
  constexpr int kHalfSteps = kHalfWords / 8;                       // MMAs (K = 32 rows of the table) per half chunk
  constexpr int kMeta = fwd_meta_cols(F);
  constexpr int kParts = SPLIT ? 2 : 1;
  constexpr int NSTH = SPLIT ? 0 : kStagedPerHalf;
  constexpr int SW = F + 1;                                        // staging words per thread (one spare, see LIN)
  const int r = P.r;
  const uint32_t c_bytes = (uint32_t)(kChunkKeys * 4 * F * r * 2);
  const int CS = P.cstages;
  uint8_t* c_base = smem;                                          // [cstage][c_bytes]
  uint8_t* stage_base = c_base + (size_t)CS * c_bytes;             // [warp][SW][32 lanes]
  uint64_t* bars = reinterpret_cast<uint64_t*>(stage_base + (size_t)128 * GROUPS * SW * 4);
  uint64_t* full = bars;                          // [group][half]  producers -> MMA
  uint64_t* empty = full + 2 * GROUPS;            // [group][half]  MMA -> producers
  uint64_t* cfull = empty + 2 * GROUPS;           // [cstage]       TMA -> MMA
  uint64_t* cempty = cfull + kMaxCStages;       // [cstage]       MMA -> TMA
  uint64_t* done = cempty + kMaxCStages;        // [group]
  uint64_t* part = done + GROUPS;               // [group]        MMA -> producers: kSplitChain chunks are complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(part + GROUPS);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const WaitCtx wc{abort_flag, P.status, kStatusTimeoutFwd, P.wait_cycles};

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int chunk_begin = blockIdx.y * P.chunks_per_split;
  const int nch = min(P.chunks_per_split, P.chunks_total - chunk_begin);
  const int64_t tile_base = (int64_t)blockIdx.x * (128 * GROUPS);
  const uint32_t grp_cols = (uint32_t)(kParts * kChunkKeys * F + 2 * kMeta + r);
  uint32_t tmem_cols = 32;
  while (tmem_cols < GROUPS * grp_cols) tmem_cols <<= 1;

  if (tid == 0) {
    for (int i = 0; i < 2 * GROUPS; ++i) { mbar_init(full + i, 4); mbar_init(empty + i, 1); }
    for (int i = 0; i < 2 * GROUPS; ++i) mbar_init(done + i, 1);
    for (int i = 0; i < kMaxCStages; ++i) { mbar_init(cfull + i, 1); mbar_init(cempty + i, GROUPS); }
    *abort_flag = 0;
    mbar_init_fence();
  }
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
    // word w of this thread's staging row; the word index carries the bias kWordBias
    const uint32_t srow = smem_u32(stage_base) + (uint32_t)(warp * SW * 128 + lane * 4);
    const uint32_t srow_biased = srow - (kWordBias << 7);
    const bool up = (lane & 8) != 0;
    const uint32_t sel_send = up ? 0x5410u : 0x7632u;               // halves of two metadata words the other row needs
    const uint32_t sel_0 = up ? 0x3254u : 0x5410u, sel_1 = up ? 0x3276u : 0x7610u;
    // accumulator -> float32 partial of this key split; `more`: added to what this thread has put there
    auto drain_acc = [&](bool more) {
      const int64_t n4 = n & ~(int64_t)3;
      float* prow = P.partial + ((size_t)blockIdx.y * P.N + n4) * r + 4 * (lane & 3);
      const uint32_t daddr = lane_addr + (uint32_t)(kParts * kChunkKeys * F + 2 * kMeta);
      for (int c0 = 0; c0 < r; c0 += 16) {
        float v[16];
        tmem_ld16(daddr + c0, v);
        quad_transpose(v);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (n4 + j < P.N) {
            float* dst = prow + (size_t)j * r + c0;
            const float* q = v + 4 * j;
            if (SPLIT && more) red_add4(dst, q[0], q[1], q[2], q[3]);
            else *reinterpret_cast<float4*>(dst) = make_float4(q[0], q[1], q[2], q[3]);
          }
        }
      }
    };
    for (int ci = 0; ci < nch; ++ci) {
      if constexpr (SPLIT) {
        if (ci > 0 && ci % kSplitChain == 0) {           // the MMAs of this chunk wait for its words, hence for this
          mbar_wait(part + grp, (uint32_t)(ci / kSplitChain - 1) & 1u, wc);
          tc_fence_after();
          drain_acc(ci > kSplitChain);
          tc_fence_before();
        }
      }
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
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t W[kHalfWords];
        uint32_t meta[kHalfSteps];
#pragma unroll
        for (int j = 0; j < kHalfSteps; ++j) meta[j] = 0x44444444u;
        uint32_t x0[kHalfKeys], x1[kHalfKeys], wp[kHalfKeys], r0[kHalfKeys], r1[kHalfKeys];
#pragma unroll
        for (int pq = 0; pq < kHalfKeys / 2; ++pq) {
          // knot interval and weights, two keys (one packed z word) at a time; rows past N read z = 0 and their
          // accumulator rows are never stored
          uint32_t a0[2], a1[2], aw2[2];
          phi_pair_words2<LIN, SPLIT>(zw[half * (kHalfKeys / 2) + pq], P.g, a0, a1, aw2, r0 + 2 * pq, r1 + 2 * pq);
#pragma unroll
          for (int e = 0; e < 2; ++e) { x0[2 * pq + e] = a0[e]; x1[2 * pq + e] = a1[e]; wp[2 * pq + e] = aw2[e]; }
        }
#pragma unroll
        for (int q = 0; q < kHalfKeys; ++q) {
          // fold: first or second halves, and the word index within the F groups
          const bool hi = wp[q] >= kWordBias + (uint32_t)(F - 1);
          if (hi) wp[q] -= (uint32_t)(F - 1);
#pragma unroll
          for (int j = 0; j < kHalfSteps; ++j) {                   // nibbles q * F .. q * F + F - 1 of the half's 4 F
            uint32_t m = 0u;
#pragma unroll
            for (int i = 0; i < F; ++i)
              if ((q * F + i) / 8 == j) m |= 0xAu << (4 * ((q * F + i) % 8));
            if (m != 0u && hi) meta[j] |= m;
          }
          if (q < NSTH) {
            // (the linear spline's last interval may store a zero word in the spare one)
            const uint32_t pos = srow_biased + (wp[q] << 7);
            sts32(pos, x0[q]);
            sts32(pos + 128u, x1[q]);
#pragma unroll
            for (int i = 0; i < F; ++i) W[q * F + i] = lds32(srow + (uint32_t)i * 128u);
            sts32(pos, 0u);
            sts32(pos + 128u, 0u);
          }
        }
        auto place = [&](int q, uint32_t v0, uint32_t v1) {
          // Placement at word-pair granularity: the word index is 2 * qd + s.  The two words land in pair qd as
          // (v0, v1) when s = 0, or as (0, v0) there and (v1, 0) in pair qd + 1 when s = 1.  Each word is its value times
          // a 0/1 mask in packed f16 arithmetic (x * 1 and x * 0 are exact for finite weights, and at
          // most one term of a sum is non-zero), which runs on the FMA pipe; compare/select chains would run on the ALU
          // pipe.  The biased index >> 1 times 0x10001 is an f16 pair with bit patterns qd (low: a subnormal, or zero) and
          // (kKnotBias >> 18) + qd (high), distinct per qd; f16 comparisons do not flush subnormals.
          const bool odd = (wp[q] & 1u) != 0u;
          const uint32_t y0 = odd ? 0u : v0, y1 = odd ? v0 : v1, y2 = odd ? v1 : 0u;
          const uint32_t q2 = (wp[q] >> 1) * 0x00010001u;
          const __half2 qh = *reinterpret_cast<const __half2*>(&q2);
          const __half2 h0 = *reinterpret_cast<const __half2*>(&y0), h1 = *reinterpret_cast<const __half2*>(&y1),
                        h2 = *reinterpret_cast<const __half2*>(&y2);
          __half2 m[F / 2];
#pragma unroll
          for (int i = 0; i < F / 2; ++i) {
            const uint32_t c2 = (((kKnotBias >> 18) + (uint32_t)i) << 16) | (uint32_t)i;
            m[i] = __heq2(qh, *reinterpret_cast<const __half2*>(&c2));
          }
#pragma unroll
          for (int i = 0; i < F / 2; ++i) {
            __half2 e = __hmul2(m[i], h0);
            if (i > 0) e = __hfma2(m[i - 1], h2, e);
            const __half2 o = __hmul2(m[i], h1);
            W[q * F + 2 * i] = *reinterpret_cast<const uint32_t*>(&e);
            W[q * F + 2 * i + 1] = *reinterpret_cast<const uint32_t*>(&o);
          }
        };
#pragma unroll
        for (int q = NSTH; q < kHalfKeys; ++q) place(q, x0[q], x1[q]);
#pragma unroll
        for (int j = 0; j < kHalfSteps; j += 2) {
          const int j1 = j + 1 < kHalfSteps ? j + 1 : j;
          const uint32_t got = __shfl_xor_sync(0xffffffffu, __byte_perm(meta[j], meta[j1], sel_send), 8);
          const uint32_t m1 = __byte_perm(meta[j1], got, sel_1);
          meta[j] = __byte_perm(meta[j], got, sel_0);
          if (j1 != j) meta[j1] = m1;
        }
        if (ci > 0) {
          mbar_wait(empty + grp * 2 + half, (uint32_t)(ci - 1) & 1u, wc);
          tc_fence_after();
        }
        tmem_st_words<kHalfWords>(lane_addr + (uint32_t)(half * kHalfWords), W);
        tmem_st_words<kHalfSteps>(lane_addr + (uint32_t)(kParts * kChunkKeys * F + half * kMeta), meta);
        if constexpr (SPLIT) {
#pragma unroll
          for (int q = 0; q < kHalfKeys; ++q) place(q, r0[q], r1[q]);
          tmem_st_words<kHalfWords>(lane_addr + (uint32_t)(kChunkKeys * F + half * kHalfWords), W);
        }
        tmem_wait_st();
        tc_fence_before();
        mbar_arrive_warp(full + grp * 2 + half);
      }
      if (arow && valid) *reinterpret_cast<uint4*>(arow + ci * kChunkKeys) = make_uint4(aw[0], aw[1], aw[2], aw[3]);
    }
    mbar_wait(done + grp, 0, wc);
    tc_fence_after();
    drain_acc(nch > kSplitChain);
    tc_fence_before();
  } else if (warp < 5 * GROUPS) {
    // ------------------------------------------------------------------ MMA issue, one warp per token group
    // (one thread cannot issue N = r MMAs faster than about one per 45 cycles)
    if (elect_one()) {
      const int grp = warp - 4 * GROUPS;
      const uint32_t idesc = instr_desc(0, 0, 0, 1, 128, r) | kSparse;
      const uint32_t b_hi = desc_hi(P.b_sbo);
      const uint32_t b_step = (4u * (uint32_t)(r / 8) * 128u) >> 4;          // per K=32 step
      const uint32_t a_addr0 = tmem_base + (uint32_t)grp * grp_cols;
      const uint32_t m_addr0 = a_addr0 + (uint32_t)(kParts * kChunkKeys * F);
      const uint32_t d_addr = m_addr0 + (uint32_t)(2 * kMeta);
      for (int ci = 0; ci < nch; ++ci) {
        const int cs = ci % CS;
        const bool fresh = SPLIT ? ci % kSplitChain == 0 : ci == 0;      // the accumulator starts anew
        if (SPLIT && fresh && ci > 0) umma_commit(part + grp);
        bool drain = mbar_wait(cfull + cs, (uint32_t)(ci / CS) & 1u, wc);
        uint32_t b_lo = desc_lo(smem_u32(c_base + (size_t)cs * c_bytes), P.b_lbo);
        uint32_t a_addr = a_addr0;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          drain = drain || mbar_wait(full + grp * 2 + half, (uint32_t)ci & 1u, wc);
          if (drain) break;                          // draining: issue nothing more
          tc_fence_after();
#pragma unroll
          for (int ks = 0; ks < kHalfSteps; ++ks) {     // 8 columns of A (16 kept of 32 K elements) per step
#pragma unroll
            for (int p = 0; p < kParts; ++p)
              umma_f16_sparse_ta(d_addr, a_addr + (uint32_t)(p * kChunkKeys * F), b_lo, b_hi,
                                 m_addr0 + (uint32_t)(half * kMeta + (ks & ~1)), idesc | (uint32_t)(ks & 1),
                                 (!fresh || half > 0 || ks > 0 || p > 0) ? 1u : 0u);
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

template <int G, int F, int ACT, bool LIN, bool SPLIT>
cudaError_t fwd_launch_one(const FwdParams& P, dim3 grid, size_t smem, cudaStream_t stream) {
  if constexpr (G * ((SPLIT ? 2 : 1) * kChunkKeys * F + 2 * fwd_meta_cols(F) + 16) <= 512)
    return launch_chained<tc_forward_kernel<G, F, ACT, LIN, SPLIT>>(grid, 160 * G + 32, smem, stream, P);
  else
    return cudaErrorInvalidValue;
}

template <int ACT, bool LIN, bool SPLIT>
cudaError_t fwd_launch(int groups, int fold, const FwdParams& P, dim3 grid, size_t smem, cudaStream_t stream) {
#define SKV_FWD_FOLD(F_)                                                               \
  if (fold == F_) {                                                                    \
    if (groups == 4) return fwd_launch_one<4, F_, ACT, LIN, SPLIT>(P, grid, smem, stream);    \
    if (groups == 3) return fwd_launch_one<3, F_, ACT, LIN, SPLIT>(P, grid, smem, stream);    \
    if (groups == 2) return fwd_launch_one<2, F_, ACT, LIN, SPLIT>(P, grid, smem, stream);    \
    return fwd_launch_one<1, F_, ACT, LIN, SPLIT>(P, grid, smem, stream);                     \
  }
  SKV_FWD_FOLD(4) SKV_FWD_FOLD(6) SKV_FWD_FOLD(8) SKV_FWD_FOLD(10) SKV_FWD_FOLD(12) SKV_FWD_FOLD(18)
#undef SKV_FWD_FOLD
  return cudaErrorInvalidValue;
}

}  // namespace tc
}  // namespace skv
