// tcgen05 kernel for dz (token-major, like the forward):
//   S[n, (j,m)] = sum_c g[n,c] * T[j,m,c]   on the tensor cores (M = 128 tokens, N = 8L, K = r)
//   where T is the code table transformed along the knot axis so that the three-of-L selection
//   becomes a dense weighted sum with one saturating add per column:
//       T[j,0]   = C[j,1] - C[j,0]
//       T[j,m+1] = C[j,m] - 2 C[j,m+1] + C[j,m+2]      (m = 0..G-1),   T[j,L-1] = 0
//       dz_spline[n,j] = scale * 1[0 <= u <= G-1] * ( S[n,(j,0)] + sum_m sat(u_c - m) * S[n,(j,m+1)] )
//   (sat(u_c - m) is 1 below the token's knot interval, tau inside it and 0 above, which telescopes
//   to -(1-tau) C[bin] + (1-2tau) C[bin+1] + tau C[bin+2], the B-spline derivative weights.)
//   One thread per token reads its S row from tensor memory, adds the base-path term
//   g_a * phi'(z) and stores dz in bf16.
#pragma once

#include "skv_tc_prep.cuh"

namespace skv {
namespace tc {

struct DzParams {
  const __nv_bfloat16* z;
  int64_t zs;
  const __nv_bfloat16* g_act;
  int64_t gas;
  __nv_bfloat16* dz;
  int64_t dzs;
  const __half* gimg;
  const __half* timg;
  const uint32_t* amax_bits;
  int64_t N;
  int h, L, r;
  GridParams g;
  int act;
  float coef;                // lambda * scale
  int chunks_total, chunks_per_split;
  int tstages;               // depth of the transformed-table ring (2..kTStages)
  int dz_f32;                // dz is float32 [N][dzs] instead of bf16
  int32_t* status;
  long long wait_cycles;     // limit of every bounded wait, in clock cycles
};

// Tensor-memory loads of one key's S columns: the first NC of its LB blocks of 8 float32 columns of
// this warp's lanes (the padding columns are never read: the kernel's time follows the bytes it moves
// out of tensor memory, 4 * NC per pair).  The loads are issued without waiting; tmem_wait_key waits
// for all outstanding loads and ties the destination registers to the wait so that no use can be
// scheduled ahead of it.
template <int N> __device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t* r);
template <> __device__ __forceinline__ void tmem_ld_cols<8>(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
template <> __device__ __forceinline__ void tmem_ld_cols<4>(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr)
               : "memory");
}
template <> __device__ __forceinline__ void tmem_ld_cols<2>(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(taddr) : "memory");
}
template <> __device__ __forceinline__ void tmem_ld_cols<1>(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(r[0]) : "r"(taddr) : "memory");
}
template <> __device__ __forceinline__ void tmem_ld_cols<16>(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
      "[%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// All 8 * LB columns of the key, in as few instructions as possible (a load instruction costs more
// than the columns it moves: loading only the NC useful columns as 8 + 8 + 4 + 1 was slower, 1.16 ms
// against 1.11 ms at the d20 shape).
template <int LB, int NC>
__device__ __forceinline__ void tmem_ld_key(uint32_t taddr, uint32_t (&r)[LB][8]) {
  uint32_t* flat = &r[0][0];
  int o = 0;
#pragma unroll
  for (int i = 0; i < LB / 2; ++i) { tmem_ld_cols<16>(taddr + (uint32_t)o, flat + o); o += 16; }
  if constexpr ((LB & 1) != 0) tmem_ld_cols<8>(taddr + (uint32_t)o, flat + o);
}
template <int LB, int NC>
__device__ __forceinline__ void tmem_wait_key(uint32_t (&r)[LB][8]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int blk = 0; blk < LB; ++blk)
#pragma unroll
    for (int i = 0; i < 8; ++i) asm volatile("" : "+r"(r[blk][i]) : : "memory");
}

// S_0 + sum_m sat(uc - m) * S_{m+1} over the first NC of the 8*LB columns of one key.  Columns
// L-1 and up are padding (zero rows of the table image, and their weight sat(uc - m) is zero as
// well since uc <= G-1 < m); with NC = L-1 known at compile time they cost nothing.
// Columns are taken in aligned pairs with the packed two-wide float32 FMA of sm_100
// (fma.rn.f32x2): weight 1 for column 0, sat(uc - (m-1)) for column m.
template <int LB, int NC>
__device__ __forceinline__ float dz_key_sum(const uint32_t (&r)[LB][8], float uc) {
  unsigned long long acc2 = 0ull;                     // (0.0f, 0.0f)
  float tail = 0.0f;
#pragma unroll
  for (int blk = 0; blk < LB; ++blk) {
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      const int m = blk * 8 + i;
      if (m >= NC) continue;
      const float w0 = m == 0 ? 1.0f : __saturatef(uc - (float)(m - 1));
      if (m + 1 >= NC) {                              // last column of an odd count
        tail = w0 * __uint_as_float(r[blk][i]);
        continue;
      }
      const float w1 = __saturatef(uc - (float)m);
      unsigned long long w2, s2;
      asm("mov.b64 %0, {%1, %2};" : "=l"(w2) : "f"(w0), "f"(w1));
      asm("mov.b64 %0, {%1, %2};" : "=l"(s2) : "r"(r[blk][i]), "r"(r[blk][i + 1]));
      asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc2) : "l"(w2), "l"(s2));
    }
  }
  float a0, a1;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a0), "=f"(a1) : "l"(acc2));
  return (a0 + a1) + tail;
}

constexpr int kTStages = 4;

// RELU: the base path is ReLU^2 (compile-time, so that the code of the other activations stays
// out of the hot loop); otherwise P.act (identity or gelu) is evaluated at run time.
// LIN: the derivative of the linear spline is C[bin+1] - C[bin]; with the same table its column weights
// are the steps 1[bin >= m + 1] = sat(bin - m), so the only change is bin in the place of u_c.
template <int GROUPS, int LB, int NC, bool RELU, bool LIN>
__global__ void __launch_bounds__(128 * GROUPS + 64, 1) tc_dz_kernel(const DzParams P) {
  extern __shared__ __align__(128) uint8_t smem[];
  const int r = P.r;
  constexpr int LP = 8 * LB;                                         // padded knot columns per key
  const uint32_t g_bytes = (uint32_t)(128 * r * 2);
  const uint32_t t_bytes = (uint32_t)(kChunkKeys * LP * r * 2);
  constexpr uint32_t ncols = (uint32_t)(kChunkKeys * LP);            // S columns per group
  uint8_t* g_base = smem;                                             // [group][g_bytes]
  uint8_t* t_base = smem + (size_t)GROUPS * g_bytes;                  // [kTStages][t_bytes]
  const int TS = P.tstages;
  uint64_t* bars = reinterpret_cast<uint64_t*>(t_base + (size_t)TS * t_bytes);
  uint64_t* gfull = bars;                    // [1]
  uint64_t* tfull = gfull + 1;               // [kTStages]
  uint64_t* tempty = tfull + kTStages;       // [kTStages]
  uint64_t* sfull = tempty + kTStages;       // [GROUPS]  MMA -> consumers
  uint64_t* sempty = sfull + GROUPS;         // [GROUPS]  consumers -> MMA
  uint64_t* done = sempty + GROUPS;          // [1]       all MMAs of this CTA complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const WaitCtx wc{abort_flag, P.status, kStatusTimeoutDz, P.wait_cycles};

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int chunk_begin = blockIdx.y * P.chunks_per_split;
  const int nch = min(P.chunks_per_split, P.chunks_total - chunk_begin);
  const int64_t tile_base = (int64_t)blockIdx.x * (128 * GROUPS);
  uint32_t tmem_cols = 32;
  while (tmem_cols < GROUPS * ncols) tmem_cols <<= 1;

  if (tid == 0) {
    mbar_init(gfull, 1);
    for (int i = 0; i < kTStages; ++i) { mbar_init(tfull + i, 1); mbar_init(tempty + i, 1); }
    for (int i = 0; i < GROUPS; ++i) { mbar_init(sfull + i, 1); mbar_init(sempty + i, 4); }
    mbar_init(done, 1);
    *abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == 4 * GROUPS) tmem_alloc(tmem_slot, tmem_cols);
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch();
  pdl_wait();

  if (warp < 4 * GROUPS) {
    // ------------------------------------------------------------------ one thread per token
    const int grp = warp >> 2;
    const int t = tid & 127;
    const int64_t n = tile_base + grp * 128 + t;
    const bool valid = n < P.N;
    const int64_t nn = valid ? n : 0;
    const __nv_bfloat16* zrow = P.z + nn * P.zs + (int64_t)chunk_begin * kChunkKeys;
    const __nv_bfloat16* garow = P.g_act ? P.g_act + nn * P.gas + (int64_t)chunk_begin * kChunkKeys : nullptr;
    __nv_bfloat16* dzrow = P.dz + nn * P.dzs + (int64_t)chunk_begin * kChunkKeys;
    float gscale, ginv;
    pow2_scales(*P.amax_bits, gscale, ginv);
    float cscale, cinv;
    pow2_scales(P.amax_bits[kAmaxC], cscale, cinv);
    const float coef = P.coef * ginv * cinv;
    const int act = P.act;
    const uint32_t trow = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)grp * ncols;
    uint4 znext = valid && nch > 0 ? ld16(zrow) : make_uint4(0, 0, 0, 0);
    uint4 ganext = valid && nch > 0 && garow ? ld16(garow) : make_uint4(0, 0, 0, 0);

    for (int ci = 0; ci < nch; ++ci) {
      const uint4 zc = znext, gac = ganext;
      if (ci + 1 < nch && valid) {
        znext = ld16(zrow + (ci + 1) * kChunkKeys);
        if (garow) ganext = ld16(garow + (ci + 1) * kChunkKeys);
      }
      const uint32_t zw[4] = {zc.x, zc.y, zc.z, zc.w};
      const uint32_t gw[4] = {gac.x, gac.y, gac.z, gac.w};
      uint32_t bufa[LB][8], bufb[LB][8];
      float outv[kChunkKeys];
      mbar_wait(sfull + grp, (uint32_t)ci & 1u, wc);
      tc_fence_after();
      tmem_ld_key<LB, NC>(trow, bufa);
#pragma unroll
      for (int q = 0; q < kChunkKeys; ++q) {
        // the loads of key q are in flight; wait, start the loads of key q+1, then do key q's math
        if (q & 1) tmem_wait_key<LB, NC>(bufb); else tmem_wait_key<LB, NC>(bufa);
        if (q + 1 < kChunkKeys) {
          if (q & 1) tmem_ld_key<LB, NC>(trow + (uint32_t)((q + 1) * LP), bufa);
          else tmem_ld_key<LB, NC>(trow + (uint32_t)((q + 1) * LP), bufb);
        }
        const float zz = (q & 1) ? bf_hi(zw[q >> 1]) : bf_lo(zw[q >> 1]);
        // same u and the same single-comparison range test as knot_of
        const float u = __fmaf_rn(__fsub_rn(zz, P.g.lo), P.g.scale, 0.0f);
        const bool active = __float_as_uint(u) <= __float_as_uint(P.g.Gm1f);
        float uc = fminf(fmaxf(u, 0.0f), P.g.Gm1f);
        if constexpr (LIN) uc = __fsub_rn(__fadd_rd(uc, 8388608.0f), 8388608.0f);
        const float acc = (q & 1) ? dz_key_sum<LB, NC>(bufb, uc) : dz_key_sum<LB, NC>(bufa, uc);
        float o = active ? coef * acc : 0.0f;
        if (garow) {
          const float ga = (q & 1) ? bf_hi(gw[q >> 1]) : bf_lo(gw[q >> 1]);
          const float dphi = RELU ? 2.0f * fmaxf(zz, 0.0f) : act_grad(zz, act);
          o = fmaf(ga, dphi, o);
        }
        outv[q] = o;
      }
      // (Handing the S columns back two keys earlier, with the loads running two keys ahead in a third
      // register buffer, was measured slower: 1.14 ms against 1.11 ms at the d20 shape.)
      tc_fence_before();
      mbar_arrive_warp(sempty + grp);
      if (valid) {
        if (P.dz_f32) {
          float* o = reinterpret_cast<float*>(P.dz) + nn * P.dzs + (int64_t)(chunk_begin + ci) * kChunkKeys;
          *reinterpret_cast<float4*>(o) = make_float4(outv[0], outv[1], outv[2], outv[3]);
          *reinterpret_cast<float4*>(o + 4) = make_float4(outv[4], outv[5], outv[6], outv[7]);
        } else {
          *reinterpret_cast<uint4*>(dzrow + ci * kChunkKeys) =
              make_uint4(pack_bf2(outv[0], outv[1]), pack_bf2(outv[2], outv[3]), pack_bf2(outv[4], outv[5]),
                         pack_bf2(outv[6], outv[7]));
        }
      }
    }
  } else if (warp == 4 * GROUPS) {
    // ------------------------------------------------------------------ MMA issue
    if (lane == 0) {
      mbar_wait(gfull, 0, wc);
      const uint32_t rb = (uint32_t)(r / 8) * 128u;          // bytes between 8-row groups of the T image
      const uint32_t a_hi = desc_hi(128u), b_hi = desc_hi(rb);
      // The groups are served in a fixed order.  (Serving whichever group has released its S columns
      // first, by polling both, was measured slower: 1.32 ms against 1.21 ms at the d20 shape.)
      for (int ci = 0; ci < nch; ++ci) {
        const int s = ci % TS;
        bool drain = mbar_wait(tfull + s, (uint32_t)(ci / TS) & 1u, wc);
        const uint32_t b_addr = smem_u32(t_base + (size_t)s * t_bytes);
        for (int grp = 0; grp < GROUPS && !drain; ++grp) {
          if (ci > 0) drain = mbar_wait(sempty + grp, (uint32_t)(ci - 1) & 1u, wc);
          if (drain) break;                          // draining: issue nothing more
          tc_fence_after();
          const uint32_t a_lo0 = desc_lo(smem_u32(g_base + (size_t)grp * g_bytes), 2048u);
          for (uint32_t c0 = 0; c0 < ncols; c0 += 256) {
            const uint32_t npiece = min(256u, ncols - c0);
            const uint32_t idesc = instr_desc(0, 0, 0, 0, 128, (int)npiece);
            uint32_t a_lo = a_lo0;
            uint32_t b_lo = desc_lo(b_addr + (c0 / 8) * rb, 128u);
            const uint32_t d_addr = tmem_base + (uint32_t)grp * ncols + c0;
            for (int ks = 0; ks < r / 16; ++ks) {
              umma_f16_split(d_addr, a_lo, a_hi, b_lo, b_hi, idesc, ks > 0 ? 1u : 0u);
              a_lo += 4096u >> 4;
              b_lo += 256u >> 4;
            }
          }
          umma_commit(sfull + grp);
        }
        if (drain) break;
        umma_commit(tempty + s);
      }
      umma_commit(done);
    }
  } else {
    // ------------------------------------------------------------------ loader
    if (lane == 0) {
      mbar_arrive_expect_tx(gfull, GROUPS * g_bytes);
      for (int grp = 0; grp < GROUPS; ++grp)
        bulk_g2s(g_base + (size_t)grp * g_bytes,
                 reinterpret_cast<const uint8_t*>(P.gimg) + (size_t)(blockIdx.x * GROUPS + grp) * g_bytes, g_bytes,
                 gfull);
      const uint8_t* src = reinterpret_cast<const uint8_t*>(P.timg) + (size_t)chunk_begin * t_bytes;
      for (int ci = 0; ci < nch; ++ci) {
        const int s = ci % TS;
        if (ci >= TS)
          mbar_wait(tempty + s, (uint32_t)((ci / TS) - 1) & 1u, wc);
        if (*abort_flag) break;
        mbar_arrive_expect_tx(tfull + s, t_bytes);
        bulk_g2s(t_base + (size_t)s * t_bytes, src + (size_t)ci * t_bytes, t_bytes, tfull + s);
      }
      if (*abort_flag) {
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) {}
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 4 * GROUPS) {
    mbar_wait_drain(done, 0, P.wait_cycles);
    tc_fence_after();
    tmem_free(tmem_base, tmem_cols);
  }
}

struct DzPlan { int groups, lb, splits, chunks_per_split, tstages; size_t smem; };

// NC_ = L - 1 useful columns per key for the knot counts in common use, all 8 * LB_ otherwise.
template <bool LIN>
cudaError_t dz_launch(const DzPlan& zp, int L, bool relu, const DzParams& P, dim3 grid, cudaStream_t stream) {
  const unsigned threads = 128 * zp.groups + 64;
#define SKV_DZ_CASE(G_, LB_, NC_, COND_)                                                                           \
  if (zp.groups == G_ && zp.lb == LB_ && (COND_))                                                                  \
    return relu ? launch_chained<tc_dz_kernel<G_, LB_, NC_, true, LIN>>(grid, threads, zp.smem, stream, P)         \
                : launch_chained<tc_dz_kernel<G_, LB_, NC_, false, LIN>>(grid, threads, zp.smem, stream, P);
  if constexpr (LIN) {
    SKV_DZ_CASE(2, 3, 20, L == 21)
  } else {
    SKV_DZ_CASE(2, 3, 21, L == 22) SKV_DZ_CASE(2, 2, 15, L == 16) SKV_DZ_CASE(1, 6, 41, L == 42)
  }
  SKV_DZ_CASE(2, 1, 8, true) SKV_DZ_CASE(2, 2, 16, true) SKV_DZ_CASE(2, 3, 24, true) SKV_DZ_CASE(2, 4, 32, true)
  SKV_DZ_CASE(1, 5, 40, true) SKV_DZ_CASE(1, 6, 48, true)
  SKV_DZ_CASE(1, 7, 56, true) SKV_DZ_CASE(1, 8, 64, true)
#undef SKV_DZ_CASE
  return cudaErrorInvalidValue;
}

}  // namespace tc
}  // namespace skv
