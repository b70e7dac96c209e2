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
#include "skv_tma.cuh"

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
  int rstages;               // boxes of z and g_act per token group (2 or 3)
  int dz_f32;                // dz is float32 [N][dzs] instead of bf16
  int32_t* status;
  long long wait_cycles;     // limit of every bounded wait, in clock cycles
};

// Tensor-memory loads of one key's S columns, LB blocks of 8 float32 columns of this warp's lanes.  The loads are issued
// without waiting; tmem_wait_key waits for all outstanding loads and ties the destination registers to the wait so that
// no use can be scheduled ahead of it.
template <int N> __device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t* r);
template <> __device__ __forceinline__ void tmem_ld_cols<8>(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
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
// All 8 * LB columns of the key, in as few instructions as possible: a load instruction costs more than the columns it
// moves.  (Measured on an earlier form of the kernel with one S block of 8 keys: the NC useful columns as 8 + 8 + 4 + 1
// took 1.16 ms at the d20 shape, all 24 as 16 + 8 1.11 ms.)
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
constexpr int kRowStages = 3;                 // boxes of z (and g_act) per token group, two where wide r needs the room
constexpr int kBoxChunks = kBoxKeys / kChunkKeys;

// Keys of one S block: S columns of a token group are computed and consumed in blocks of 4 keys (2 from 33 knot
// columns on), two blocks in tensor memory per group.
__host__ __device__ constexpr int dz_block_keys(int lb) { return lb <= 4 ? 4 : 2; }

// Launch shape: grid = (token tiles of 128*GROUPS tokens, key splits).  Per token group
//   eight consumer warps, two threads per token, one for each S buffer: z and g_act from their boxes, S from
//                        tensor memory, dz into the place of z
//   one warp (lane 0)    issues the group's S MMAs, a block ahead of the consumers
//   one warp (lane 0)    moves the group's boxes: loads of z and g_act, stores of dz
// and one loader warp for the transformed table.
//
// Bound: instruction issue of the consumers (71 instructions per 32 pairs at L = 22, 32 of them the saturating adds and the
// packed FMAs; 72 % of the issue slots).  What it took to get near it, at the d20 shape: MMAs issued by an elected thread (300-400 cycles
// per pair of MMAs before, 150 now), which is what makes smaller S blocks affordable; two blocks per group, so that
// one is computed while the other is read (with one block of 8 keys a group waited 670 cycles per chunk); a
// block given back as soon as its last key is in registers; the boxes' copies on a warp of their own (a consumer
// warp that also moved them held its group up by 680 cycles per box).
//
// RELU: the base path is ReLU^2 (compile-time, so that the code of the other activations stays
// out of the hot loop); otherwise P.act (identity or gelu) is evaluated at run time.
// LIN: the derivative of the linear spline is C[bin+1] - C[bin]; with the same table its column weights
// are the steps 1[bin >= m + 1] = sat(bin - m), so the only change is bin in the place of u_c.
// SPLIT: the table's values are two f16 (K runs over 2 r channels of it, over g twice).  A template case: a run-time count in the
// issuing thread's loop cost 4 % (0.964 -> 1.003 ms at the d20 shape).
template <int GROUPS, int LB, int NC, bool RELU, bool LIN, bool SPLIT>
__global__ void __launch_bounds__(320 * GROUPS + 32, 1)
    tc_dz_kernel(const DzParams P, const __grid_constant__ CUtensorMap map_z, const __grid_constant__ CUtensorMap map_ga,
                 const __grid_constant__ CUtensorMap map_dz) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* row_base = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);   // [group][rstages][z, g_act]
  const int RS = P.rstages;
  uint8_t* smem = row_base + (size_t)GROUPS * RS * 2 * kBoxBytes;
  const int r = P.r;
  constexpr int LP = 8 * LB;                                         // padded knot columns per key
  constexpr int KB = dz_block_keys(LB);
  constexpr int kParts = SPLIT ? 2 : 1;
  constexpr int NBLK = kChunkKeys / KB;                              // blocks per chunk
  constexpr bool DB = LB <= 4;                                       // two keys' columns in registers
  const uint32_t g_bytes = (uint32_t)(128 * r * 2);
  const uint32_t t_bytes = (uint32_t)(kChunkKeys * LP * r * 2 * kParts);
  constexpr uint32_t bcols = (uint32_t)(KB * LP);                    // columns of one S block
  uint8_t* g_base = smem;                                             // [group][g_bytes]
  uint8_t* t_base = smem + (size_t)GROUPS * g_bytes;                  // [kTStages][t_bytes]
  const int TS = P.tstages;
  uint64_t* bars = reinterpret_cast<uint64_t*>(t_base + (size_t)TS * t_bytes);
  uint64_t* gfull = bars;                       // [1]
  uint64_t* tfull = gfull + 1;                  // [kTStages]
  uint64_t* tempty = tfull + kTStages;          // [kTStages]           one arrival per group
  uint64_t* sfull = tempty + kTStages;          // [GROUPS][2]          MMA -> consumers
  uint64_t* sempty = sfull + 2 * GROUPS;        // [GROUPS][2]          consumers -> MMA
  uint64_t* done = sempty + 2 * GROUPS;         // [GROUPS]             all MMAs of the group complete
  uint64_t* zfull = done + GROUPS;              // [GROUPS][kRowStages] box landed
  uint64_t* zdone = zfull + GROUPS * kRowStages;  // [GROUPS][kRowStages] box consumed, dz in place
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(zdone + GROUPS * kRowStages);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const WaitCtx wc{abort_flag, P.status, kStatusTimeoutDz, P.wait_cycles};

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int chunk_begin = blockIdx.y * P.chunks_per_split;
  const int nch = min(P.chunks_per_split, P.chunks_total - chunk_begin);
  const int64_t tile_base = (int64_t)blockIdx.x * (128 * GROUPS);
  uint32_t tmem_cols = 32;
  while (tmem_cols < GROUPS * 2 * bcols) tmem_cols <<= 1;

  if (tid == 0) {
    mbar_init(gfull, 1);
    for (int i = 0; i < kTStages; ++i) { mbar_init(tfull + i, 1); mbar_init(tempty + i, GROUPS); }
    for (int i = 0; i < 2 * GROUPS; ++i) { mbar_init(sfull + i, 1); mbar_init(sempty + i, 4); }
    for (int i = 0; i < GROUPS; ++i) mbar_init(done + i, 1);
    for (int i = 0; i < GROUPS * kRowStages; ++i) { mbar_init(zfull + i, 1); mbar_init(zdone + i, 8); }
    *abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == 8 * GROUPS) tmem_alloc(tmem_slot, tmem_cols);
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch();
  pdl_wait();

  if (warp < 8 * GROUPS) {
    // ------------------------------------------------------------------ two threads per token, one per S buffer
    const int grp = warp >> 3, half = (warp >> 2) & 1;
    const int t = tid & 127;
    const int64_t n = tile_base + grp * 128 + t;
    const bool has_ga = P.g_act != nullptr;
    float gscale, ginv;
    pow2_scales(*P.amax_bits, gscale, ginv);
    float cscale, cinv;
    pow2_scales(P.amax_bits[kAmaxC], cscale, cinv);
    const float coef = P.coef * ginv * cinv;
    const int act = P.act;
    const uint32_t trow = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(grp * 2 + half) * bcols;
    uint64_t* sf = sfull + 2 * grp + half;
    uint64_t* se = sempty + 2 * grp + half;
    const uint32_t boxes = smem_u32(row_base + (size_t)grp * RS * 2 * kBoxBytes);
    int st = 0;
    uint32_t zpar = 0u;                                // stage and phase of the current box

    for (int ci = 0; ci < nch; ++ci) {
      if (ci % kBoxChunks == 0) mbar_wait(zfull + grp * kRowStages + st, zpar, wc);
      const uint32_t zaddr = boxes + (uint32_t)st * 2u * kBoxBytes + box_piece((uint32_t)t, (uint32_t)(ci % kBoxChunks)) +
                             (uint32_t)half * (KB == 4 ? 8u : 4u);
      // this thread's four keys of the chunk: two packed words of z and of g_act
      uint32_t zw[2], gw[2] = {0u, 0u};
      if constexpr (KB == 4) {
        lds64(zaddr, zw);
        if (has_ga) lds64(zaddr + kBoxBytes, gw);
      } else {
        zw[0] = lds32(zaddr);
        zw[1] = lds32(zaddr + 8u);
        if (has_ga) { gw[0] = lds32(zaddr + kBoxBytes); gw[1] = lds32(zaddr + kBoxBytes + 8u); }
      }
      float outv[4];
      uint32_t buf[DB ? 2 : 1][LB][8];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        constexpr int kAlt = DB ? 1 : 0;
        if (i % KB == 0) {                             // first key of a block
          mbar_wait(sf, (uint32_t)(ci * (4 / KB) + i / KB) & 1u, wc);
          tc_fence_after();
          tmem_ld_key<LB, NC>(trow, buf[(i & kAlt)]);
        } else if (!DB) {
          tmem_ld_key<LB, NC>(trow + (uint32_t)((i % KB) * LP), buf[0]);
        }
        tmem_wait_key<LB, NC>(buf[i & kAlt]);
        if (i % KB == KB - 1) {                        // the last key of the block is in registers: hand it back
          tc_fence_before();
          mbar_arrive_warp(se);
        } else if (DB) {
          tmem_ld_key<LB, NC>(trow + (uint32_t)((i % KB + 1) * LP), buf[(i + 1) & kAlt]);
        }
        const float zz = (i & 1) ? bf_hi(zw[i >> 1]) : bf_lo(zw[i >> 1]);
        // same u and the same single-comparison range test as knot_of
        const float u = __fmaf_rn(__fsub_rn(zz, P.g.lo), P.g.scale, 0.0f);
        const bool active = __float_as_uint(u) <= __float_as_uint(P.g.Gm1f);
        float uc = fminf(fmaxf(u, 0.0f), P.g.Gm1f);
        if constexpr (LIN) uc = __fsub_rn(__fadd_rd(uc, 8388608.0f), 8388608.0f);
        const float acc = dz_key_sum<LB, NC>(buf[i & kAlt], uc);
        float o = active ? coef * acc : 0.0f;
        if (has_ga) {
          const float ga = (i & 1) ? bf_hi(gw[i >> 1]) : bf_lo(gw[i >> 1]);
          const float dphi = RELU ? 2.0f * fmaxf(zz, 0.0f) : act_grad(zz, act);
          o = fmaf(ga, dphi, o);
        }
        outv[i] = o;
      }
      if (P.dz_f32) {
        if (n < P.N) {
          float* o = reinterpret_cast<float*>(P.dz) + n * P.dzs + (int64_t)(chunk_begin + ci) * kChunkKeys + half * KB;
          *reinterpret_cast<float2*>(o) = make_float2(outv[0], outv[1]);
          *reinterpret_cast<float2*>(o + (KB == 4 ? 2 : 4)) = make_float2(outv[2], outv[3]);
        }
      } else {
        // dz takes the place of the z words this thread has read
        const uint32_t w0 = pack_bf2(outv[0], outv[1]), w1 = pack_bf2(outv[2], outv[3]);
        if constexpr (KB == 4) sts64(zaddr, w0, w1);
        else { sts32(zaddr, w0); sts32(zaddr + 8u, w1); }
      }
      if (ci % kBoxChunks == kBoxChunks - 1 || ci + 1 == nch) {
        fence_async_smem();
        mbar_arrive_warp(zdone + grp * kRowStages + st);
        if (++st == RS) { st = 0; zpar ^= 1u; }
      }
    }
  } else if (warp < 9 * GROUPS) {
    // ------------------------------------------------------------------ MMA issue, one warp per token group
    if (elect_one()) {
      const int grp = warp - 8 * GROUPS;
      mbar_wait(gfull, 0, wc);
      const uint32_t rb = (uint32_t)(r * kParts / 8) * 128u;   // bytes between 8-row groups of the T image
      const uint32_t a_hi = desc_hi(128u), b_hi = desc_hi(rb);
      constexpr uint32_t idesc = instr_desc(0, 0, 0, 0, 128, (int)bcols);
      const uint32_t a_lo0 = desc_lo(smem_u32(g_base + (size_t)grp * g_bytes), 2048u);
      const uint32_t d0 = tmem_base + (uint32_t)grp * 2u * bcols;
      const int ksteps = r / 16;
      uint64_t* sf = sfull + 2 * grp;
      uint64_t* se = sempty + 2 * grp;
      bool drain = false;
      int ts = 0;
      uint32_t tpar = 0u;
      for (int ci = 0; ci < nch && !drain; ++ci) {
        drain = mbar_wait(tfull + ts, tpar, wc);
        uint32_t b_blk = desc_lo(smem_u32(t_base + (size_t)ts * t_bytes), 128u);
#pragma unroll
        for (int b = 0; b < NBLK; ++b) {
          const uint32_t use = (uint32_t)(ci * NBLK + b) >> 1;
          if (use > 0) drain = drain || mbar_wait(se + (b & 1), (use - 1u) & 1u, wc);
          if (drain) break;                            // draining: issue nothing more
          tc_fence_after();
          uint32_t b_lo = b_blk;
          const uint32_t d_addr = d0 + (uint32_t)(b & 1) * bcols;
#pragma unroll
          for (int part = 0; part < kParts; ++part) {
            uint32_t a_lo = a_lo0;
            for (int ks = 0; ks < ksteps; ++ks) {
              umma_f16_split(d_addr, a_lo, a_hi, b_lo, b_hi, idesc, ks + part > 0 ? 1u : 0u);
              a_lo += 4096u >> 4;
              b_lo += 256u >> 4;
            }
          }
          umma_commit(sf + (b & 1));
          b_blk += ((bcols / 8u) * rb) >> 4;
        }
        if (!drain) umma_commit(tempty + ts);
        if (++ts == TS) { ts = 0; tpar ^= 1u; }
      }
      umma_commit(done + grp);
    }
  } else if (warp < 10 * GROUPS) {
    // ------------------------------------------------------------------ boxes of z, g_act and dz, one warp per group
    if (elect_one()) {
      const int grp = warp - 9 * GROUPS;
      const int row0 = (int)(tile_base + grp * 128);
      const bool has_ga = P.g_act != nullptr, store = !P.dz_f32 && row0 < P.N;
      const int steps = (nch + kBoxChunks - 1) / kBoxChunks, key_begin = chunk_begin * kChunkKeys;
      auto load = [&](int step, int st) {
        uint8_t* box = row_base + (size_t)(grp * RS + st) * 2 * kBoxBytes;
        uint64_t* bar = zfull + grp * kRowStages + st;
        mbar_arrive_expect_tx(bar, has_ga ? 2 * kBoxBytes : kBoxBytes);
        tma_load_2d(box, &map_z, key_begin + step * kBoxKeys, row0, bar);
        if (has_ga) tma_load_2d(box + kBoxBytes, &map_ga, key_begin + step * kBoxKeys, row0, bar);
      };
      for (int i = 0; i < RS && i < steps; ++i) load(i, i);
      int st = 0;
      uint32_t par = 0u;
      for (int step = 0; step < steps; ++step) {
        if (mbar_wait(zdone + grp * kRowStages + st, par, wc)) break;
        if (store)
          tma_store_2d(&map_dz, row_base + (size_t)(grp * RS + st) * 2 * kBoxBytes, key_begin + step * kBoxKeys, row0);
        bulk_commit();
        bulk_wait_read<0>();                           // before the stage is loaded again, and before the CTA ends
        if (step + RS < steps) load(step + RS, st);
        if (++st == RS) { st = 0; par ^= 1u; }
      }
      if (*abort_flag) {                               // loads of a drained CTA may be in flight
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) {}
      }
    }
  } else {
    // ------------------------------------------------------------------ table loader
    if (elect_one()) {
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
  if (warp == 8 * GROUPS) {
    for (int i = 0; i < GROUPS; ++i) mbar_wait_drain(done + i, 0, P.wait_cycles);
    tc_fence_after();
    tmem_free(tmem_base, tmem_cols);
  }
}

struct DzPlan { int groups, lb, splits, chunks_per_split, tstages, rstages; size_t smem; };

// Columns whose weights are formed: the L - 1 useful ones, known at compile time, where that spares three to seven of
// 8 * LB and the spline is one that the package's defaults and sweeps use; all 8 * LB otherwise (the padding's weights are
// zero).  dz at 65536 x 5120, r = 32, exact against all: L = 22 0.973 / 1.043 ms, L = 42 1.70 / 1.83 ms, linear L = 21
// 1.10 / 1.17 ms.  One column spared (L = 16, 15 of 16) costs a pair its partner: 0.888 / 0.854 ms.
template <bool LIN, bool SPLIT>
cudaError_t dz_launch(const DzPlan& zp, int L, bool relu, const DzParams& P, dim3 grid, cudaStream_t stream) {
  CUtensorMap mz, mg, md;
  if (!make_box_map(&mz, P.z, P.N, P.h, P.zs) || (P.g_act && !make_box_map(&mg, P.g_act, P.N, P.h, P.gas)) ||
      (!P.dz_f32 && !make_box_map(&md, P.dz, P.N, P.h, P.dzs)))
    return cudaErrorInvalidValue;
  if (!P.g_act) mg = mz;
  if (P.dz_f32) md = mz;
  const unsigned threads = 320 * zp.groups + 32;
#define SKV_DZ_CASE(G_, LB_, NC_, COND_)                                                                           \
  if (zp.groups == G_ && zp.lb == LB_ && (COND_))                                                                  \
    return relu ? launch_chained<tc_dz_kernel<G_, LB_, NC_, true, LIN, SPLIT>>(grid, threads, zp.smem, stream, P, mz, mg, md)         \
                : launch_chained<tc_dz_kernel<G_, LB_, NC_, false, LIN, SPLIT>>(grid, threads, zp.smem, stream, P, mz, mg, md);
  if constexpr (LIN) {
    SKV_DZ_CASE(2, 3, 20, L == 21)
  } else {
    SKV_DZ_CASE(2, 3, 21, L == 22) SKV_DZ_CASE(2, 6, 41, L == 42)
  }
  SKV_DZ_CASE(2, 1, 8, true) SKV_DZ_CASE(2, 2, 16, true) SKV_DZ_CASE(2, 3, 24, true) SKV_DZ_CASE(2, 4, 32, true)
  SKV_DZ_CASE(2, 5, 40, true) SKV_DZ_CASE(2, 6, 48, true) SKV_DZ_CASE(2, 7, 56, true) SKV_DZ_CASE(2, 8, 64, true)
  SKV_DZ_CASE(1, 1, 8, true) SKV_DZ_CASE(1, 2, 16, true) SKV_DZ_CASE(1, 3, 24, true) SKV_DZ_CASE(1, 4, 32, true)
  SKV_DZ_CASE(1, 5, 40, true) SKV_DZ_CASE(1, 6, 48, true) SKV_DZ_CASE(1, 7, 56, true) SKV_DZ_CASE(1, 8, 64, true)
#undef SKV_DZ_CASE
  return cudaErrorInvalidValue;
}

}  // namespace tc
}  // namespace skv
