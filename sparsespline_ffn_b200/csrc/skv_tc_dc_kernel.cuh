// tcgen05 kernel for dC (key-major):
//   dC[(j,b), c] = sum_n Phi[n,(j,b)] * g[n,c]  (M = knot rows of a key chunk, N = r, K = tokens)
//   A CTA owns a slab of keys, keeps the slab's accumulators in tensor memory and streams
//   64-token tiles: producer groups take turns, each building the f16 Phi tile of its token
//   tile for one key chunk in its own shared-memory stage while the MMAs of the others run.
//   The work, slab after slab and tile after tile within a slab, is cut into equal runs, one per CTA: a run may end one
//   slab and begin the next, which fills the chip evenly, or stay within a slab, which saves an epilogue and a refill where
//   there is little to do (make_dc_plan weighs the two).  A run is worked off in segments that end with the slab or after a chain
//   of tiles (kDcChain); a CTA's segments of one slab go to one partial, and a reduce kernel sums a slab's
//   partials in a fixed order.
//
// Where a weight goes.  A pair's three weights are two neighbouring f16x2 words (knot rows 2w, 2w+1 and the next
// two).  The operand layout (MN-major, un-swizzled) wants 16-byte pieces of eight M rows of one token, four banks
// wide, at a bank that depends on the token modulo 8.  M rows may be in any order, so a piece holds the same
// word w of FOUR keys: row ((j * HL + w) * 8 + 2 * kq + (b & 1)) for the chunk's key KJ * kq + j, knot row b and HL
// words per key.  A warp works on 8 tokens x 4 values of kq at a time, hence bank = 4 * (token & 7) + kq = lane: the
// scattered stores never conflict, whatever the knot intervals are.  (With the rows in knot order the four tokens
// that share a piece's banks picked one of them by their interval and a store took three wavefronts; that
// and clearing behind it was half of the shared-memory time of a kernel bound by it: 1.35 ms at the d20 shape.)
#pragma once

#include "skv_tc_prep.cuh"

namespace skv {
namespace tc {

struct DcParams {
  const __nv_bfloat16* z;
  int64_t zs;
  const __half* gimg;
  float* part;               // [runs that touch a slab][h*L][r]
  int64_t N;
  int h, L, r;
  GridParams g;
  int words;                 // f16x2 words per key in the Phi^T tile: L / 2 rounded up (an odd L's last row is zero)
  int ngroups;               // producer groups, one stage each
  int gring;                 // slots of the ring of g tiles, more than groups
  int mtiles;                // 128-row MMA tiles per chunk
  int slab_chunks;           // chunks per CTA slab
  uint32_t tiles;            // 64-token tiles
  uint32_t pitch;            // places per slab in the runs' count: the tiles, or whole runs (then no run crosses slabs)
  uint32_t run, total;       // places of a CTA's run, and of all slabs together
  uint32_t chain;            // tiles of a segment at most
  int32_t* status;
  long long wait_cycles;     // limit of every bounded wait, in clock cycles
};

constexpr int kDcTokens = 64;                        // tokens per tile
constexpr uint32_t kDcUnit = kDcTokens * 16;         // bytes of one 8-row group of a tile
constexpr int kDcMaxGroups = 4;
constexpr int kDcMaxRing = 8;                        // slots of the ring of g tiles
// Tiles whose MMAs follow one another in an accumulator; what they gave is then added to the partial in float32.  The tensor
// core cuts a sum off at the accumulator's last bit, always towards zero: the error grows with the number of MMAs
// and does not average out.  Error of dC against 64 bits at 65536 x 5120, r = 32 / r = 128, all gradients positive (so that
// every bit lost counts): one accumulator for 443 / 1024 tiles 6.8e-5 / 1.9e-4, 256 tiles 5.0e-5 / 5.4e-5, 192 tiles
// 4.7e-5 / 4.7e-5 (what rounding the operands to f16 gives), dC alone 0.81 / 1.53, 0.82 / 1.57, 0.83 / 1.60 ms.
// With pairs of f16 there is no such floor: 65536 x 5113, r = 32: 443 tiles 9.9e-5, 32 tiles 7.0e-6, 16 tiles 3.4e-6,
// 8 tiles 1.8e-6; 1.94, 2.03, 2.14, 2.36 ms; 4096 x 1024, linear: 37, 37, 38, 45 us.  (float32 arithmetic on the CUDA
// cores: 3.2e-6 at the former size, 13.7 ms.)
constexpr uint32_t kDcChain = 192, kDcSplitChain = 16;
constexpr int kDcIssuers = 3;                        // warps that issue MMAs, each for every third M tile
// One unit behind a stage: the linear spline's last interval stores a zero word there.
__host__ __device__ constexpr uint32_t dc_stage_bytes(int mtiles) { return (uint32_t)mtiles * 16u * kDcUnit + kDcUnit; }

// KJ = keys per lane and token (a chunk is 4 * KJ keys), GW = warps per producer group.  SPLIT: a stage is filled twice, with
// the weights and with their remainders at the same places.  RUNS: a run may have several segments; without it their loop is
// gone at compile time (5 % on the cases of one segment).
template <int KJ, int GW, bool LIN, bool SPLIT, bool RUNS>
__global__ void __launch_bounds__(640, 1) tc_dc_kernel(const DcParams P) {
  extern __shared__ __align__(128) uint8_t smem[];
  constexpr int KCH = 4 * KJ;
  constexpr int TI = kDcTokens / GW / 8;                            // tokens per lane
  const int L = P.L, r = P.r, NG = P.ngroups;
  const uint32_t phi_bytes = dc_stage_bytes(P.mtiles);             // [m groups][8 token groups][8 tok][8 m]
  const uint32_t g_bytes = (uint32_t)(kDcTokens * r * 2);
  uint8_t* phi_base = smem;                                         // [NG][phi_bytes]
  const int GR = P.gring;
  uint8_t* g_base = smem + NG * (size_t)phi_bytes;                  // [GR][g_bytes]
  uint64_t* bars = reinterpret_cast<uint64_t*>(g_base + GR * (size_t)g_bytes);
  uint64_t* pfull = bars;                       // [NG] producers -> MMA
  uint64_t* pempty = pfull + kDcMaxGroups;      // [NG] MMA -> producers
  uint64_t* gfull = pempty + kDcMaxGroups;      // [GR] TMA -> MMA
  uint64_t* gempty = gfull + kDcMaxRing;        // [GR] MMA -> TMA
  uint64_t* done = gempty + kDcMaxRing;         // [1]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const WaitCtx wc{abort_flag, P.status, kStatusTimeoutDc, P.wait_cycles};

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int mma_warp = NG * GW;
  uint32_t tmem_cols = 32;
  while (tmem_cols < (uint32_t)(P.slab_chunks * P.mtiles * r)) tmem_cols <<= 1;

  if (tid == 0) {
    for (int i = 0; i < kDcMaxGroups; ++i) {
      mbar_init(pfull + i, GW);
      mbar_init(pempty + i, kDcIssuers);
    }
    for (int i = 0; i < kDcMaxRing; ++i) {
      mbar_init(gfull + i, 1);
      mbar_init(gempty + i, kDcIssuers);
    }
    mbar_init(done, kDcIssuers);
    *abort_flag = 0;
    mbar_init_fence();
  }
  {
    uint4* p = reinterpret_cast<uint4*>(phi_base);
    const uint32_t n16 = (uint32_t)NG * phi_bytes / 16;
    for (uint32_t i = tid; i < n16; i += blockDim.x) p[i] = make_uint4(0, 0, 0, 0);
  }
  if (warp == mma_warp) tmem_alloc(tmem_slot, tmem_cols);
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch();
  pdl_wait();

  const uint32_t lin_end = min(P.total, (blockIdx.x + 1) * P.run);
  int seg = 0;
  // what each role carries from segment to segment
  int use = 0;                                         // producers: fills of the group's stage
  uint32_t old[TI][KJ];
  uint32_t ppar = 0u, gpar0 = 0u, lpar = 1u;           // MMA issuers: phase per group, ring phase; loader: ring phase
  int slot0 = 0, lslot = 0;
#pragma unroll
  for (int i = 0; i < TI; ++i)
#pragma unroll
    for (int j = 0; j < KJ; ++j) old[i][j] = 0u;
  for (uint32_t lin = blockIdx.x * P.run; RUNS ? lin < lin_end : seg == 0; ++seg) {
    const uint32_t slab = lin / P.pitch, tile_begin = lin - slab * P.pitch;
    if (RUNS && tile_begin >= P.tiles) break;            // places past the tiles end the last run of a slab
    const uint32_t places = min(min(P.pitch - tile_begin, lin_end - lin), RUNS ? P.chain : ~0u);
    const bool more = RUNS && seg > 0 && tile_begin > 0; // this CTA's partial of the slab has been begun
    const int ntiles = (int)min(P.tiles - tile_begin, places);
    const int key0 = (int)slab * P.slab_chunks * KCH;
    const int nchunks = min(P.slab_chunks, (P.h - key0 + KCH - 1) / KCH);
    lin += places;
    if (warp < mma_warp) {
      // ------------------------------------------------------------------ producers
      const int pg = warp / GW, wi = warp % GW;
      const int tq = lane >> 2, kq = lane & 3;
      // address of this lane's word 0 of key j and token i, less the bias that the word index carries
      const uint32_t row = smem_u32(phi_base + (size_t)pg * phi_bytes) + (uint32_t)(wi * TI * 128 + tq * 16 + kq * 4) -
                           kWordBias * kDcUnit;
      const uint32_t jstep = (uint32_t)P.words * kDcUnit;
      const int tk0 = wi * TI * 8 + tq;                                // the lane's first token of the tile
      auto load_z = [&](int ti, int ch, uint32_t (&zv)[TI][KJ / 2]) {
        const int key = key0 + ch * KCH + KJ * kq;
#pragma unroll
        for (int i = 0; i < TI; ++i) {
          const int64_t n = (int64_t)(tile_begin + (uint32_t)ti) * kDcTokens + tk0 + 8 * i;
          const bool ok = ti < ntiles && n < P.N && key < P.h;         // g is zero past N; keys past h are never stored
          const __nv_bfloat16* src = P.z + n * P.zs + key;
          if constexpr (KJ == 4) {
            const uint2 v = ok ? ld8(src) : make_uint2(0, 0);
            zv[i][0] = v.x;
            zv[i][1] = v.y;
          } else {
            zv[i][0] = ok ? ld4(src) : 0u;
          }
        }
      };
      uint32_t znext[TI][KJ / 2];
      load_z(pg, 0, znext);
      int ti = pg, ch = 0;
      for (; ti < ntiles; ++use) {
        uint32_t x0[TI][KJ], x1[TI][KJ], ad[TI][KJ], r0[SPLIT ? TI : 1][KJ], r1[SPLIT ? TI : 1][KJ];
#pragma unroll
        for (int i = 0; i < TI; ++i)
#pragma unroll
          for (int q = 0; q < KJ / 2; ++q) {
            uint32_t a0[2], a1[2], wp[2];
            phi_pair_words2<LIN, SPLIT>(znext[i][q], P.g, a0, a1, wp, &r0[SPLIT ? i : 0][2 * q], &r1[SPLIT ? i : 0][2 * q]);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              x0[i][2 * q + e] = a0[e];
              x1[i][2 * q + e] = a1[e];
              ad[i][2 * q + e] = row + (uint32_t)(i * 128) + (uint32_t)(2 * q + e) * jstep + wp[e] * kDcUnit;
            }
          }
        if (++ch == nchunks) { ch = 0; ti += NG; }
        load_z(ti, ch, znext);                          // the next fill's rows are requested now
        if (use > 0) {
          mbar_wait(pempty + pg, (uint32_t)(use - 1) & 1u, wc);
#pragma unroll
          for (int i = 0; i < TI; ++i)
#pragma unroll
            for (int j = 0; j < KJ; ++j) {
              sts32(old[i][j], 0u);
              sts32(old[i][j] + kDcUnit, 0u);
            }
        }
        // keys in ascending order: the linear spline's zero word of a last interval falls on the next key's first
#pragma unroll
        for (int i = 0; i < TI; ++i)
#pragma unroll
          for (int j = 0; j < KJ; ++j) {
            sts32(ad[i][j], x0[i][j]);
            sts32(ad[i][j] + kDcUnit, x1[i][j]);
            old[i][j] = ad[i][j];
          }
        fence_async_smem();
        mbar_arrive_warp(pfull + pg);
        if constexpr (SPLIT) {
          ++use;
          mbar_wait(pempty + pg, (uint32_t)(use - 1) & 1u, wc);
#pragma unroll
          for (int i = 0; i < TI; ++i)
#pragma unroll
            for (int j = 0; j < KJ; ++j) {
              sts32(ad[i][j], r0[i][j]);
              sts32(ad[i][j] + kDcUnit, r1[i][j]);
            }
          fence_async_smem();
          mbar_arrive_warp(pfull + pg);
        }
      }
      // ---- epilogue: accumulators -> float32 partial of this token split
      mbar_wait(done, (uint32_t)seg & 1u, wc);
      tc_fence_after();
      const int lane_row = (warp & 3) * 32 + lane;
      float* part = P.part + (size_t)(blockIdx.x - slab * P.pitch / P.run) * P.h * L * r;
      for (int e = warp >> 2; e < nchunks * P.mtiles; e += mma_warp >> 2) {
        const int c = e / P.mtiles, mt = e - c * P.mtiles;
        const int unit = mt * 16 + (lane_row >> 3), j = unit / P.words;
        const int bb = 2 * (unit - j * P.words) + (lane_row & 1);
        const int key = key0 + c * KCH + KJ * ((lane_row & 7) >> 1) + j;
        const bool ok = j < KJ && key < P.h && bb < L;                   // the pad row of an odd L is dropped
        const uint32_t at = ok ? (uint32_t)(key * L + bb) : ~0u;         // row of the partial
        const uint32_t taddr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(e * r);
        for (int c0 = 0; c0 < r; c0 += 16) {
          float v[16];
          tmem_ld16(taddr + c0, v);
          quad_transpose(v);
#pragma unroll
          for (int j4 = 0; j4 < 4; ++j4) {
            const uint32_t row4 = __shfl_sync(0xffffffffu, at, (lane & ~3) + j4);
            if (row4 != ~0u) {
              float* dst = part + (size_t)row4 * r + c0 + 4 * (lane & 3);
              const float* q = v + 4 * j4;
              if (more) red_add4(dst, q[0], q[1], q[2], q[3]);             // to what this thread has put there
              else *reinterpret_cast<float4*>(dst) = make_float4(q[0], q[1], q[2], q[3]);
            }
          }
        }
      }
      tc_fence_before();
    } else if (warp < mma_warp + kDcIssuers) {
      // ------------------------------------------------------------------ MMA issue
      if (elect_one()) {
        const int m0 = warp - mma_warp;
        const uint32_t idesc = instr_desc(0, 0, 1, 1, 128, r);
        const uint32_t ab_hi = desc_hi(kDcUnit);
        const uint32_t a_tile0 = desc_lo(smem_u32(phi_base) + (uint32_t)m0 * 16u * kDcUnit, 128u);
        const uint32_t b_ring = desc_lo(smem_u32(g_base), 128u);
        bool drain = false;
        for (int tp = 0; tp < ntiles && !drain; tp += NG) {
          const int npg = min(NG, ntiles - tp);
          constexpr int kParts = SPLIT ? 2 : 1;
          for (int cp = 0; cp < nchunks * kParts && !drain; ++cp) {
            const int ch = cp / kParts, part = cp % kParts;
            const bool last = cp + 1 == nchunks * kParts;
            int slot = slot0;
            uint32_t gpar = gpar0;
            for (int pg = 0; pg < npg; ++pg) {
              if (cp == 0) drain = drain || mbar_wait(gfull + slot, gpar, wc);
              drain = drain || mbar_wait(pfull + pg, (ppar >> pg) & 1u, wc);
              ppar ^= 1u << pg;
              if (drain) break;                          // draining: issue nothing more
              tc_fence_after();
              uint32_t a_lo0 = a_tile0 + (uint32_t)pg * (phi_bytes >> 4);
              const uint32_t b_lo0 = b_ring + (uint32_t)slot * (g_bytes >> 4);
              uint32_t d_addr = tmem_base + (uint32_t)((ch * P.mtiles + m0) * r);
              const uint32_t first = tp + pg + part == 0 ? 0u : 1u;
              for (int mt = m0; mt < P.mtiles; mt += kDcIssuers) {
#pragma unroll
                for (int ks = 0; ks < kDcTokens / 16; ++ks)
                  umma_f16_split(d_addr, a_lo0 + (uint32_t)ks * 16u, ab_hi, b_lo0 + (uint32_t)ks * 16u, ab_hi, idesc,
                                 ks > 0 ? 1u : first);
                a_lo0 += (kDcIssuers * 16u * kDcUnit) >> 4;
                d_addr += (uint32_t)(kDcIssuers * r);
              }
              umma_commit(pempty + pg);
              if (last) umma_commit(gempty + slot);
              if (++slot == GR) { slot = 0; gpar ^= 1u; }
            }
            if (last) { slot0 = slot; gpar0 = gpar; }
          }
        }
        umma_commit(done);
      }
    } else {
      // ------------------------------------------------------------------ gradient-tile loader
      if (elect_one()) {
        const uint8_t* img = reinterpret_cast<const uint8_t*>(P.gimg);
        int slot = lslot;
        uint32_t par = lpar;                             // a fresh barrier passes a wait for the phase before its first
        for (int ti = 0; ti < ntiles; ++ti) {
          mbar_wait(gempty + slot, par, wc);
          if (*abort_flag) break;
          mbar_arrive_expect_tx(gfull + slot, g_bytes);
          // the image has 128-token tiles [r/8][16 token groups][128 B]; this tile is one half of each channel group
          const int64_t t64 = (int64_t)tile_begin + ti;
          const uint8_t* src = img + (size_t)(t64 >> 1) * 128 * r * 2 + (size_t)(t64 & 1) * kDcUnit;
          for (int cg = 0; cg < r / 8; ++cg)
            bulk_g2s(g_base + (size_t)slot * g_bytes + (size_t)cg * kDcUnit, src + (size_t)cg * 2 * kDcUnit, kDcUnit,
                     gfull + slot);
          if (++slot == GR) { slot = 0; par ^= 1u; }
        }
        lslot = slot;
        lpar = par;
        if (*abort_flag) {
          const long long t0 = clock64();
          while (clock64() - t0 < 2000000) {}
        }
      }
    }
    tc_fence_before();
    __syncthreads();                                     // the accumulators have been read
    tc_fence_after();
  }
  if (warp == mma_warp) {
    mbar_wait_drain(done, (uint32_t)(seg - 1) & 1u, P.wait_cycles);
    tc_fence_after();
    tmem_free(tmem_base, tmem_cols);
  }
}

// `runs`: a run may cross slabs; the number of partials of a slab and the room for them follow it.
struct DcPlan {
  int kj, gw, ngroups, gring, mtiles, slab_chunks, parts;
  bool runs;
  uint32_t tiles, pitch, run, total, chain;
  size_t smem;
};

}  // namespace tc
}  // namespace skv
