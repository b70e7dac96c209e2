// tcgen05 kernel for dC (key-major):
//   dC[(j,b), c] = sum_n Phi[n,(j,b)] * g[n,c]  (M = knot rows of a key chunk, N = r, K = tokens)
//   A CTA owns a slab of keys, keeps the slab's accumulators in tensor memory and streams
//   128-token tiles: two producer groups alternate, each building the f16 Phi tile of its token
//   tile for one key chunk in its own shared-memory stage while the MMAs of the other run.
//   The token range is split over CTAs; a reduce kernel sums the splits in a fixed order.
#pragma once

#include "skv_tc_prep.cuh"

namespace skv {
namespace tc {

struct DcParams {
  const __nv_bfloat16* z;
  int64_t zs;
  const __half* gimg;
  float* part;               // [splits][h*L][r]
  int64_t N;
  int h, L, r;
  GridParams g;
  int LR;                    // knot rows per key in the Phi^T tile: L rounded up to even (pad row zero)
  int kch;                   // keys per chunk (8 or 16)
  int mtiles;                // 128-row MMA tiles per chunk
  int slab_chunks;           // chunks per CTA slab
  int64_t tiles_per_split;   // 128-token tiles per token split
  int64_t tiles_total;
  int32_t* status;
  long long wait_cycles;     // limit of every bounded wait, in clock cycles
};

// KCH = keys per chunk.  Two producer groups of 128 threads (thread = token of the group's tile).
template <int KCH, int HLC, bool LIN>
__global__ void __launch_bounds__(256 + 64, 1) tc_dc_kernel(const DcParams P) {
  extern __shared__ __align__(128) uint8_t smem[];
  const int L = P.L, LR = HLC ? 2 * HLC : P.LR, r = P.r;
  const uint32_t phi_bytes = (uint32_t)P.mtiles * 16u * 2048u;     // [m groups][16 token groups][8 tok][8 m]
  const uint32_t g_bytes = (uint32_t)(128 * r * 2);
  uint8_t* phi_base = smem;                                         // [2][phi_bytes]
  uint8_t* g_base = smem + 2 * (size_t)phi_bytes;                   // [2][g_bytes]
  uint64_t* bars = reinterpret_cast<uint64_t*>(g_base + 2 * (size_t)g_bytes);
  uint64_t* pfull = bars;          // [2] producers -> MMA
  uint64_t* pempty = pfull + 2;    // [2][3] MMA -> producers, per 128-row tile
  uint64_t* gfull = pempty + 6;    // [2] TMA -> MMA
  uint64_t* gempty = gfull + 2;    // [2] MMA -> TMA
  uint64_t* done = gempty + 2;     // [1]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const WaitCtx wc{abort_flag, P.status, kStatusTimeoutDc, P.wait_cycles};

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rows = KCH * LR;                                         // (padded) knot rows per chunk
  const int key0 = blockIdx.x * P.slab_chunks * KCH;
  const int nchunks = min(P.slab_chunks, (P.h - key0 + KCH - 1) / KCH);
  const int64_t tile_begin = (int64_t)blockIdx.y * P.tiles_per_split;
  const int ntiles = (int)min(P.tiles_per_split, P.tiles_total - tile_begin);
  uint32_t tmem_cols = 32;
  while (tmem_cols < (uint32_t)(P.slab_chunks * P.mtiles * r)) tmem_cols <<= 1;

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(pfull + i, 4);
      mbar_init(gfull + i, 1);
      mbar_init(gempty + i, 1);
    }
    for (int i = 0; i < 6; ++i) mbar_init(pempty + i, 1);
    mbar_init(done, 1);
    *abort_flag = 0;
    mbar_init_fence();
  }
  {
    uint4* p = reinterpret_cast<uint4*>(phi_base);
    const uint32_t n16 = 2 * phi_bytes / 16;
    for (uint32_t i = tid; i < n16; i += blockDim.x) p[i] = make_uint4(0, 0, 0, 0);
  }
  if (warp == 8) tmem_alloc(tmem_slot, tmem_cols);
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch();
  pdl_wait();

  if (warp < 8) {
    // ------------------------------------------------------------------ producers
    const int pg = warp >> 2;
    const int t = tid & 127;
    const uint32_t t_off = (uint32_t)(t & 7) * 16u + (uint32_t)(t >> 3) * 128u;
    const uint32_t row = smem_u32(phi_base + (size_t)pg * phi_bytes) + t_off;
    const uint32_t halfL = (uint32_t)LR >> 1;
    uint32_t saved[KCH];
#pragma unroll
    for (int i = 0; i < KCH; ++i) saved[i] = 0;
    bool have_saved = false;
    int use = 0;                                     // how often this group's stage has been filled
    for (int ti = pg; ti < ntiles; ti += 2) {
      const int64_t n = (tile_begin + ti) * 128 + t;
      const bool valid = n < P.N;
      const __nv_bfloat16* zrow = P.z + (valid ? n : 0) * P.zs + key0;
      // pre-activations of the chunk after this one are requested before this one is processed
      uint4 znext[KCH / 8];
#pragma unroll
      for (int i = 0; i < KCH / 8; ++i)
        znext[i] = valid && key0 + i * 8 < P.h ? ld16(zrow + i * 8) : make_uint4(0, 0, 0, 0);
      for (int ch = 0; ch < nchunks; ++ch, ++use) {
        uint4 zq[KCH / 8];
#pragma unroll
        for (int i = 0; i < KCH / 8; ++i) {
          zq[i] = znext[i];
          const bool in_h = ch + 1 < nchunks && key0 + (ch + 1) * KCH + i * 8 < P.h;
          znext[i] = valid && in_h ? ld16(zrow + (ch + 1) * KCH + i * 8)
                                   : make_uint4(0, 0, 0, 0);
        }
        // The MMA thread releases a stage tile by tile (128 knot rows each); with the words per key
        // known at compile time (HLC) a tile is waited for just before the first key that touches it,
        // so this stage's first keys are written while the MMAs still read the later tiles of the
        // previous use.  Otherwise all tiles are waited for first.
        if (!HLC && use > 0)
          for (int m = 0; m < P.mtiles; ++m) mbar_wait(pempty + pg * 3 + m, (uint32_t)(use - 1) & 1u, wc);
        const int keys_left = P.h - (key0 + ch * KCH);         // keys of this chunk that exist
#pragma unroll
        for (int q = 0; q < KCH; ++q) {
          if (HLC && use > 0) {
            // tiles touched by words q * HLC .. (q + 1) * HLC - 1 (word w lies in tile w >> 6) that no
            // earlier key touched
            const int t_lo = q == 0 ? 0 : (((q * HLC - 1) >> 6) + 1), t_hi = ((q + 1) * HLC - 1) >> 6;
#pragma unroll
            for (int m = 0; m < 3; ++m)
              if (m >= t_lo && m <= t_hi) mbar_wait(pempty + pg * 3 + m, (uint32_t)(use - 1) & 1u, wc);
          }
          if (have_saved) {
            sts32(row + (saved[q] & 0xffffu) * 4u, 0u);
            sts32(row + (saved[q] >> 16) * 4u, 0u);
          }
          if (valid) {
            const uint4& zc = zq[q >> 3];
            const uint32_t zw[4] = {zc.x, zc.y, zc.z, zc.w};
            const int qq = q & 7;
            const float zz = (qq & 1) ? bf_hi(zw[qq >> 1]) : bf_lo(zw[qq >> 1]);
            uint32_t x0, x1, wo0, wo1;
            phi_pair<LIN>(zz, P.g, (uint32_t)q * halfL, x0, x1, wo0, wo1);
            if (q >= keys_left) { x0 = 0u; x1 = 0u; }
            sts32(row + wo1 * 4u, x1);
            sts32(row + wo0 * 4u, x0);
            saved[q] = wo0 | (wo1 << 16);
          }
        }
        have_saved = valid;
        fence_async_smem();
        mbar_arrive_warp(pfull + pg);
      }
    }
    // ---- epilogue: accumulators -> float32 partial of this token split
    mbar_wait(done, 0, wc);
    tc_fence_after();
    const int lane_row = (warp & 3) * 32 + lane;
    float* part = P.part + (size_t)blockIdx.y * P.h * L * r;
    for (int ch = pg; ch < nchunks; ch += 2) {
      for (int mt = 0; mt < P.mtiles; ++mt) {
        const int rr = mt * 128 + lane_row;                        // padded knot row within the chunk
        const int kl = rr / LR, bb = rr - kl * LR;
        const int key = key0 + ch * KCH + kl;
        const bool ok = rr < rows && key < P.h && bb < L;           // the pad row of an odd L is dropped
        float* dst = part + ((size_t)key * L + bb) * r;
        const uint32_t taddr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)((ch * P.mtiles + mt) * r);
        for (int c0 = 0; c0 < r; c0 += 16) {
          float v[16];
          tmem_ld16(taddr + c0, v);
          if (ok) {
#pragma unroll
            for (int i = 0; i < 16; i += 4)
              *reinterpret_cast<float4*>(dst + c0 + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
          }
        }
      }
    }
    tc_fence_before();
  } else if (warp == 8) {
    // ------------------------------------------------------------------ MMA issue
    if (elect_one()) {
      const uint32_t idesc = instr_desc(0, 0, 1, 1, 128, r);
      const uint32_t ab_hi = desc_hi(2048u);
      int guse[2] = {0, 0}, puse[2] = {0, 0};
      bool drain = false;
      for (int tp = 0; tp < ntiles; tp += 2) {
        const int npg = min(2, ntiles - tp);
        for (int pg = 0; pg < npg; ++pg)
          drain = mbar_wait(gfull + pg, (uint32_t)guse[pg] & 1u, wc) || drain;
        if (drain) break;
        for (int ch = 0; ch < nchunks; ++ch) {
          for (int pg = 0; pg < npg; ++pg) {
            drain = mbar_wait(pfull + pg, (uint32_t)puse[pg] & 1u, wc);
            ++puse[pg];
            if (drain) break;                        // draining: issue nothing more
            tc_fence_after();
            const uint32_t a_addr = smem_u32(phi_base + (size_t)pg * phi_bytes);
            const uint32_t b_addr = smem_u32(g_base + (size_t)pg * g_bytes);
            const uint32_t first = (tp == 0 && pg == 0) ? 0u : 1u;
            const uint32_t b_lo0 = desc_lo(b_addr, 128u);
            for (int mt = 0; mt < P.mtiles; ++mt) {
              uint32_t a_lo = desc_lo(a_addr + (uint32_t)mt * 16u * 2048u, 128u);
              uint32_t b_lo = b_lo0;
              const uint32_t d_addr = tmem_base + (uint32_t)((ch * P.mtiles + mt) * r);
              umma_f16_split(d_addr, a_lo, ab_hi, b_lo, ab_hi, idesc, first);
#pragma unroll
              for (int ks = 1; ks < 8; ++ks) {
                a_lo += 256u >> 4;
                b_lo += 256u >> 4;
                umma_f16_split(d_addr, a_lo, ab_hi, b_lo, ab_hi, idesc, 1u);
              }
              umma_commit(pempty + pg * 3 + mt);
            }
          }
          if (drain) break;
        }
        if (drain) break;
        for (int pg = 0; pg < npg; ++pg) { umma_commit(gempty + pg); ++guse[pg]; }
      }
      umma_commit(done);
    }
  } else {
    // ------------------------------------------------------------------ gradient-tile loader
    if (elect_one()) {
      int guse[2] = {0, 0};
      for (int ti = 0; ti < ntiles; ++ti) {
        const int pg = ti & 1;
        if (guse[pg] > 0)
          mbar_wait(gempty + pg, (uint32_t)(guse[pg] - 1) & 1u, wc);
        if (*abort_flag) break;
        mbar_arrive_expect_tx(gfull + pg, g_bytes);
        bulk_g2s(g_base + (size_t)pg * g_bytes,
                 reinterpret_cast<const uint8_t*>(P.gimg) + (size_t)(tile_begin + ti) * g_bytes, g_bytes, gfull + pg);
        ++guse[pg];
      }
      if (*abort_flag) {
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) {}
      }
    }
  }
  __syncthreads();
  if (warp == 8) {
    mbar_wait_drain(done, 0, P.wait_cycles);
    tc_fence_after();
    tmem_free(tmem_base, tmem_cols);
  }
}

struct DcPlan { int kch, mtiles, slab_chunks, slabs, splits; int64_t tiles_total, tiles_per_split; size_t smem; };

}  // namespace tc
}  // namespace skv
