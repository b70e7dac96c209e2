// Backward as one kernel (opt-in): dz and dC in one CTA.
//
// A CTA owns a slab of 16 keys and a range of 128-token tiles; tile i belongs to token group i % 2.
// The dz kernel is bound by instruction issue and the dC kernel by shared-memory bandwidth (its
// producers wait half the time for the MMAs that read their stage); run as separate warps of one
// CTA the two fill each other's gaps, and the g tile in shared memory serves both.
//
//   warps 0..7    dz role, groups 0 and 1 (thread = token): the S columns of 4 keys at a time
//                 (S = g T^T, in one of the group's two tensor-memory blocks, so that the next
//                 block is computed while this one is read) -> dz, as tc_dz_kernel does
//   warps 8..15   Phi role, groups 0 and 1: a group fills stages of 64 tokens x 16 keys (two
//                 threads per token, 8 keys each): knot interval and weights -> the two non-zero
//                 words of each key's Phi^T segment, scattered into the stage (A operand of the dC
//                 MMAs); two stages per group, so that one is filled while the other is read
//   warp 16       lane 0 issues the S MMAs of both groups (whichever is ready first)
//   warp 17       lane 0 issues the dC MMAs of both groups (3 M-tiles x 4 K-steps per stage)
//   warp 18       lane 0 loads the slab's transformed table once and streams the g tiles (3-deep ring)
//
// Registers are re-balanced between the roles with setmaxnreg (the kernel starts every warp with
// the same count): the helper warps give registers up, the dz warps take them.
//
// Tensor memory: [group 0: S block 0, S block 1 | group 1: ... | dC accumulators of the slab]
// = 4 * 4*LP + mtiles*r columns.
// Shared memory: four Phi^T stages of 16*L knot rows x 64 tokens, the g ring, the table slab.  A
// stage holds exactly 16*L rows; the MMAs of its last M-tile read up to the next multiple of 128
// rows, i.e. into whatever follows the stage.  Each accumulator row depends on its own A row only
// and the rows past 16*L are never stored, so those reads are harmless.
#include "skv_tc_bwd_fused.cuh"

namespace skv {
namespace tc {
namespace {

struct BfParams {
  const __nv_bfloat16* z;
  int64_t zs;
  const __nv_bfloat16* g_act;
  int64_t gas;
  __nv_bfloat16* dz;
  int64_t dzs;
  const __half* gimg;
  const __half* timg;
  const uint32_t* amax_bits;
  float* part;               // [splits][h*L][r]
  int64_t N;
  int h, L, r;
  GridParams g;
  int act;
  float coef;                // lambda * scale
  int mtiles;                // 128-row MMA tiles over the slab's 16*L knot rows
  int dz_f32;                // dz is float32 [N][dzs] instead of bf16
  int roles;                 // bit 0: the dz role runs, bit 1: the Phi role and the dC MMAs run
  int64_t tiles_per_split, tiles_total;
  int32_t* status;
  long long wait_cycles;
};

constexpr int kSlabKeys = 16;
constexpr int kGRing = 3;
constexpr int kBfThreads = 640;
constexpr int kAux0 = 16;                      // first helper warp
// register counts per role (multiples of 8); 256 * kRegsDz + 256 * kRegsPhi + 128 * kRegsAux must
// not exceed kBfThreads * the count the kernel is compiled for (96)
constexpr int kRegsDz = 128, kRegsPhi = 88, kRegsAux = 40;
#ifndef SKV_POLL_NS
#define SKV_POLL_NS 20
#endif
constexpr unsigned kPollNs = SKV_POLL_NS;               // pause of an MMA issuer that found nothing ready

template <int R> __device__ __forceinline__ void reg_inc() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R));
}
template <int R> __device__ __forceinline__ void reg_dec() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R));
}

template <int LB, int NC, bool RELU>
__global__ void __launch_bounds__(kBfThreads, 1) tc_bwd_fused_kernel(const BfParams P) {
  extern __shared__ __align__(128) uint8_t smem[];
  const int L = P.L, r = P.r;
  constexpr int LP = 8 * LB;
  constexpr uint32_t bcols = (uint32_t)(4 * LP);                    // columns of one S block (4 keys)
  const uint32_t phi_bytes = (uint32_t)((kSlabKeys * L + 7) / 8) * 1024u;   // one 64-token stage
  const uint32_t g_bytes = (uint32_t)(128 * r * 2);
  const uint32_t t_bytes = (uint32_t)(kChunkKeys * LP * r * 2);     // table image of 8 keys
  uint8_t* phi_base = smem;                                          // [2 groups][2][phi_bytes]
  uint8_t* g_base = phi_base + 4 * (size_t)phi_bytes;                // [kGRing][g_bytes]
  uint8_t* t_base = g_base + (size_t)kGRing * g_bytes;               // [2][t_bytes]
  uint64_t* bars = reinterpret_cast<uint64_t*>(t_base + 2 * (size_t)t_bytes);
  uint64_t* gfull = bars;                  // [kGRing] loader -> MMA issuers
  uint64_t* gempty = gfull + kGRing;       // [kGRing] both MMA issuers -> loader (2 arrivals)
  uint64_t* tfull = gempty + kGRing;       // [1]
  uint64_t* sfull = tfull + 1;             // [2 groups][2] S issuer -> dz group
  uint64_t* sempty = sfull + 4;            // [2 groups][2] dz group -> S issuer
  uint64_t* pfull = sempty + 4;            // [2 groups][2] Phi group -> dC issuer
  uint64_t* pempty = pfull + 4;            // [2 groups][2] dC issuer -> Phi group
  uint64_t* done = pempty + 4;             // [2] all MMAs of the S issuer / the dC issuer complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const WaitCtx wc{abort_flag, P.status, kStatusTimeoutBwd, P.wait_cycles};

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int key0 = blockIdx.x * kSlabKeys;
  const int64_t tile_begin = (int64_t)blockIdx.y * P.tiles_per_split;
  const int ntiles = (int)min(P.tiles_per_split, P.tiles_total - tile_begin);
  const uint32_t dcol0 = 4u * bcols;
  uint32_t tmem_cols = 32;
  while (tmem_cols < dcol0 + (uint32_t)(P.mtiles * r)) tmem_cols <<= 1;

  if (tid == 0) {
    const uint32_t issuers = (uint32_t)((P.roles & 1) + ((P.roles >> 1) & 1));
    for (int i = 0; i < kGRing; ++i) { mbar_init(gfull + i, 1); mbar_init(gempty + i, issuers); }
    mbar_init(tfull, 1);
    for (int i = 0; i < 4; ++i) {
      mbar_init(sfull + i, 1);
      mbar_init(sempty + i, 4);
      mbar_init(pfull + i, 4);
      mbar_init(pempty + i, 1);
    }
    mbar_init(done + 0, 1);
    mbar_init(done + 1, 1);
    *abort_flag = 0;
    mbar_init_fence();
  }
  {
    uint4* p = reinterpret_cast<uint4*>(phi_base);
    const uint32_t n16 = 4 * phi_bytes / 16;
    for (uint32_t i = tid; i < n16; i += blockDim.x) p[i] = make_uint4(0, 0, 0, 0);
  }
  if (warp == kAux0) tmem_alloc(tmem_slot, tmem_cols);
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch();
  pdl_wait();

  if (warp < 8) {
    // ------------------------------------------------------------------ dz role
    reg_inc<kRegsDz>();
    const int pg = warp >> 2;
    const int t = tid & 127;
    const uint32_t trow = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)pg * 2u * bcols;
    float gscale, ginv;
    pow2_scales(*P.amax_bits, gscale, ginv);
    float cscale, cinv;
    pow2_scales(P.amax_bits[kAmaxC], cscale, cinv);
    const float coef = P.coef * ginv * cinv;
    const int act = P.act;
    const bool has_ga = P.g_act != nullptr;
    auto load_rows = [&](int ti, uint4 (&zv)[2], uint4 (&gv)[2], bool& valid, __nv_bfloat16*& dzrow) {
      const int64_t n = (tile_begin + ti) * 128 + t;
      valid = ti < ntiles && n < P.N;
      const int64_t nn = valid ? n : 0;
      const __nv_bfloat16* zrow = P.z + nn * P.zs + key0;
      const __nv_bfloat16* garow = has_ga ? P.g_act + nn * P.gas + key0 : nullptr;
      dzrow = P.dz + nn * P.dzs + key0;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        zv[i] = valid ? ld16(zrow + i * 8) : make_uint4(0, 0, 0, 0);
        gv[i] = valid && has_ga ? ld16(garow + i * 8) : make_uint4(0, 0, 0, 0);
      }
    };
    uint4 znext[2], ganext[2];
    bool vnext;
    __nv_bfloat16* dznext;
    load_rows(pg, znext, ganext, vnext, dznext);
    int use = 0;                                     // S blocks this group has consumed
    for (int ti = pg; ti < ntiles && (P.roles & 1); ti += 2) {
      const uint4 zq[2] = {znext[0], znext[1]}, gaq[2] = {ganext[0], ganext[1]};
      const bool valid = vnext;
      __nv_bfloat16* dzrow = dznext;
      load_rows(ti + 2, znext, ganext, vnext, dznext);   // the group's next tile: request its rows now
#pragma unroll 1
      for (int hf = 0; hf < 2; ++hf) {               // 8 keys per pass: two S blocks of 4 keys, unrolled
        const uint4 zc = hf ? zq[1] : zq[0], gc = hf ? gaq[1] : gaq[0];
        const uint32_t zw[4] = {zc.x, zc.y, zc.z, zc.w};
        const uint32_t gw[4] = {gc.x, gc.y, gc.z, gc.w};
        float outv[kChunkKeys];
#pragma unroll
        for (int qt = 0; qt < 2; ++qt, ++use) {
          const uint32_t blk = trow + (uint32_t)(use & 1) * bcols;
          uint32_t bufa[LB][8], bufb[LB][8];
          mbar_wait(sfull + pg * 2 + (use & 1), (uint32_t)(use >> 1) & 1u, wc);
          tc_fence_after();
          tmem_ld_key<LB, NC>(blk, bufa);
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4) {
            const int q = qt * 4 + q4;
            if (q4 & 1) tmem_wait_key<LB, NC>(bufb); else tmem_wait_key<LB, NC>(bufa);
            if (q4 + 1 < 4) {
              if (q4 & 1) tmem_ld_key<LB, NC>(blk + (uint32_t)((q4 + 1) * LP), bufa);
              else tmem_ld_key<LB, NC>(blk + (uint32_t)((q4 + 1) * LP), bufb);
            }
            const float zz = (q & 1) ? bf_hi(zw[q >> 1]) : bf_lo(zw[q >> 1]);
            const float u = __fmaf_rn(__fsub_rn(zz, P.g.lo), P.g.scale, 0.0f);
            const bool active = __float_as_uint(u) <= __float_as_uint(P.g.Gm1f);
            const float uc = fminf(fmaxf(u, 0.0f), P.g.Gm1f);
            const float acc = (q4 & 1) ? dz_key_sum<LB, NC>(bufb, uc) : dz_key_sum<LB, NC>(bufa, uc);
            float o = active ? coef * acc : 0.0f;
            if (has_ga) {
              const float ga = (q & 1) ? bf_hi(gw[q >> 1]) : bf_lo(gw[q >> 1]);
              const float dphi = RELU ? 2.0f * fmaxf(zz, 0.0f) : act_grad(zz, act);
              o = fmaf(ga, dphi, o);
            }
            outv[q] = o;
          }
          tc_fence_before();
          mbar_arrive_warp(sempty + pg * 2 + (use & 1));
        }
        if (valid) {
          if (P.dz_f32) {
            float* o = reinterpret_cast<float*>(P.dz) + (dzrow - P.dz) + hf * 8;
            *reinterpret_cast<float4*>(o) = make_float4(outv[0], outv[1], outv[2], outv[3]);
            *reinterpret_cast<float4*>(o + 4) = make_float4(outv[4], outv[5], outv[6], outv[7]);
          } else {
            *reinterpret_cast<uint4*>(dzrow + hf * 8) =
                make_uint4(pack_bf2(outv[0], outv[1]), pack_bf2(outv[2], outv[3]), pack_bf2(outv[4], outv[5]),
                           pack_bf2(outv[6], outv[7]));
          }
        }
      }
    }
    // ---- epilogue: the slab's accumulators -> float32 partial of this token split
    if (P.roles & 2) mbar_wait(done + 1, 0, wc);
    tc_fence_after();
    const int lane_row = (warp & 3) * 32 + lane;
    const int rows = kSlabKeys * L;
    float* part = P.part + ((size_t)blockIdx.y * P.h + key0) * L * r;
    for (int mt = pg; mt < P.mtiles && (P.roles & 2); mt += 2) {
      const int rr = mt * 128 + lane_row;
      const bool ok = rr < rows;
      float* dst = part + (size_t)rr * r;
      const uint32_t taddr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + dcol0 + (uint32_t)(mt * r);
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
    tc_fence_before();
  } else if (warp < kAux0) {
    // ------------------------------------------------------------------ Phi role
    reg_dec<kRegsPhi>();
    const int pg = (warp - 8) >> 2;
    const int t = tid & 127;
    const int tok = t & 63, kh = t >> 6;             // token of the half tile, key half of the slab
    const uint32_t t_off = (uint32_t)(tok & 7) * 16u + (uint32_t)(tok >> 3) * 128u;
    const uint32_t row0 = smem_u32(phi_base + (size_t)(pg * 2) * phi_bytes) + t_off;
    const uint32_t halfL = (uint32_t)L >> 1;
    // first word index (< 16 * L / 2 <= 255) of the pair each key wrote, per stage: 8 keys x 8 bits
    // in two registers; the positions are cleared before the stage is filled again
    uint32_t sav[2][2] = {{0u, 0u}, {0u, 0u}};
    // fill f of this group: tile pg + 2 * (f / 2), token half f % 2, stage f % 2
    const int nfill = 2 * ((ntiles - pg + 1) / 2);
    auto load_z = [&](int f, uint4& zv, bool& valid) {
      const int ti = pg + 2 * (f >> 1);
      const int64_t n = (tile_begin + ti) * 128 + (f & 1) * 64 + tok;
      valid = f < nfill && n < P.N;
      zv = valid ? ld16(P.z + n * P.zs + key0 + kh * 8) : make_uint4(0, 0, 0, 0);
    };
    uint4 znext;
    bool vnext;
    load_z(0, znext, vnext);
#pragma unroll 1
    for (int f = 0; f < nfill && (P.roles & 2); ++f) {
      const int st = f & 1;
      const uint4 zc = znext;
      const bool valid = vnext;
      load_z(f + 1, znext, vnext);                   // the next fill's rows are requested now
      const uint32_t row = row0 + (uint32_t)st * phi_bytes;
      // the stage is free once the dC MMAs of its previous fill are done
      if (f > 1) mbar_wait(pempty + pg * 2 + st, (uint32_t)((f >> 1) - 1) & 1u, wc);
#pragma unroll 1
      for (int i = 0; i < 2; ++i) {                  // 4 keys per pass (small body, see the dz role)
        const uint32_t zw[2] = {i ? zc.z : zc.x, i ? zc.w : zc.y};
        const uint32_t old = st ? (i ? sav[1][1] : sav[1][0]) : (i ? sav[0][1] : sav[0][0]);
        uint32_t now = 0u;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (f > 1) {
            const uint32_t c0 = (old >> (8 * q)) & 0xffu, c1 = c0 + 1u;
            sts32(row + (c0 + (c0 >> 2) * 252u) * 4u, 0u);
            sts32(row + (c1 + (c1 >> 2) * 252u) * 4u, 0u);
          }
          const float zz = (q & 1) ? bf_hi(zw[q >> 1]) : bf_lo(zw[q >> 1]);
          uint32_t x0, x1, s0;
          phi_pair_s(zz, P.g, (uint32_t)(kh * 8 + i * 4 + q) * halfL, x0, x1, s0);
          if (!valid) { x0 = 0u; x1 = 0u; }
          const uint32_t s1 = s0 + 1u;
          sts32(row + (s0 + (s0 >> 2) * 252u) * 4u, x0);
          sts32(row + (s1 + (s1 >> 2) * 252u) * 4u, x1);
          now |= s0 << (8 * q);
        }
        if (st) { if (i) sav[1][1] = now; else sav[1][0] = now; }
        else { if (i) sav[0][1] = now; else sav[0][0] = now; }
      }
      fence_async_smem();
      mbar_arrive_warp(pfull + pg * 2 + st);
    }
  } else {
    reg_dec<kRegsAux>();
    if (warp == kAux0) {
      // ---------------------------------------------------------------- S MMAs (both groups)
      if ((P.roles & 1) && elect_one()) {
        mbar_wait(tfull, 0, wc);
        const uint32_t rb = (uint32_t)(r / 8) * 128u;
        const uint32_t a_hi = desc_hi(128u), b_hi = desc_hi(rb);
        const uint32_t idesc = instr_desc(0, 0, 0, 0, 128, (int)bcols);
        // whichever group is ready first is served (the groups drift apart; serving them in a fixed
        // order would tie each to the slower one)
        int it[2] = {0, 0};
        const int total[2] = {4 * ((ntiles + 1) / 2), 4 * (ntiles / 2)};
        long long t_last = clock64();
        while ((it[0] < total[0] || it[1] < total[1]) && !*abort_flag) {
          bool progressed = false;
#pragma unroll
          for (int pg = 0; pg < 2; ++pg) {
            if (it[pg] >= total[pg]) continue;
            const int k = it[pg], ti = pg + 2 * (k >> 2), qt = k & 3, sb = k & 1, b = ti % kGRing;
            if (qt == 0 && !mbar_test_wait(gfull + b, (uint32_t)(ti / kGRing) & 1u)) continue;
            if (k > 1 && !mbar_test_wait(sempty + pg * 2 + sb, (uint32_t)((k >> 1) - 1) & 1u)) continue;
            tc_fence_after();
            uint32_t a_lo = desc_lo(smem_u32(g_base + (size_t)b * g_bytes), 2048u);
            uint32_t b_lo = desc_lo(smem_u32(t_base) + (uint32_t)qt * (uint32_t)(LP / 2) * rb, 128u);
            const uint32_t d_addr = tmem_base + (uint32_t)(pg * 2 + sb) * bcols;
            for (int ks = 0; ks < r / 16; ++ks) {
              umma_f16_split(d_addr, a_lo, a_hi, b_lo, b_hi, idesc, ks > 0 ? 1u : 0u);
              a_lo += 4096u >> 4;
              b_lo += 256u >> 4;
            }
            umma_commit(sfull + pg * 2 + sb);
            if (qt == 3) umma_commit(gempty + b);        // this issuer is done with the g tile
            ++it[pg];
            progressed = true;
          }
          if (progressed) t_last = clock64();
          else if (clock64() - t_last > P.wait_cycles) wait_give_up(wc);
          else __nanosleep(kPollNs);
        }
        umma_commit(done + 0);
      }
    } else if (warp == kAux0 + 1) {
      // ---------------------------------------------------------------- dC MMAs (both groups)
      if ((P.roles & 2) && elect_one()) {
        const uint32_t idesc = instr_desc(0, 0, 1, 1, 128, r);
        const uint32_t a_hi = desc_hi(1024u), b_hi = desc_hi(2048u);
        int it[2] = {0, 0};
        const int total[2] = {2 * ((ntiles + 1) / 2), 2 * (ntiles / 2)};
        bool first = true;
        long long t_last = clock64();
        while ((it[0] < total[0] || it[1] < total[1]) && !*abort_flag) {
          bool progressed = false;
#pragma unroll
          for (int pg = 0; pg < 2; ++pg) {
            if (it[pg] >= total[pg]) continue;
            const int f = it[pg], ti = pg + 2 * (f >> 1), st = f & 1, b = ti % kGRing;
            if (!mbar_test_wait(pfull + pg * 2 + st, (uint32_t)(f >> 1) & 1u)) continue;
            if (!mbar_test_wait(gfull + b, (uint32_t)(ti / kGRing) & 1u)) continue;
            tc_fence_after();
            const uint32_t a_addr = smem_u32(phi_base + (size_t)(pg * 2 + st) * phi_bytes);
            // tokens 64 * st .. of the g tile: token groups 8 * st ..
            const uint32_t b_lo0 = desc_lo(smem_u32(g_base + (size_t)b * g_bytes) + (uint32_t)st * 8u * 128u, 128u);
            for (int mt = 0; mt < P.mtiles; ++mt) {
              uint32_t a_lo = desc_lo(a_addr + (uint32_t)mt * 16u * 1024u, 128u);
              uint32_t b_lo = b_lo0;
              const uint32_t d_addr = tmem_base + dcol0 + (uint32_t)(mt * r);
              umma_f16_split(d_addr, a_lo, a_hi, b_lo, b_hi, idesc, first ? 0u : 1u);
#pragma unroll
              for (int ks = 1; ks < 4; ++ks) {
                a_lo += 256u >> 4;
                b_lo += 256u >> 4;
                umma_f16_split(d_addr, a_lo, a_hi, b_lo, b_hi, idesc, 1u);
              }
            }
            first = false;
            umma_commit(pempty + pg * 2 + st);
            if (st == 1) umma_commit(gempty + b);
            ++it[pg];
            progressed = true;
          }
          if (progressed) t_last = clock64();
          else if (clock64() - t_last > P.wait_cycles) wait_give_up(wc);
          else __nanosleep(kPollNs);
        }
        umma_commit(done + 1);
      }
    } else if (warp == kAux0 + 2) {
      // ---------------------------------------------------------------- loader
      if (elect_one()) {
        mbar_arrive_expect_tx(tfull, 2 * t_bytes);
        bulk_g2s(t_base, reinterpret_cast<const uint8_t*>(P.timg) + (size_t)(key0 / kChunkKeys) * t_bytes,
                 2 * t_bytes, tfull);
        for (int ti = 0; ti < ntiles; ++ti) {
          const int b = ti % kGRing;
          if (ti >= kGRing) mbar_wait(gempty + b, (uint32_t)((ti / kGRing) - 1) & 1u, wc);
          if (*abort_flag) break;
          mbar_arrive_expect_tx(gfull + b, g_bytes);
          bulk_g2s(g_base + (size_t)b * g_bytes,
                   reinterpret_cast<const uint8_t*>(P.gimg) + (size_t)(tile_begin + ti) * g_bytes, g_bytes, gfull + b);
        }
        if (*abort_flag) {
          const long long t0 = clock64();
          while (clock64() - t0 < 2000000) {}
        }
      }
    }
  }
  __syncthreads();
  if (warp == kAux0) {
    if (P.roles & 1) mbar_wait_drain(done + 0, 0, P.wait_cycles);
    if (P.roles & 2) mbar_wait_drain(done + 1, 0, P.wait_cycles);
    tc_fence_after();
    tmem_free(tmem_base, tmem_cols);
  }
}

}  // namespace

// The fused kernel covers shapes whose slab fits: even L up to 24 (16 keys x L rows in three M-tiles),
// r small enough for the tensor-memory plan, h a multiple of the slab.
bool plan_fused(const skv_problem& p, FusedPlan* o) {
  if (p.spline_order == 1 || p.L % 2 || p.L > 24 || p.h % kSlabKeys || p.N < 1) return false;
  const int rp = padded_r(p);
  const int lb = (p.L - 1 + 7) / 8;
  if (lb < 1 || lb > 3) return false;
  const int mtiles = (kSlabKeys * p.L + 127) / 128;
  if (2 * kChunkKeys * 8 * lb + mtiles * rp > 512) return false;
  const size_t phi_bytes = (size_t)((kSlabKeys * p.L + 7) / 8) * 1024;      // one 64-token stage
  const size_t smem = 4 * phi_bytes + (size_t)kGRing * 128 * rp * 2 + 2 * (size_t)kChunkKeys * 8 * lb * rp * 2 + 256;
  if (smem > kSmemLimit) return false;
  // the last M-tile of the last stage reads past the stage: that read must stay inside the allocation
  if (3 * phi_bytes + (size_t)mtiles * 16 * 1024 > smem) return false;
  o->lb = lb;
  o->mtiles = mtiles;
  o->slabs = p.h / kSlabKeys;
  o->smem = smem;
  o->tiles_total = (p.N + 127) / 128;
  const int64_t tt = o->tiles_total;
  int best = 1;
  double best_eff = 0.0;
  const int64_t max_splits = tt / 4 < 1 ? 1 : (tt / 4 > 32 ? 32 : tt / 4);
  for (int ns = 1; ns <= max_splits; ++ns) {
    const double waves = (double)o->slabs * ns / kPlanSMs;
    const double eff = waves / (double)(int64_t)(waves + 0.999999);
    if (eff > best_eff + 0.04) { best_eff = eff; best = ns; }
  }
  o->tiles_per_split = (tt + best - 1) / best;
  o->splits = (int)((tt + o->tiles_per_split - 1) / o->tiles_per_split);
  return true;
}

cudaError_t fused_launch(const FusedPlan& fp, int L, const DzParams& Z, float* part, cudaStream_t stream) {
  BfParams P;
  P.z = Z.z;
  P.zs = Z.zs;
  P.g_act = Z.g_act;
  P.gas = Z.gas;
  P.dz = Z.dz;
  P.dzs = Z.dzs;
  P.gimg = Z.gimg;
  P.timg = Z.timg;
  P.amax_bits = Z.amax_bits;
  P.part = part;
  P.N = Z.N;
  P.h = Z.h;
  P.L = Z.L;
  P.r = Z.r;
  P.g = Z.g;
  P.act = Z.act;
  P.coef = Z.coef;
  P.mtiles = fp.mtiles;
  P.dz_f32 = Z.dz_f32;
  P.roles = fused_backward_roles();
  P.tiles_per_split = fp.tiles_per_split;
  P.tiles_total = fp.tiles_total;
  P.status = Z.status;
  P.wait_cycles = Z.wait_cycles;
  const dim3 grid((unsigned)fp.slabs, (unsigned)fp.splits);
  const bool relu = Z.act == SKV_ACT_RELU_SQ;
#define SKV_BF_CASE(LB_, NC_, COND_)                                                                                 \
  if (fp.lb == LB_ && (COND_))                                                                                       \
    return relu ? launch_chained<tc_bwd_fused_kernel<LB_, NC_, true>>(grid, kBfThreads, fp.smem, stream, P)          \
                : launch_chained<tc_bwd_fused_kernel<LB_, NC_, false>>(grid, kBfThreads, fp.smem, stream, P);
  SKV_BF_CASE(3, 21, L == 22) SKV_BF_CASE(2, 15, L == 16) SKV_BF_CASE(1, 8, true) SKV_BF_CASE(2, 16, true)
  SKV_BF_CASE(3, 24, true)
#undef SKV_BF_CASE
  return cudaErrorInvalidValue;
}

}  // namespace tc
}  // namespace skv
