// Backward of the tensor-core family: which problems it takes, launch shapes, the chain of launches (scan and
// pack g and C, dz, dC, add the token splits).
//
// The upstream gradient is converted once per call to f16, multiplied by a power of two chosen
// from its largest magnitude so that small gradients do not underflow; the inverse factor is
// applied to the float32 results.
#include "skv_tc_bwd_fused.cuh"
#include "skv_tc_dc_kernel.cuh"
#include "skv_tc_dz_kernel.cuh"

namespace skv {
namespace tc {

bool fwd_eligible(const skv_problem& p);
cudaError_t dz_launch_quad(const DzPlan&, int L, bool relu, const DzParams&, dim3, cudaStream_t);
cudaError_t dz_launch_split(const DzPlan&, int L, bool relu, const DzParams&, dim3, cudaStream_t);
cudaError_t dz_launch_lin(const DzPlan&, int L, bool relu, const DzParams&, dim3, cudaStream_t);
cudaError_t dc_launch(const DcPlan&, bool lin, bool split, const DcParams&, dim3, cudaStream_t);

namespace {

// Splits s of `units` of work per tile, `tiles` tiles: waves of CTAs on the chip, each with its share of the
// units and a fixed prologue (both in microseconds), and what one more split costs.
struct Split { int splits, per; double time; };
Split best_split(int64_t tiles, int64_t units, int64_t most, double unit, double prologue, double per_split) {
  Split b{1, (int)units, 0.0};
  int64_t last = 0;
  for (int64_t s = 1; s <= most; ++s) {
    const int64_t per = (units + s - 1) / s, splits = (units + per - 1) / per;
    if (splits == last) continue;
    last = splits;
    const double t = (double)((tiles * splits + kPlanSMs - 1) / kPlanSMs) * (per * unit + prologue) + splits * per_split;
    if (b.time == 0.0 || t < b.time) b = {(int)splits, (int)per, t};
  }
  return b;
}

bool make_dz_plan(const skv_problem& p, DzPlan* o) {
  const int lb = (p.L - 1 + 7) / 8, rp = padded_r(p);    // 8-column blocks per key; columns L-1.. are padding
  const int parts = split_operands(p) ? 2 : 1;
  if (lb < 1 || lb > 8) return false;
  o->lb = lb;
  // two token groups where their rows, g and the table ring fit shared memory
  bool fits = false;
  for (int groups = 2; groups >= 1 && !fits; --groups)
    for (int rs = kRowStages; rs >= 2 && !fits; --rs)
      for (int ts = kTStages; ts >= 2 && !fits; --ts) {
        o->groups = groups;
        o->rstages = rs;
        o->tstages = ts;
        o->smem = 1024 + (size_t)groups * rs * 2 * kBoxBytes + (size_t)groups * 128 * rp * 2 +
                  (size_t)ts * kChunkKeys * 8 * lb * rp * parts * 2 + 512;
        fits = o->smem <= kSmemLimit;
      }
  if (!fits) return false;
  const int groups = o->groups;
  if (o->smem < kSmemOnePerSM) o->smem = kSmemOnePerSM;
  const int chunks = padded_h(p) / kChunkKeys;
  const int64_t tiles = ((p.N > 0 ? p.N : 1) + 128 * groups - 1) / (128 * groups);
  // 1.0 us per chunk of two groups at L = 22, r = 32; the MMAs grow with r
  const double chunk = 0.5 * groups * lb / 3.0 * (0.8 + rp / 160.0);
  const int boxes = (chunks + kBoxChunks - 1) / kBoxChunks;                  // a split is a whole number of boxes
  const Split s = best_split(tiles, boxes, boxes, chunk * kBoxChunks, 4.5, 0.0);
  o->chunks_per_split = s.per * kBoxChunks;
  o->splits = s.splits;
  return true;
}

bool make_dc_plan(const skv_problem& p, DcPlan* o) {
  const int words = (p.L + 1) / 2, rp = padded_r(p), hp = padded_h(p);
  for (int kj = 4; kj >= 2; kj /= 2) {
    const int kch = 4 * kj, mtiles = (kch * 2 * words + 127) / 128;
    if (mtiles * rp > 512) continue;
    // as many producer groups (stages) as fit shared memory beside a longer ring of g tiles; two groups of eight
    // warps where it cannot be three of four
    const size_t stage = dc_stage_bytes(mtiles), slot = (size_t)kDcTokens * rp * 2;
    int ng = kDcMaxGroups;
    while (ng > 1 && ng * stage + (ng + 1) * slot + 512 > kSmemLimit) --ng;
    if (ng < 2) continue;
    o->kj = kj;
    o->gw = ng >= 3 ? 4 : 8;
    o->ngroups = ng;
    int ring = (int)((kSmemLimit - 512 - ng * stage) / slot);
    o->gring = ring > kDcMaxRing ? kDcMaxRing : ring;
    o->mtiles = mtiles;
    o->smem = ng * stage + o->gring * slot + 512;
    if (o->smem < kSmemOnePerSM) o->smem = kSmemOnePerSM;
    int most = 512 / (mtiles * rp);
    if (most > 8) most = 8;
    const int chunks = (hp + kch - 1) / kch;
    const int64_t tiles = ((p.N > 0 ? p.N : 1) + kDcTokens - 1) / kDcTokens;
    if (tiles >= 1ll << 31) return false;                    // places are counted in 32 bits
    o->tiles = (uint32_t)tiles;
    // 0.38 us per tile and chunk of 16 keys at L = 22, r = 32, and the wait for a tile's g; a CTA's prologue, an epilogue per
    // segment; a segment's partials written and read again through L2 or HBM
    const double unit = 0.38 * (split_operands(p) ? 1.6 : 1.0) * kch / 16.0 * words / 11.0 * (0.8 + rp / 160.0), tile = 0.002 * rp;
    const double per_part = (double)hp * p.L * rp * 8.0 / 5.0e6 + 0.1;
    o->chain = split_operands(p) ? kDcSplitChain : kDcChain;
    // what a CTA pays for the segments of a slab after its first: its accumulators' way to the partial (8 to 10 us for 480
    // columns of tensor memory, 1.5 to 3 for 96)
    auto flush = [&](uint64_t run, uint64_t T, int slab) {
      const uint64_t len = run < T ? run : T;
      return (double)((len - 1) / o->chain * (run / len)) * (1.0 + 0.017 * slab * mtiles * rp);
    };
    double best = 0.0;
    for (int slab = most < chunks ? most : chunks; slab >= 1; --slab) {
      const uint64_t slabs = (chunks + slab - 1) / slab, T = o->tiles;
      auto take = [&](double t, bool runs, uint64_t run, uint64_t pitch, uint64_t parts) {
        if ((best != 0.0 && t >= best) || slabs * pitch >= 1ull << 31) return;
        best = t;
        o->slab_chunks = slab;
        o->runs = runs;
        o->pitch = (uint32_t)pitch;
        o->run = (uint32_t)run;
        o->total = (uint32_t)(slabs * pitch);
        o->parts = (int)parts;
      };
      // runs within a slab
      uint64_t last = 0;
      for (uint64_t n = 1; n <= 32; ++n) {
        const uint64_t run = (T + n - 1) / n, s = (T + run - 1) / run;
        if (s == last) continue;
        last = s;
        const double waves = (double)((slabs * s + kPlanSMs - 1) / kPlanSMs);
        take(waves * (run * (unit * slab + tile) + 4.0 + 0.8 * slab + flush(run, T, slab)) + s * per_part, false, run,
             run * s, s);
      }
      // One run per SM over all slabs.  Where a slab is a whole number of runs none crosses: as many partials as runs then,
      // else up to one more than fit, the first and the last of them shorter.
      const uint64_t run = (slabs * T + kPlanSMs - 1) / kPlanSMs;
      const double segs = (double)((run + T - 1) / T) + 1.0;
      const bool cross = T % run != 0;
      take(run * (unit * slab + tile) + 4.0 + segs * (0.8 * slab + 6.0) + flush(run, T, slab) +
               ((double)T / run + 1.0) * per_part, cross, run, T, cross ? (T - 1) / run + 2 : T / run);
    }
    return best != 0.0;
  }
  return false;
}

struct BwdPlan { bool ok; DzPlan dz; DcPlan dc; };

// The plans of the last problem this thread asked about: a call asks several times (eligibility, scratch, launch).
const BwdPlan& plan_backward(const skv_problem& p) {
  static thread_local struct { int64_t N; int h, L, r, order; BwdPlan b; } last{-1, 0, 0, 0, 0, {}};
  if (last.N != p.N || last.h != p.h || last.L != p.L || last.r != p.r || last.order != p.spline_order) {
    BwdPlan b{};
    b.ok = make_dz_plan(p, &b.dz) && make_dc_plan(p, &b.dc);
    last = {p.N, p.h, p.L, p.r, p.spline_order, b};
  }
  return last.b;
}

// What the reduce adds for the knot rows of a slab under this plan.
DcParts dc_parts(const DcPlan& d, int L) {
  return {d.runs ? 0 : d.parts, d.pitch, d.run, (uint32_t)(d.slab_chunks * 4 * d.kj * L)};
}

size_t timg_bytes(const skv_problem& p) {
  return align256((size_t)padded_h(p) * 8 * ((p.L - 1 + 7) / 8) * padded_r(p) * sizeof(__half)) * (split_operands(p) ? 2 : 1);
}

int64_t gimg_tiles(const skv_problem& p) { return ((p.N > 0 ? p.N : 1) + 255) / 256 * 2; }
size_t gimg_bytes(const skv_problem& p) { return align256((size_t)gimg_tiles(p) * 128 * padded_r(p) * 2); }

size_t part_bytes(const skv_problem& p) {
  int splits = plan_backward(p).dc.parts;
  FusedPlan f;
  if (fused_backward_roles() && plan_fused(p, &f) && f.splits > splits) splits = f.splits;
  return align256((size_t)splits * padded_h(p) * p.L * padded_r(p) * sizeof(float));
}

// Padded copies of z and g_act and a padded dz, when their rows cannot be used in place.
size_t row_bytes(const skv_problem& p, int esz) { return align256((size_t)(p.N > 0 ? p.N : 1) * padded_h(p) * esz); }

}  // namespace

bool bwd_eligible(const skv_problem& p) { return fwd_eligible(p) && plan_backward(p).ok; }

void describe_dc_plan(const skv_problem& p, int64_t slab, int64_t* out) {
  const DcPlan& d = plan_backward(p).dc;
  const int64_t v[8] = {d.runs, d.tiles, d.pitch, d.run, d.total, d.parts, d.slab_chunks * 4 * d.kj,
                        dc_parts(d, p.L).of((uint32_t)slab)};
  for (int i = 0; i < 8; ++i) out[i] = v[i];
}

size_t bwd_scratch_bytes(const skv_problem& p, bool rows_ok) {
  return kHeaderBytes + gimg_bytes(p) + timg_bytes(p) + part_bytes(p) +
         (rows_ok ? 0 : 2 * row_bytes(p, 2) + row_bytes(p, p.dz_f32 ? 4 : 2));
}

int backward(const LaunchCtx& c, const void* z, int64_t zs, const void* C, const void* g_act, int64_t gas,
             const void* g_delta, int64_t gds, void* dz, int64_t dzs, float* dC, void* dC_cast, void* scratch,
             bool rows_ok) {
  const skv_problem& p = c.p;
  const BwdPlan& b = plan_backward(p);
  const bool want_dC = dC || dC_cast, lin = c.g.order == 1, split = split_operands(p);
  const int hp = padded_h(p), rp = padded_r(p);
  uint8_t* base = static_cast<uint8_t*>(scratch);
  uint32_t* hdr = reinterpret_cast<uint32_t*>(base);
  uint8_t* next = base + kHeaderBytes;
  __half* gimg = reinterpret_cast<__half*>(next);
  next += gimg_bytes(p);
  __half* timg = reinterpret_cast<__half*>(next);
  next += timg_bytes(p);
  float* part = reinterpret_cast<float*>(next);
  next += part_bytes(p);

  PrepParams Q{};
  Q.C = static_cast<const __nv_bfloat16*>(C);
  Q.h = p.h; Q.hp = hp; Q.L = p.L; Q.r = p.r; Q.rp = rp;
  if (dz) {
    Q.lpt = 8 * b.dz.lb;
    Q.tparts = split ? 2 : 1;
    Q.timg = timg;
  }
  Q.g = static_cast<const __nv_bfloat16*>(g_delta);
  Q.gds = gds;
  Q.N = p.N;
  Q.tiles = gimg_tiles(p);
  Q.gimg = gimg;
  Q.hdr = hdr;
  Q.contain = split;
  void* user_dz = dz;
  const int64_t user_dzs = dzs;
  if (!rows_ok) {
    __nv_bfloat16* zp = reinterpret_cast<__nv_bfloat16*>(next);
    __nv_bfloat16* gap = reinterpret_cast<__nv_bfloat16*>(next + row_bytes(p, 2));
    Q.copy[0] = {static_cast<const __nv_bfloat16*>(z), zs, zp, nullptr, 0};
    z = zp;
    zs = hp;
    if (dz && g_act) {
      Q.copy[1] = {static_cast<const __nv_bfloat16*>(g_act), gas, gap, nullptr, 0};
      g_act = gap;
      gas = hp;
    }
    if (dz) {
      dz = next + 2 * row_bytes(p, 2);
      dzs = hp;
    }
  }
  FusedPlan fp;
  const bool fused = fused_backward_roles() && rows_ok && !split && dz && want_dC && plan_fused(p, &fp);
  if (fused) {                                           // C and g one after the other, as it has always run
    PrepParams G = Q;
    G.lpt = 0;
    Q.g = nullptr;
    if (int e = launch_prep(G, c)) return e;
  }
  if (int e = launch_prep(Q, c)) return e;

  DzParams Z;
  Z.z = static_cast<const __nv_bfloat16*>(z);
  Z.zs = zs;
  Z.g_act = static_cast<const __nv_bfloat16*>(g_act);
  Z.gas = gas;
  Z.dz = static_cast<__nv_bfloat16*>(dz);
  Z.dzs = dzs;
  Z.gimg = gimg;
  Z.timg = timg;
  Z.amax_bits = hdr;
  Z.N = p.N;
  Z.h = hp;
  Z.L = p.L;
  Z.r = rp;
  Z.g = c.g;
  Z.act = p.activation;
  Z.coef = p.lambda_scale * c.g.scale;
  Z.chunks_total = hp / kChunkKeys;
  Z.chunks_per_split = b.dz.chunks_per_split;
  Z.tstages = b.dz.tstages;
  Z.rstages = b.dz.rstages;
  Z.dz_f32 = p.dz_f32;
  Z.wait_cycles = wait_cycle_limit();
  Z.status = c.status;

  DcParts parts{1, 0, 0, 0};
  if (fused) {
    if (fused_launch(fp, p.L, Z, part, c.stream) != cudaSuccess) { cudaGetLastError(); return SKV_ERR_LAUNCH; }
    note_launches(1);
    parts.count = fp.splits;
  } else {
    if (dz) {
      const dim3 grid((unsigned)((p.N + 128 * b.dz.groups - 1) / (128 * b.dz.groups)), (unsigned)b.dz.splits);
      if ((lin ? dz_launch_lin : split ? dz_launch_split : dz_launch_quad)(b.dz, p.L, p.activation == SKV_ACT_RELU_SQ, Z, grid, c.stream) !=
          cudaSuccess) {
        cudaGetLastError();
        return SKV_ERR_LAUNCH;
      }
      note_launches(1);
    }
    if (want_dC) {
      DcParams P;
      P.z = static_cast<const __nv_bfloat16*>(z);
      P.zs = zs;
      P.gimg = gimg;
      P.part = part;
      P.N = p.N;
      P.h = hp;
      P.L = p.L;
      P.r = rp;
      P.g = c.g;
      P.words = (p.L + 1) / 2;
      P.ngroups = b.dc.ngroups;
      P.gring = b.dc.gring;
      P.mtiles = b.dc.mtiles;
      P.slab_chunks = b.dc.slab_chunks;
      P.tiles = b.dc.tiles;
      P.pitch = b.dc.pitch;
      P.run = b.dc.run;
      P.total = b.dc.total;
      P.chain = b.dc.chain;
      P.status = c.status;
      P.wait_cycles = wait_cycle_limit();
      if (dc_launch(b.dc, lin, split, P, dim3((b.dc.total + b.dc.run - 1) / b.dc.run), c.stream) != cudaSuccess) {
        cudaGetLastError();
        return SKV_ERR_LAUNCH;
      }
      note_launches(1);
      parts = dc_parts(b.dc, p.L);
    }
  }
  // padded rows of dz: brought to their place by the last kernel where there is one that knows how, else by one of its own
  const bool with_reduce = dz != user_dz && want_dC && split;
  if (dz != user_dz && !with_reduce)
    if (int e = launch_unpad(dz, dzs, user_dz, user_dzs, p.N, p.h, p.dz_f32 != 0, c.stream)) return e;
  Contain K{};
  if (split) {
    K.z = Z.z; K.zs = zs; K.C = Q.C; K.g = Q.g; K.gds = gds; K.N = p.N;
    K.h = p.h; K.L = p.L; K.r = p.r; K.grid = c.g;
    K.dz = user_dz; K.dzs = user_dzs;
    if (with_reduce) { K.dz_rows = dz; K.dz_rows_stride = dzs; }
    K.coef = Z.coef; K.dz_f32 = p.dz_f32 != 0;
  }
  if (want_dC)
    return launch_dc_reduce(part, parts, (int64_t)p.h * p.L, (int64_t)hp * p.L, p.r, rp, p.lambda_scale, hdr, dC,
                            dC_cast, K, c.stream);
  return split ? launch_dz_contain(K, hdr, c.stream) : (int)SKV_OK;
}

}  // namespace tc
}  // namespace skv
