// Forward of the tensor-core family: which problems it takes, the launch shape, the chain of launches
// (scan C, build its operand image, contract, add the key splits).
#include "skv_tc_fwd_kernel.cuh"

namespace skv {
namespace tc {

cudaError_t fwd_launch_quad_relu(int, int, const FwdParams&, dim3, size_t, cudaStream_t);
cudaError_t fwd_launch_quad_other(int, int, const FwdParams&, dim3, size_t, cudaStream_t);
cudaError_t fwd_launch_split_relu(int, int, const FwdParams&, dim3, size_t, cudaStream_t);
cudaError_t fwd_launch_split_other(int, int, const FwdParams&, dim3, size_t, cudaStream_t);
cudaError_t fwd_launch_lin_relu(int, int, const FwdParams&, dim3, size_t, cudaStream_t);
cudaError_t fwd_launch_lin_other(int, int, const FwdParams&, dim3, size_t, cudaStream_t);

namespace {

struct FwdPlan {
  int groups, fold, splits, chunks_per_split, cstages;
  size_t smem;
};

size_t fwd_cimg_bytes(const skv_problem& p) {
  return align256((size_t)padded_h(p) * 4 * fwd_fold(p.L) * padded_r(p) * sizeof(__half));
}

FwdPlan make_plan(const skv_problem& p) {
  FwdPlan f{};
  const int rp = padded_r(p);
  const int F = f.fold = fwd_fold(p.L);
  const int chunks = padded_h(p) / kChunkKeys;
  const int64_t N = p.N > 0 ? p.N : 1;
  const size_t c_bytes = (size_t)kChunkKeys * 4 * F * rp * 2;
  // Splits are bounded by what their partials may take: below 16 MiB of scratch together with the image, or
  // sixteen of them.  A split of fewer than four chunks is mostly prologue.
  const size_t part = (size_t)N * rp * sizeof(float);
  const size_t room = (size_t)SKV_NOALLOC_SCRATCH_BYTES - kHeaderBytes - 256;
  int64_t most = room > fwd_cimg_bytes(p) ? (int64_t)((room - fwd_cimg_bytes(p)) / part) : 0;
  if (most < 16) most = 16;
  if (most > (chunks + 3) / 4) most = (chunks + 3) / 4;
  double best = 0.0;
  for (int g = fwd_max_groups(F, rp, split_operands(p)); g >= 1; --g) {
    const size_t stage_bytes = (size_t)128 * g * (F + 1) * 4;
    int cstages = (int)((kSmemLimit - 512 - stage_bytes) / c_bytes);
    if (cstages > kMaxCStages) cstages = kMaxCStages;
    // what the ring does not need is L1 for the strided rows of z and phi(z)
    while (cstages > 3 && cstages * c_bytes + stage_bytes + 512 > kSmemOnePerSM) --cstages;
    if (cstages < 2) continue;
    const int64_t tiles = (N + 128 * g - 1) / (128 * g);
    // microseconds: a chunk of g groups (instruction issue, or the MMAs of wide r), a CTA's prologue and
    // epilogue, and the partials' way through L2 and their sum, eight loads at a time (measured: 1.3 us per chunk of four groups at L = 22, 0.9
    // of one: four warps cannot hide their own latencies)
    const double issue = (0.75 + 0.14 * g) * (F + 14) / 20.0 * (split_operands(p) ? 1.4 : 1.0), mma = g * F * rp * 0.5 / 1800.0;
    const double chunk = issue > mma ? issue : mma;
    int last = 0;
    for (int64_t s = 1; s <= most; ++s) {
      const int per = (int)((chunks + s - 1) / s), splits = (chunks + per - 1) / per;
      if (splits == last) continue;
      last = splits;
      const double t = (double)((tiles * splits + kPlanSMs - 1) / kPlanSMs) * (per * chunk + 4.5) +
                       splits * (part * 2.0 / 4.0e6 + 0.08);
      if (best == 0.0 || t < best) {
        best = t;
        f.groups = g;
        f.splits = splits;
        f.chunks_per_split = per;
        f.cstages = cstages;
        f.smem = (size_t)cstages * c_bytes + stage_bytes + 512;       // ring + staging rows + barriers
        if (f.smem < kSmemOnePerSM) f.smem = kSmemOnePerSM;
      }
    }
  }
  return f;
}

// The plan of the last problem this thread asked about: a call asks several times (scratch size, launch).
const FwdPlan& plan_forward(const skv_problem& p) {
  static thread_local struct { int64_t N; int h, L, r, order; FwdPlan f; } last{-1, 0, 0, 0, 0, {}};
  if (last.N != p.N || last.h != p.h || last.L != p.L || last.r != p.r || last.order != p.spline_order)
    last = {p.N, p.h, p.L, p.r, p.spline_order, make_plan(p)};
  return last.f;
}

// Rows of z (and of act_out) the kernel can move in 16-byte pieces; otherwise z is copied to padded rows.
size_t fwd_copy_bytes(const skv_problem& p) { return align256((size_t)(p.N > 0 ? p.N : 1) * padded_h(p) * 2); }

}  // namespace

bool fwd_eligible(const skv_problem& p) {
  if (p.dtype != SKV_BF16 || p.r > 128 || p.L < 4 || p.L > 64) return false;
  const int F = fwd_fold(p.L), rp = padded_r(p);
  return fwd_max_groups(F, rp, split_operands(p)) >= 1 &&
         2 * (size_t)kChunkKeys * 4 * F * rp * 2 + (size_t)128 * (F + 1) * 4 + 512 <= kSmemLimit;
}

// `rows_ok`: the token-major arrays can be read and written in place.
size_t fwd_scratch_bytes(const skv_problem& p, bool rows_ok) {
  const FwdPlan& f = plan_forward(p);
  return kHeaderBytes + fwd_cimg_bytes(p) + align256((size_t)f.splits * (p.N > 0 ? p.N : 1) * padded_r(p) * sizeof(float)) +
         (rows_ok ? 0 : fwd_copy_bytes(p));
}

int forward(const LaunchCtx& c, const void* z, int64_t zs, const void* C, void* act_out, int64_t as,
            void* delta_out, int64_t ds, void* scratch, bool rows_ok) {
  const skv_problem& p = c.p;
  const FwdPlan& f = plan_forward(p);
  const int hp = padded_h(p), rp = padded_r(p), lp = 4 * f.fold;
  uint8_t* base = static_cast<uint8_t*>(scratch);
  uint32_t* hdr = reinterpret_cast<uint32_t*>(base);
  __half* img = reinterpret_cast<__half*>(base + kHeaderBytes);
  float* partial = reinterpret_cast<float*>(base + kHeaderBytes + fwd_cimg_bytes(p));

  PrepParams Q{};
  Q.C = static_cast<const __nv_bfloat16*>(C);
  Q.h = p.h; Q.hp = hp; Q.L = p.L; Q.r = p.r; Q.rp = rp;
  Q.lpc = lp;
  Q.cimg = img;
  Q.N = p.N;
  Q.act = p.activation;
  Q.hdr = hdr;
  Q.contain = split_operands(p);
  if (!rows_ok) {
    __nv_bfloat16* zp = reinterpret_cast<__nv_bfloat16*>(
        base + kHeaderBytes + fwd_cimg_bytes(p) + align256((size_t)f.splits * p.N * rp * sizeof(float)));
    Q.copy[0] = {static_cast<const __nv_bfloat16*>(z), zs, zp, static_cast<__nv_bfloat16*>(act_out), as};
    z = zp;
    zs = hp;
    act_out = nullptr;                                   // written by the copy
  }
  if (int e = launch_prep(Q, c)) return e;

  FwdParams P;
  P.z = static_cast<const __nv_bfloat16*>(z);
  P.zs = zs;
  P.act_out = static_cast<__nv_bfloat16*>(act_out);
  P.as = as;
  P.cimg = img;
  P.partial = partial;
  P.N = p.N;
  P.r = rp;
  P.g = c.g;
  P.act = p.activation;
  P.chunks_total = hp / kChunkKeys;
  P.chunks_per_split = f.chunks_per_split;
  P.status = c.status;
  P.cstages = f.cstages;
  P.wait_cycles = wait_cycle_limit();
  P.skip_copy = debug_skip_copy() == 1;
  // B: code-table chunk, N(=channel)-major; core matrices 128 B apart along channels, r/8*128 B along k
  P.b_lbo = (uint32_t)(rp / 8) * 128u;
  P.b_sbo = 128;
  const dim3 grid((unsigned)((p.N + 128 * f.groups - 1) / (128 * f.groups)), (unsigned)f.splits);
  const bool lin = c.g.order == 1, relu = p.activation == SKV_ACT_RELU_SQ;
  auto* launch = lin                 ? (relu ? fwd_launch_lin_relu : fwd_launch_lin_other)
                 : split_operands(p) ? (relu ? fwd_launch_split_relu : fwd_launch_split_other)
                                     : (relu ? fwd_launch_quad_relu : fwd_launch_quad_other);
  if (launch(f.groups, f.fold, P, grid, f.smem, c.stream) != cudaSuccess) { cudaGetLastError(); return SKV_ERR_LAUNCH; }
  note_launches(1);
  Contain K{};
  if (Q.contain) {
    K.z = P.z; K.zs = zs; K.C = Q.C; K.N = p.N;
    K.h = p.h; K.L = p.L; K.r = p.r; K.grid = c.g;
  }
  return launch_finalize(partial, f.splits, p.N, p.r, rp, p.lambda_scale, hdr, delta_out, ds, p.delta_f32 != 0, K, c.stream);
}

}  // namespace tc
}  // namespace skv
