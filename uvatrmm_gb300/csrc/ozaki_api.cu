// C ABI of the Ozaki-style emulated FP64 TRMM (see ozaki.cuh for the method).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <new>
#include <string>
#include <vector>

#include "api_internal.h"
#include "common.cuh"
#include "ozaki.cuh"

namespace uvt {
namespace {

constexpr int kErrSamples = 8;
static_assert(kHandleCountersOffset + kScaleTiles * sizeof(int) <= kHandleSlotsOffset &&
                  kHandleSlotsOffset + kFusedSlots * sizeof(unsigned long long) <= kHandleCtlBytes &&
                  kHandleCtlOffset + sizeof(OzCtl) <= kHandleCountersOffset,
              "the handle's control block holds the decision word and the scaling's counters");

// Builds the two residue operands of the canonical GEMM for a normalised TRMM.
void operands(const Trmm &t, const double *dA, int64_t lda, const double *dB, int64_t ldb, OzOperand &L,
              OzOperand &R) {
  const bool lower = (t.uplo == CblasLower) != (t.trans != 0);
  if (t.side == CblasLeft) {
    // Lft = op(A) (m x m), Rgt = B (m x n).
    L = OzOperand{dA, lda, t.m, t.m, t.trans != 0, true, true, lower, t.unit != 0};
    R = OzOperand{dB, ldb, t.n, t.m, true, false, false, false, false};
  } else {
    // Lft = B (m x n), Rgt = op(A) (n x n): Rgt[k, j] = op(A)[k, j].
    L = OzOperand{dB, ldb, t.m, t.n, false, false, false, false, false};
    R = OzOperand{dA, lda, t.n, t.n, t.trans == 0, true, false, lower, t.unit != 0};
  }
}

// Sample positions of the error report: S evenly spaced result columns
// (side Left) or rows (side Right) out of `cnt`.
int64_t sample_index(int S, int s, int64_t cnt) { return S > 1 ? (cnt - 1) * s / (S - 1) : 0; }

// Copies the S sampled vectors of the column-major matrix X (leading
// dimension ld; host memory, or device memory when `device`) into `out`,
// vector after vector.
int gather_samples(uvatrmm_handle_t h, const Trmm &t, int S, const double *X, int64_t ld, bool device,
                   double *out) {
  const bool left = t.side == CblasLeft;
  const int64_t len = left ? t.m : t.n, cnt = left ? t.n : t.m;
  for (int s = 0; s < S; ++s) {
    const int64_t idx = sample_index(S, s, cnt);
    double *o = out + (int64_t)s * len;
    if (device) {
      cudaError_t e = left ? cudaMemcpyAsync(o, X + idx * ld, len * 8, cudaMemcpyDeviceToHost, h->stream)
                           : cudaMemcpy2DAsync(o, 8, X + idx, ld * 8, 8, len, cudaMemcpyDeviceToHost, h->stream);
      if (e != cudaSuccess) return cuda_fail(e, "error-report sample");
    } else if (left) {
      std::memcpy(o, X + idx * ld, (size_t)len * 8);
    } else {
      for (int64_t k = 0; k < len; ++k) o[k] = X[idx + k * ld];
    }
  }
  if (device) {
    cudaError_t e = cudaStreamSynchronize(h->stream);
    if (e != cudaSuccess) return cuda_fail(e, "error-report sample");
  }
  return UVATRMM_OK;
}

// Slicing, residue GEMMs and reassembly of one integer product (the scales
// are known): C = alpha * Lft * Rgt + beta * C.
struct IntProduct {
  OzOperand L, R;
  OzPlan plan;
  bool tri_left = true, tri_lower = true, tri_none = false;
  double alpha = 1.0, beta = 0.0;
  double *C = nullptr, *stage = nullptr;
  int64_t ldc = 0, lds = 0;
  const int *e_row = nullptr, *e_col = nullptr;
  const OzCtl *ctl = nullptr;
  int G = 1;  // moduli per pass over the planes
  bool sliced = false;  // the planes are there already (one pass)
  uint16_t *planes = nullptr, *res = nullptr;
};

// `mark(kind)` follows every stage of each pass (1 slicing, 2 residue GEMM).
template <class Mark>
int int_product(uvatrmm_handle_t h, const IntProduct &ip, Mark &&mark) {
  const OzPlan &plan = ip.plan;
  for (int l0 = 0; l0 < plan.n_moduli; l0 += ip.G) {
    const int l1 = std::min(plan.n_moduli, l0 + ip.G);
    uint16_t *LR = ip.planes, *RR = ip.planes + (int64_t)(l1 - l0) * plan.Mp * plan.Kp;
    int rc = UVATRMM_OK;
    if (!ip.sliced) rc = oz_residues(ip.L, ip.R, ip.e_row, ip.e_col, plan, ip.ctl, l0, l1, LR, RR, h->stream);
    if (rc != UVATRMM_OK) return fail(rc, "Ozaki residue slicing failed to launch");
    mark(1);
    OzGemmLaunch g;
    g.LR = LR;
    g.RR = RR;
    g.res = ip.res;
    g.Mp = plan.Mp; g.Np = plan.Np; g.Kp = plan.Kp;
    g.M = plan.M; g.N = plan.N; g.K = plan.K;
    g.l0 = l0; g.l1 = l1;
    g.n_moduli = plan.n_moduli;
    g.tri_left = ip.tri_left;
    g.tri_lower = ip.tri_lower;
    g.tri_none = ip.tri_none;
    g.ctl = ip.ctl;
    g.status = h->dctl + 1;
    g.num_sms = h->num_sms;
    g.raster_group = h->oz_raster;
    const char *why = nullptr;
    rc = launch_oz_gemm(g, h->stream, &why);
    if (rc != UVATRMM_OK) return fail(rc, why ? why : "residue GEMM launch failed");
    mark(2);
  }
  const int rc = oz_reassemble(plan, ip.ctl, ip.res, ip.e_row, ip.e_col, ip.alpha, ip.beta, ip.C, ip.ldc,
                               ip.stage, ip.lds, h->stream);
  return rc == UVATRMM_OK ? UVATRMM_OK : fail(rc, "CRT reassembly failed to launch");
}

}  // namespace

int ozaki_device(uvatrmm_handle_t h, int layout, int side, int uplo, int transa, int diag, int64_t m, int64_t n,
                 double alpha, const double *dA, int64_t lda, double *dB, int64_t ldb, int moduli, double *relerr,
                 int *bits_out) {
  if (int bad = check_args(layout, side, uplo, transa, diag, m, n, lda, ldb))
    return fail(UVATRMM_EINVAL, "parameter " + std::to_string(bad) + " had an illegal value");
  if (moduli != 0 && (moduli < 2 || moduli > kMaxModuli))
    return fail(UVATRMM_EINVAL, "moduli must be 0 (automatic) or 2.." + std::to_string(kMaxModuli));
  const Trmm t = normalise(layout, side, uplo, transa, diag, m, n, alpha);
  if (relerr) *relerr = 0.0;
  if (t.m == 0 || t.n == 0) return ok();
  if (alpha == 0.0) {
    cudaError_t e = cudaMemset2DAsync(dB, ldb * 8, 0, t.m * 8, t.n, h->stream);
    return e == cudaSuccess ? ok() : cuda_fail(e, "zero fill");
  }
  OzOperand L, R;
  operands(t, dA, lda, dB, ldb, L, R);
  OzPlan plan;
  plan.M = t.m;
  plan.N = t.n;
  plan.K = t.side == CblasLeft ? t.m : t.n;
  plan.n_moduli = moduli ? moduli : ozaki_auto_moduli(plan.K);
  plan.bits = ozaki_bits(plan.n_moduli, plan.K);
  plan.Mp = oz_pad_rows(plan.M);
  plan.Np = oz_pad_cols(plan.N);
  plan.Kp = round_up(plan.K, 64);
  if (bits_out) *bits_out = plan.bits;

  // Residue planes per modulus: (Mp + Np) x Kp bf16; passes of G moduli.
  const int64_t per_mod = (plan.Mp + plan.Np) * plan.Kp * 2;
  const int G = (int)std::max<int64_t>(1, std::min<int64_t>(plan.n_moduli, (h->ozaki_scratch_mb << 20) / per_mod));
  void *e = workspace(h, 4, oz_scale_bytes(plan.Mp, plan.Np, plan.K));
  uint16_t *res =
      static_cast<uint16_t *>(workspace(h, 6, (size_t)oz_res_planes(plan.n_moduli) * plan.Mp * plan.Np * sizeof(uint16_t)));
  uint16_t *planes = static_cast<uint16_t *>(workspace(h, 5, (size_t)G * per_mod));
  if (!e || !res || !planes) return uvatrmm_last_status();
  const OzScaleBuf sb = oz_scale_buf(e, plan.Mp, plan.Np, plan.K);

  // Error estimate: keep the sampled inputs (columns of B for side Left,
  // rows for side Right) before B is overwritten.
  const int S = relerr ? (int)std::min<int64_t>(kErrSamples, t.side == CblasLeft ? t.n : t.m) : 0;
  double *samp = nullptr;
  const int64_t len = t.side == CblasLeft ? t.m : t.n;  // entries per sampled column / row
  if (S) {
    samp = static_cast<double *>(workspace(h, 7, (size_t)3 * S * round_up(len, 16) * 8));
    if (!samp) return uvatrmm_last_status();
    const int64_t cnt = t.side == CblasLeft ? t.n : t.m;
    for (int s = 0; s < S; ++s) {
      const int64_t idx = S > 1 ? (cnt - 1) * s / (S - 1) : 0;
      cudaError_t ce = t.side == CblasLeft
                           ? cudaMemcpyAsync(samp + s * round_up(len, 16), dB + idx * ldb, len * 8,
                                             cudaMemcpyDeviceToDevice, h->stream)
                           : cudaMemcpy2DAsync(samp + s, S * 8, dB + idx, ldb * 8, 8, len,
                                               cudaMemcpyDeviceToDevice, h->stream);
      if (ce != cudaSuccess) return cuda_fail(ce, "error-estimate sample");
    }
  }

  h->n_sev = 0;
  auto mark = [&](int kind) {
    if (h->stage_timing && h->n_sev < uvatrmm_handle_st::kStageEvents) {
      h->sev_kind[h->n_sev] = kind;
      cudaEventRecord(h->sev[h->n_sev++], h->stream);
    }
  };
  mark(-1);
  // (Stage times are taken between the two kernels.)
  bool sliced = false;
  int rc = UVATRMM_OK;
  if (G == plan.n_moduli && !h->stage_timing)
    rc = oz_prep_once(L, R, sb, plan, nullptr, nullptr, nullptr, planes, planes + (int64_t)G * plan.Mp * plan.Kp, h->dctl + 1,
                      h->num_sms, 0, h->stream, &sliced);
  if (rc == UVATRMM_OK && !sliced) rc = oz_scales(L, R, sb, scale_counters(h), nullptr, nullptr, h->stream);
  if (rc != UVATRMM_OK) return fail(rc, "Ozaki scaling failed to launch");
  mark(0);
  IntProduct ip;
  ip.L = L;
  ip.R = R;
  ip.plan = plan;
  ip.tri_left = t.side == CblasLeft;
  ip.tri_lower = (t.uplo == CblasLower) != (t.trans != 0);
  ip.alpha = t.alpha;
  ip.C = dB;
  ip.ldc = ldb;
  ip.e_row = sb.e_row;
  ip.e_col = sb.e_col;
  ip.G = G;
  ip.planes = planes;
  ip.res = res;
  ip.sliced = sliced;
  if ((rc = int_product(h, ip, mark)) != UVATRMM_OK) return rc;
  mark(3);

  if (S) {
    // Plain FP64 reference for the sampled columns / rows, then the error.
    const int64_t lp = round_up(len, 16);
    double *ref = samp + (int64_t)S * lp, *got = samp + 2 * (int64_t)S * lp;
    const int64_t cnt = t.side == CblasLeft ? t.n : t.m;
    for (int s = 0; s < S; ++s) {
      const int64_t idx = S > 1 ? (cnt - 1) * s / (S - 1) : 0;
      cudaError_t ce = t.side == CblasLeft
                           ? cudaMemcpyAsync(got + s * lp, dB + idx * ldb, len * 8, cudaMemcpyDeviceToDevice,
                                             h->stream)
                           : cudaMemcpy2DAsync(got + s, S * 8, dB + idx, ldb * 8, 8, len, cudaMemcpyDeviceToDevice,
                                               h->stream);
      if (ce != cudaSuccess) return cuda_fail(ce, "error-estimate sample");
    }
    if (t.side == CblasLeft)
      rc = device_trmm(h, CblasColMajor, CblasLeft, t.uplo, t.trans ? CblasTrans : CblasNoTrans,
                       t.unit ? CblasUnit : CblasNonUnit, t.m, S, t.alpha, dA, lda, samp, lp, ref, lp, false,
                       h->schedule, h->shape, 0.0, true);
    else
      rc = device_trmm(h, CblasColMajor, CblasRight, t.uplo, t.trans ? CblasTrans : CblasNoTrans,
                       t.unit ? CblasUnit : CblasNonUnit, S, t.n, t.alpha, dA, lda, samp, S, ref, S, false,
                       h->schedule, h->shape, 0.0, true);
    if (rc != UVATRMM_OK) return rc;
    rc = t.side == CblasLeft ? rel_frobenius(h, len, S, got, lp, ref, lp, relerr)
                             : rel_frobenius(h, S, len, got, S, ref, S, relerr);
    if (rc != UVATRMM_OK) return rc;
    rc = collect_status(h);
    if (rc != UVATRMM_OK) return rc;
  }
  return ok();
}

// The lossless route (see OzCtl).  Scratch: at most kExactBytes and the
// handle's UVATRMM_OPT_OZAKI_SCRATCH_MB, split between the product residues of
// a panel of the minor dimension (the one without the triangle) and the
// residue planes of a pass over the moduli.  Down to the option's least value
// the panels and passes are faster than the tile kernel wherever they fit (us,
// 64 MiB / tile kernel: 1000 x 1000 146 / 2010, 2000 x 2000 1610 / 7050, 2700 x
// 2700 8227 / 16952, 300 x 50000 2054 / 4105).
namespace {
constexpr int64_t kExactBytes = 16ll << 30;
}

namespace {
bool thin_gemm(int64_t M, int64_t K, bool tri) { return !tri && M < 16 && K >= 64; }
}  // namespace

double tile_us(int64_t M, int64_t N, int64_t K, bool tri) {
  // An SM takes about 1 us per k of a 64 x 64 tile (2 FP64 FMAs per clock;
  // edge tiles by their 16-wide blocks), a little more for the one tile the
  // others wait for; diagonal blocks of 64 cost three quarters.
  const double k = (double)K;
  auto part = [](int64_t x) { return std::min<int64_t>(64, (x + 15) / 16 * 16) / 64.0; };
  const double per_k = part(M) * part(N);
  const double chain = 1.12 * k * (tri && K <= 64 ? 0.75 : 1.0);
  const double tiles = std::ceil(M / 64.0) * std::ceil(N / 64.0);
  const double work = tiles * (tri ? std::min(k, k / 2 + 15) : k) / 152;
  // GEMMs of a few rows: rounds of two tiles per SM, whose rows go by twos (M x
  // 50000 x 600, us: M = 2 380, 8 490, 12 730, 16 940, 64 3710), a last one of one
  // per SM in half the time.
  if (thin_gemm(M, K, tri)) {
    const double full = std::floor(tiles / 304), last = tiles - 304 * full;
    const double two = 0.034 * (double)((M + 1) / 2 * 2);
    const double end = last > 152 ? std::max(0.21, two) : last > 0 ? std::max(0.21, two / 2) : 0.0;
    return 9 + k * part(N) * (full * std::max(0.21, two) + end);
  }
  return 9 + per_k * std::max(chain, 1.05 * work + 0.25 * k);
}

double exact_us(int64_t M, int64_t N, int64_t K, bool tri) {
  // At 15 moduli: launches and latencies (4 us less where scales and residues
  // are one launch, which is left out: entries of wide spans need more moduli,
  // and would lose at 240 x 240 what others gain, 40 against 29 us); scaling and slicing per operand
  // entry (half of the K x K triangular operand); rounds of 256 x 256 residue
  // tiles over the 76 SM pairs; product residues and (of few rows: little) reassembly.
  const double m = (double)M, n = (double)N, k = (double)K;
  const double entries = k * (m + n) - (tri ? 0.5 * k * k : 0.0);
  const double pm = std::ceil(m / 256), pn = std::ceil(n / 256);
  const double rounds = std::ceil(pm * pn * 15 / 76) * (1.2 + 0.0062 * k * (tri ? 0.6 : 1.0));
  return 30 + 1.05e-5 * entries + rounds + (thin_gemm(M, K, tri) ? 0.6e-5 : 1.2e-5) * pm * 256 * pn * 256;
}

// The fastest by the three estimates, which were fitted to (us, tile kernel /
// small kernel / lossless route; triangle of order K, V vectors):
//   K x V   64 x 64     51 / 9.3 / 27     64 x 100000  481 / 544 / 499
//           128 x 4000  134 / 84 / 53     256 x 256    287 / 32 / 34
//           384 x 384   439 / 75 / 38     1000 x 1     280 / 13 / 40
//           1000 x 16   280 / 30 / 41     1000 x 50    1116 / 84 / 42
//           1000 x 1000 2018 / 951 / 84   4000 x 1     1122 / 34 / 211
// `in_place`: the tile kernel's copy of B counts as well (the small kernel
// and the route need none); it does not move calls to or from the route.
// `staged`: bytes of operands that only the tile kernel copies first.
Route pick_route(int64_t M, int64_t N, int64_t K, bool tri, bool tri_left, bool in_place, int64_t staged) {
  const bool by_cols = !tri || tri_left;
  const double small = small_us(by_cols ? M : N, by_cols ? N : M, K, tri);
  const double tile = tile_us(M, N, K, tri) + staged / 0.85e6, exact = exact_us(M, N, K, tri);
  if (exact < std::min(small, tile)) return Route::kExact;
  const double copy = in_place ? 6 + 16.0 * M * N / 4e6 : 0.0;
  return small <= tile + copy ? Route::kSmall : Route::kTile;
}

bool small_behind_exact(int64_t M, int64_t N, int64_t K, bool tri_left) {
  // (Under about 3 ms the estimates lean to the tile kernel: of 106 such sizes
  // timed with a declined operand the faster kernel was missed by 2.2 % on
  // average and 40 % at most with a plain comparison, by 0.4 and 22 with this one,
  // 120 x 14785 374 -> 267 us, 102 x 14337 270 -> 221; larger ones lose by it,
  // 1289 x 7348 11300 -> 12250.)
  const double tile = tile_us(M, N, K, true);
  return small_us(K, tri_left ? N : M, K, true) < (tile < 3000 ? 1.2 : 1.0) * tile;
}

namespace {

// The route's panels and passes for an M x N x K product, and their scratch.
struct ExactPlan {
  OzPlan plan;
  int64_t w, panels, G, per_mod;  // panel width of the minor dimension, moduli per pass, bytes of planes per modulus
  size_t need[3];                 // workspace slots 4 to 6: scales, residue planes, product residues
};

// False where no panel and pass fits the limit.  by_cols: the minor dimension
// is the columns of Rgt, else the rows of Lft.
bool exact_plan(uvatrmm_handle_t h, int64_t M, int64_t N, int64_t K, bool by_cols, ExactPlan *p) {
  OzPlan &plan = p->plan;
  plan.M = M;
  plan.N = N;
  plan.K = K;
  plan.n_moduli = kCrtModuli;
  plan.bits = 0;
  plan.Mp = oz_pad_rows(plan.M);
  plan.Np = oz_pad_cols(plan.N);
  plan.Kp = round_up(plan.K, 64);
  const int64_t major = by_cols ? plan.Mp : plan.Np, minor = by_cols ? plan.Np : plan.Mp;
  const int64_t limit = std::min(kExactBytes, h->ozaki_scratch_mb << 20);
  const int64_t per_res = 2 * oz_res_planes(kCrtModuli) * major * kOzBlock;  // product residues of 256 minor lines
  const int64_t w = std::min(minor, std::max<int64_t>(1, limit / 2 / per_res) * kOzBlock);
  p->panels = (minor + w - 1) / w;
  p->w = round_up((minor + p->panels - 1) / p->panels, kOzBlock);
  const int64_t res_bytes = per_res * (p->w / kOzBlock);
  p->per_mod = (major + p->w) * plan.Kp * 2;
  p->G = std::min<int64_t>(kCrtModuli, (limit - res_bytes) / p->per_mod);
  if (p->G < 1) return false;
  p->need[0] = oz_scale_bytes(plan.Mp, plan.Np, plan.K);
  p->need[1] = (size_t)(p->G * p->per_mod);
  p->need[2] = (size_t)res_bytes;
  return true;
}

// Takes the scratch.  What is not there yet is taken only outside a stream
// capture, and only where it leaves as much memory free as it takes.
bool exact_scratch(uvatrmm_handle_t h, const ExactPlan &p) {
  size_t grow = 0;
  for (int k = 0; k < 3; ++k)
    if (h->ws_cap[4 + k] < p.need[k]) grow += p.need[k];
  if (grow) {
    if (stream_captures(h)) return false;
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess || free_b / 2 < grow) {
      cudaGetLastError();
      return false;
    }
  }
  for (int k = 0; k < 3; ++k)
    if (!workspace(h, 4 + k, p.need[k])) {
      ok();
      return false;
    }
  return true;
}

}  // namespace

void exact_reserve(uvatrmm_handle_t h, int64_t M, int64_t N, int64_t K, bool by_cols) {
  ExactPlan p;
  if (exact_plan(h, M, N, K, by_cols, &p)) exact_scratch(h, p);
}

int exact_product(uvatrmm_handle_t h, const OzOperand &L, const OzOperand &R, bool tri_none, bool tri_left,
                  bool tri_lower, double alpha, double beta, double *C, int64_t ldc, const OzCtl **gate, double *stage,
                  int64_t lds) {
  *gate = nullptr;
  const bool by_cols = tri_left;  // the minor dimension: columns of Rgt, else rows of Lft
  ExactPlan p;
  if (!exact_plan(h, L.P, R.P, L.K, by_cols, &p) || !exact_scratch(h, p)) return UVATRMM_OK;
  const OzPlan &plan = p.plan;
  const int64_t w = p.w, G = p.G;
  void *e = h->ws[4];
  uint16_t *planes = static_cast<uint16_t *>(h->ws[5]), *res = static_cast<uint16_t *>(h->ws[6]);
  OzCtl *ctl = handle_ctl(h);
  const OzScaleBuf sb = oz_scale_buf(e, plan.Mp, plan.Np, plan.K);
  bool sliced = false;
  int rc = UVATRMM_OK;
  if (p.panels == 1 && G == plan.n_moduli)
    rc = oz_prep_once(L, R, sb, plan, ctl, h->dctl, fused_slots(h), planes, planes + G * plan.Mp * plan.Kp,
                      h->dctl + 1, h->num_sms, h->exchange_expiry_polls, h->stream, &sliced);
  if (rc == UVATRMM_OK && !sliced) rc = oz_scales(L, R, sb, scale_counters(h), ctl, h->dctl, h->stream);
  if (rc != UVATRMM_OK) return fail(rc, "scaling failed to launch");
  for (int64_t c0 = 0; c0 < (by_cols ? plan.N : plan.M); c0 += w) {
    IntProduct ip;
    ip.L = L;
    ip.R = R;
    ip.plan = plan;
    ip.tri_left = tri_left;
    ip.tri_lower = tri_lower;
    ip.tri_none = tri_none;
    ip.alpha = alpha;
    ip.beta = beta;
    ip.ldc = ldc;
    ip.lds = lds;
    ip.ctl = ctl;
    ip.G = (int)G;
    ip.planes = planes;
    ip.res = res;
    ip.e_row = sb.e_row;
    ip.e_col = sb.e_col;
    ip.C = C;
    OzOperand &op = by_cols ? ip.R : ip.L;
    op.X += op.kcontig ? c0 * op.ld : c0;
    op.P = std::min(w, op.P - c0);
    if (by_cols) {
      ip.plan.N = op.P;
      ip.plan.Np = oz_pad_cols(op.P);
      ip.e_col += c0;
      ip.C += c0 * ldc;
      if (stage) ip.stage = stage + c0 * lds;
    } else {
      ip.plan.M = op.P;
      ip.plan.Mp = oz_pad_rows(op.P);
      ip.e_row += c0;
      ip.C += c0;
      if (stage) ip.stage = stage + c0;
    }
    ip.sliced = sliced;
    if ((rc = int_product(h, ip, [](int) {})) != UVATRMM_OK) return rc;
  }
  *gate = ctl;
  return UVATRMM_OK;
}

void ozaki_operands(const Trmm &t, const double *dA, int64_t lda, const double *dB, int64_t ldb, OzOperand &L,
                    OzOperand &R) {
  operands(t, dA, lda, dB, ldb, L, R);
}

}  // namespace uvt

using namespace uvt;

extern "C" {

UVATRMM_API int uvatrmm_stage_times(uvatrmm_handle_t h, double *ms4) {
  if (!(h = resolve(h))) return uvatrmm_last_status();
  if (!ms4) return fail(UVATRMM_EINVAL, "ms4 is NULL");
  std::lock_guard<std::mutex> g(h->mu);
  for (int k = 0; k < 4; ++k) ms4[k] = 0.0;
  if (h->n_sev < 2) return fail(UVATRMM_EINVAL, "no timed Ozaki call (enable UVATRMM_OPT_STAGE_TIMING)");
  cudaError_t e = cudaEventSynchronize(h->sev[h->n_sev - 1]);
  if (e != cudaSuccess) return cuda_fail(e, "stage timing");
  for (int i = 1; i < h->n_sev; ++i) {
    float ms = 0.f;
    cudaEventElapsedTime(&ms, h->sev[i - 1], h->sev[i]);
    if (h->sev_kind[i] >= 0 && h->sev_kind[i] < 4) ms4[h->sev_kind[i]] += ms;
  }
  return ok();
}

UVATRMM_API int uvatrmm_ozaki_plan(int64_t k, int moduli, int *moduli_out, int *bits_out) {
  if (k < 0 || (moduli != 0 && (moduli < 2 || moduli > kMaxModuli))) return fail(UVATRMM_EINVAL, "invalid arguments");
  const int n = moduli ? moduli : ozaki_auto_moduli(k);
  if (moduli_out) *moduli_out = n;
  if (bits_out) *bits_out = ozaki_bits(n, k);
  return ok();
}

UVATRMM_API int uvatrmm_ozaki_dtrmm_device(uvatrmm_handle_t h, int layout, int side, int uplo, int transa, int diag,
                                          int64_t m, int64_t n, double alpha, const double *dA, int64_t lda,
                                          double *dB, int64_t ldb, int moduli, double *relerr_out, int *bits_out) {
  if (!(h = resolve(h))) return uvatrmm_last_status();
  std::lock_guard<std::mutex> g(h->mu);
  if (!relerr_out || !h->oz_err_host)
    return ozaki_device(h, layout, side, uplo, transa, diag, m, n, alpha, dA, lda, dB, ldb, moduli, relerr_out,
                        bits_out);
  // Error against the host FP64 reference: the sampled inputs and op(A) are
  // copied to the host around the call.
  if (int bad = check_args(layout, side, uplo, transa, diag, m, n, lda, ldb))
    return fail(UVATRMM_EINVAL, "parameter " + std::to_string(bad) + " had an illegal value");
  const Trmm t = normalise(layout, side, uplo, transa, diag, m, n, alpha);
  // Nothing to compare (empty, alpha = 0) or an invalid slice count: the
  // plain path reports it before anything is copied.
  if (t.m == 0 || t.n == 0 || alpha == 0.0 || (moduli != 0 && (moduli < 2 || moduli > kMaxModuli)))
    return ozaki_device(h, layout, side, uplo, transa, diag, m, n, alpha, dA, lda, dB, ldb, moduli, relerr_out,
                        bits_out);
  *relerr_out = 0.0;
  const bool left = t.side == CblasLeft;
  const int64_t len = left ? t.m : t.n, cnt = left ? t.n : t.m, ka = len;
  const int S = (int)std::min<int64_t>(kErrSamples, cnt);
  std::vector<double> b((size_t)S * len), got((size_t)S * len);
  std::unique_ptr<double[]> A;  // host copy of A (not zero-filled: every entry read is copied in)
  if (S && alpha != 0.0) {
    if (int rc = gather_samples(h, t, S, dB, ldb, true, b.data())) return rc;
    A.reset(new (std::nothrow) double[(size_t)ka * ka]);
    if (!A) return fail(UVATRMM_ENOMEM, "host memory for the error report's copy of A");
    cudaError_t e = cudaMemcpy2DAsync(A.get(), ka * 8, dA, lda * 8, ka * 8, ka, cudaMemcpyDeviceToHost, h->stream);
    if (e != cudaSuccess) return cuda_fail(e, "error-report copy of A");
  }
  int rc = ozaki_device(h, layout, side, uplo, transa, diag, m, n, alpha, dA, lda, dB, ldb, moduli, nullptr,
                        bits_out);
  if (rc != UVATRMM_OK || !S || alpha == 0.0) return rc;
  if ((rc = collect_status(h)) != UVATRMM_OK) return rc;
  if ((rc = gather_samples(h, t, S, dB, ldb, true, got.data())) != UVATRMM_OK) return rc;
  *relerr_out = host_ref_relerr(t, A.get(), ka, S, b.data(), got.data());
  return ok();
}

UVATRMM_API int uvatrmm_ozaki_dtrmm(uvatrmm_handle_t h, int layout, int side, int uplo, int transa, int diag,
                                   int64_t m, int64_t n, double alpha, const double *A, int64_t lda, double *B,
                                   int64_t ldb, int moduli, double *relerr_out, int *bits_out) {
  if (!(h = resolve(h))) return uvatrmm_last_status();
  std::lock_guard<std::mutex> g(h->mu);
  if (int bad = check_args(layout, side, uplo, transa, diag, m, n, lda, ldb))
    return fail(UVATRMM_EINVAL, "parameter " + std::to_string(bad) + " had an illegal value");
  const Trmm t = normalise(layout, side, uplo, transa, diag, m, n, alpha);
  if (t.m == 0 || t.n == 0) return ok();
  const int64_t ka = t.side == CblasLeft ? t.m : t.n;
  const int64_t la = round_up(ka, 16), lb = round_up(t.m, 16);
  double *dA = static_cast<double *>(workspace(h, 0, (size_t)la * ka * 8));
  double *dB = static_cast<double *>(workspace(h, 2, (size_t)lb * t.n * 8));
  if (!dA || !dB) return uvatrmm_last_status();
  // (B first: its pages, which the caller has just written, are touched faster,
  // and A's are touched while it moves.)
  cudaError_t e = host_copy2d(h, dB, lb * 8, B, ldb * 8, t.m * 8, t.n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = copy_triangle_h2d(h, dA, la, A, lda, ka, t.uplo == CblasLower);
  if (e != cudaSuccess) return drained(h, cuda_fail(e, "host to device copy"));
  // Error report: the sampled inputs are kept before B is overwritten; the
  // reference is computed on the host from the caller's own A and B.
  const bool left = t.side == CblasLeft;
  const int64_t len = left ? t.m : t.n, cnt = left ? t.n : t.m;
  const int S = relerr_out && alpha != 0.0 ? (int)std::min<int64_t>(kErrSamples, cnt) : 0;
  if (relerr_out) *relerr_out = 0.0;
  std::vector<double> bs((size_t)S * len), got((size_t)S * len);
  if (S) gather_samples(h, t, S, B, ldb, false, bs.data());
  int rc = ozaki_device(h, CblasColMajor, t.side, t.uplo, t.trans ? CblasTrans : CblasNoTrans,
                        t.unit ? CblasUnit : CblasNonUnit, t.m, t.n, t.alpha, dA, la, dB, lb, moduli, nullptr,
                        bits_out);
  if (rc != UVATRMM_OK) return drained(h, rc);
  e = host_copy2d(h, B, ldb * 8, dB, lb * 8, t.m * 8, t.n, cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return drained(h, cuda_fail(e, "device to host copy"));
  rc = collect_status(h);
  if (rc != UVATRMM_OK) return rc;
  if (S) {
    gather_samples(h, t, S, B, ldb, false, got.data());
    *relerr_out = host_ref_relerr(t, A, lda, S, bs.data(), got.data());
  }
  return ok();
}

}  // extern "C"
