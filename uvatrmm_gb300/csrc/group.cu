// Grouped batches: many TRMMs planned once and captured into one CUDA graph.
//
// Plan (uvatrmm_group_create):
//   * FP64-tier problems: each is staged like the in-place device call (B, and
//     A when it is not 16-byte aligned with an even lda, into the group's
//     arena), gets its tile edge from the autotuner, and becomes one
//     Fp64GroupProb; problems of the same tile edge share one persistent
//     grouped launch (trmm_fp64_group_kernel), longest problems first.
//   * FP64-tier problems large enough for the lossless integer route also get
//     its scales, planes and decision word and join the waves below; the
//     copies and tiles of those it computes are passed over at run time.
//   * Ozaki-tier problems: each gets its scales, residue planes and residue
//     output in the arena; they are packed into waves that fit the Ozaki
//     scratch budget; a wave is the slicing kernels of its problems, ONE
//     grouped residue-GEMM launch over all their tiles, then the CRT
//     reassembly of each problem.
//   * Small FP64 problems share one launch of the small kernel.
//   * Everything is captured on the handle's stream into a CUDA graph; a run
//     replays it.  Descriptors are uploaded before the capture.
#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "api_internal.h"
#include "common.cuh"
#include "ozaki.cuh"
#include "trmm_fp64.cuh"

struct uvatrmm_group_st {
  uvatrmm_handle_t h = nullptr;
  void *arena = nullptr;
  size_t arena_bytes = 0;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  double flops = 0.0;
  int launches = 0, waves = 0;
  int64_t fp64_tiles = 0, oz_tiles = 0;
};

namespace uvt {

namespace {

struct ArenaPlan {
  size_t used = 0;
  size_t take(size_t bytes, size_t align = 256) {
    used = (used + align - 1) / align * align;
    const size_t off = used;
    used += bytes;
    return off;
  }
};

struct F64Item {
  Trmm t;
  const double *A;
  int64_t lda;
  double *B;
  int64_t ldb;
  int tile;
  bool stage_a;
  int64_t la, lb;
  size_t offA = 0, offB = 0, offPart = 0;
  int64_t work = 0;  // slabs of the largest tile, for the longest-first order
  int exact = -1;    // its item on the lossless route
  bool small = false;  // on the small kernel
};

struct OzItem {
  Trmm t;
  const double *A;
  int64_t lda;
  double *B;
  int64_t ldb;
  OzPlan plan;
  int raster;
  size_t bytes = 0;           // scales + planes + residues
  size_t offE = 0, offP = 0, offR = 0;  // inside the wave region
  int wave = 0;
  int ctl = -1;  // lossless route: index of its decision word
};

// Device memory a group's waves take at most once FP64 problems are in them.
constexpr size_t kExactWaveBytes = size_t(16) << 30;
size_t exact_wave_bytes(uvatrmm_handle_t h) { return std::min((size_t)h->ozaki_scratch_mb << 20, kExactWaveBytes); }

// One staging copy of the FP64 problems (see stage_wave_kernel).
struct CopyJob {
  const double *src;
  double *dst;
  int64_t lds, ldd, rows, total;  // total = rows * columns
  const OzCtl *gate;
  int64_t block_begin;
};
constexpr int kCopyPerThread = 16, kCopyPerBlock = 256 * kCopyPerThread;

// All staging copies of a group in one launch; those of problems that the
// lossless route computed are passed over.
__global__ void __launch_bounds__(256) stage_wave_kernel(const CopyJob *jobs, int n) {
  const int64_t b = blockIdx.x;
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (jobs[mid].block_begin <= b) lo = mid;
    else hi = mid - 1;
  }
  const CopyJob J = jobs[lo];
  if (J.gate && J.gate->go) return;
  // Column and row of the block's first element, then 32-bit steps from there.
  const int64_t first = (b - J.block_begin) * kCopyPerBlock;
  const int64_t c0 = first / J.rows;
  const uint64_t r0 = (uint64_t)(first - c0 * J.rows);
  const int left = (int)min((int64_t)kCopyPerBlock, J.total - first);
  double v[kCopyPerThread];
#pragma unroll
  for (int q = 0; q < kCopyPerThread; ++q) {
    const int i = threadIdx.x + q * 256;
    const uint32_t r = (uint32_t)(r0 + i), dc = r / (uint32_t)J.rows;
    if (i < left) v[q] = J.src[(c0 + dc) * J.lds + (r - dc * (uint32_t)J.rows)];
  }
#pragma unroll
  for (int q = 0; q < kCopyPerThread; ++q) {
    const int i = threadIdx.x + q * 256;
    const uint32_t r = (uint32_t)(r0 + i), dc = r / (uint32_t)J.rows;
    if (i < left) J.dst[(c0 + dc) * J.ldd + (r - dc * (uint32_t)J.rows)] = v[q];
  }
}

bool tma_aligned(const void *p, int64_t ld) { return (reinterpret_cast<uintptr_t>(p) % 16 == 0) && (ld % 2 == 0); }

Fp64Launch fp64_launch(const Trmm &t, const double *A, int64_t lda, const double *B, int64_t ldb, double *C,
                       int64_t ldc, int tile) {
  Fp64Launch L;
  const int64_t ka = t.side == CblasLeft ? t.m : t.n;
  L.M = t.m;
  L.N = t.n;
  L.K = ka;
  L.alpha = t.alpha;
  L.C = C;
  L.ldc = ldc;
  L.unit = t.unit;
  L.tri_lower = (t.uplo == CblasLower) != (t.trans != 0);
  if (t.side == CblasLeft) {
    L.tri_left = true;
    L.xl = MatRef{A, ka, ka, lda};
    L.lft_kmajor = t.trans != 0;
    L.xr = MatRef{B, t.m, t.n, ldb};
    L.rgt_kmajor = true;
  } else {
    L.tri_left = false;
    L.xl = MatRef{B, t.m, t.n, ldb};
    L.lft_kmajor = false;
    L.xr = MatRef{A, ka, ka, lda};
    L.rgt_kmajor = t.trans == 0;
  }
  L.engine = UVATRMM_ENGINE_DFMA;
  L.schedule = UVATRMM_SCHED_DYNAMIC;
  L.shape = UVATRMM_SHAPE_TRAPEZOID;
  L.tile = tile;
  return L;
}

void destroy_group(uvatrmm_group_t g) {
  if (!g) return;
  if (g->exec) cudaGraphExecDestroy(g->exec);
  if (g->graph) cudaGraphDestroy(g->graph);
  if (g->arena) cudaFree(g->arena);
  delete g;
}

// Scales, planes and residues of one integer product inside a wave.
void size_item(OzItem &it) {
  OzPlan &pl = it.plan;
  pl.M = it.t.m;
  pl.N = it.t.n;
  pl.K = it.t.side == CblasLeft ? it.t.m : it.t.n;
  pl.Mp = oz_pad_rows(pl.M);
  pl.Np = oz_pad_cols(pl.N);
  pl.Kp = round_up(pl.K, 64);
  ArenaPlan a;
  it.offE = a.take(oz_scale_bytes(pl.Mp, pl.Np, pl.K));
  it.offP = a.take((size_t)pl.n_moduli * (pl.Mp + pl.Np) * pl.Kp * 2);
  it.offR = a.take((size_t)oz_res_planes(pl.n_moduli) * pl.Mp * pl.Np * sizeof(uint16_t));
  it.bytes = round_up((int64_t)a.used, 256);
}

int build(uvatrmm_group_t g, const uvatrmm_trmm_problem *probs, int count, bool exact) {
  uvatrmm_handle_t h = g->h;
  int n_exact = 0;
  std::vector<F64Item> f64;
  std::vector<OzItem> oz;
  std::vector<std::pair<double *, Trmm>> zeros;
  std::vector<int64_t> zero_ld;
  for (int i = 0; i < count; ++i) {
    const uvatrmm_trmm_problem &p = probs[i];
    if (int bad = check_args(p.layout, p.side, p.uplo, p.transa, p.diag, p.m, p.n, p.lda, p.ldb))
      return fail(UVATRMM_EINVAL, "problem " + std::to_string(i) + ": parameter " + std::to_string(bad) +
                                      " had an illegal value");
    if (p.tier != UVATRMM_TIER_FP64 && p.tier != UVATRMM_TIER_OZAKI)
      return fail(UVATRMM_EINVAL, "problem " + std::to_string(i) + ": unknown tier");
    if (p.tier == UVATRMM_TIER_OZAKI && p.moduli != 0 && (p.moduli < 2 || p.moduli > kMaxModuli))
      return fail(UVATRMM_EINVAL, "problem " + std::to_string(i) + ": moduli out of range");
    if (!p.B || (!p.A && p.m && p.n)) return fail(UVATRMM_EINVAL, "problem " + std::to_string(i) + ": NULL buffer");
    const Trmm t = normalise(p.layout, p.side, p.uplo, p.transa, p.diag, p.m, p.n, p.alpha);
    if (t.m == 0 || t.n == 0) continue;
    g->flops += t.side == CblasLeft ? (double)t.m * t.m * t.n : (double)t.n * t.n * t.m;
    if (t.alpha == 0.0) {
      zeros.push_back({p.B, t});
      zero_ld.push_back(p.ldb);
      continue;
    }
    if (p.tier == UVATRMM_TIER_FP64) {
      F64Item it;
      it.t = t;
      it.A = p.A;
      it.lda = p.lda;
      it.B = p.B;
      it.ldb = p.ldb;
      if (int rc = tune_choice(h, UVATRMM_TIER_FP64, t.side, t.m, t.n, &it.tile)) return rc;
      const int64_t ka = t.side == CblasLeft ? t.m : t.n;
      it.stage_a = !tma_aligned(p.A, p.lda);
      it.la = round_up(ka, 16);
      it.lb = round_up(t.m, 16);
      it.work = (ka + it.tile - 1) / it.tile;
      const Route route = route_free(h, h->schedule, h->shape) ? pick_route(t.m, t.n, ka, true, t.side == CblasLeft)
                                                               : Route::kTile;
      it.small = route == Route::kSmall;
      if (exact && route == Route::kExact) {
        OzItem x;
        x.t = t;
        x.A = p.A;
        x.lda = p.lda;
        x.B = p.B;
        x.ldb = p.ldb;
        x.plan.n_moduli = kCrtModuli;
        x.plan.bits = 0;
        x.raster = 0;
        size_item(x);
        if (x.bytes <= exact_wave_bytes(h)) {
          it.exact = x.ctl = n_exact++;
          it.small = small_behind_exact(t.m, t.n, ka, t.side == CblasLeft);
          oz.push_back(x);
        }
      }
      f64.push_back(it);
    } else {
      OzItem it;
      it.t = t;
      it.A = p.A;
      it.lda = p.lda;
      it.B = p.B;
      it.ldb = p.ldb;
      const int64_t ka = t.side == CblasLeft ? t.m : t.n;
      it.plan.n_moduli = p.moduli ? p.moduli : ozaki_auto_moduli(ka);
      it.plan.bits = ozaki_bits(it.plan.n_moduli, ka);
      if (int rc = tune_choice(h, UVATRMM_TIER_OZAKI, t.side, t.m, t.n, &it.raster)) return rc;
      size_item(it);
      oz.push_back(it);
    }
  }

  // ---- arena layout: control words, FP64 descriptors + staging, Ozaki waves
  ArenaPlan A;
  const size_t off_ctl = A.take(256);
  const size_t off_gate = A.take((size_t)std::max(n_exact, 1) * sizeof(OzCtl));
  std::sort(f64.begin(), f64.end(), [](const F64Item &x, const F64Item &y) { return x.work > y.work; });
  std::vector<int> classes;  // tile edges in use
  for (auto &it : f64)
    if (!it.small && std::find(classes.begin(), classes.end(), it.tile) == classes.end()) classes.push_back(it.tile);
  std::vector<size_t> off_desc(classes.size());
  std::vector<std::vector<int>> members(classes.size());
  for (size_t c = 0; c < classes.size(); ++c) {
    for (int i = 0; i < (int)f64.size(); ++i)
      if (!f64[i].small && f64[i].tile == classes[c]) members[c].push_back(i);
    off_desc[c] = A.take(members[c].size() * sizeof(Fp64GroupProb), 64);
  }
  int n_copies = 0, n_small = 0;
  for (auto &it : f64) {
    if (it.small) it.stage_a = false;  // the small kernel reads A where it lies
    n_copies += it.stage_a ? 2 : 1;
    n_small += it.small;
  }
  const size_t off_small = A.take((size_t)std::max(n_small, 1) * sizeof(SmallJob));
  for (auto &it : f64)
    if (it.small) it.offPart = A.take(small_part_bytes(small_trmm(it.t, it.A, it.lda, it.B, it.ldb, it.B, it.ldb, 0.0)));
  const size_t off_copy = A.take((size_t)std::max(n_copies, 1) * sizeof(CopyJob));
  for (auto &it : f64) {
    it.offB = A.take((size_t)it.lb * it.t.n * 8);
    if (it.stage_a) it.offA = A.take((size_t)it.la * (it.t.side == CblasLeft ? it.t.m : it.t.n) * 8);
  }
  // Waves: greedy packing under the scratch budget, longest K first (the
  // residue GEMM's tiles go out in this order).
  std::stable_sort(oz.begin(), oz.end(), [](const OzItem &x, const OzItem &y) { return x.plan.K > y.plan.K; });
  const size_t budget = n_exact ? exact_wave_bytes(h) : (size_t)h->ozaki_scratch_mb << 20;
  std::vector<std::vector<int>> waves;
  size_t wave_bytes = 0, max_wave = 0;
  for (int i = 0; i < (int)oz.size(); ++i) {
    if (waves.empty() || (wave_bytes + oz[i].bytes > budget && !waves.back().empty())) {
      waves.emplace_back();
      wave_bytes = 0;
    }
    oz[i].wave = (int)waves.size() - 1;
    oz[i].offE += wave_bytes;
    oz[i].offP += wave_bytes;
    oz[i].offR += wave_bytes;
    wave_bytes += oz[i].bytes;
    waves.back().push_back(i);
    max_wave = std::max(max_wave, wave_bytes);
  }
  std::vector<size_t> off_wdesc(waves.size()), off_wtab(waves.size());
  for (size_t w = 0; w < waves.size(); ++w) {
    off_wdesc[w] = A.take(waves[w].size() * sizeof(OzGroupProb), 64);
    off_wtab[w] = A.take(oz_wave_table_bytes((int)waves[w].size()));
  }
  const size_t off_wave = A.take(max_wave);
  g->arena_bytes = A.used;
  if (n_exact) {  // the route's scratch leaves as much memory free as it takes
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess || free_b / 2 < g->arena_bytes) {
      cudaGetLastError();
      g->flops = 0.0;
      return build(g, probs, count, false);
    }
  }
  cudaError_t e = cudaMalloc(&g->arena, std::max<size_t>(g->arena_bytes, 256));
  if (e != cudaSuccess) {
    const std::string what = "group arena (" + std::to_string(g->arena_bytes) + " bytes)";
    return cuda_fail(e, what.c_str());
  }
  char *base = static_cast<char *>(g->arena);
  int *ctl = reinterpret_cast<int *>(base + off_ctl);
  cudaMemset(ctl, 0, 256);
  OzCtl *gates = reinterpret_cast<OzCtl *>(base + off_gate);
  if (n_exact) {
    const std::vector<OzCtl> init(n_exact, kOzCtlInit);
    e = cudaMemcpy(gates, init.data(), init.size() * sizeof(OzCtl), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return cuda_fail(e, "group decision words");
  }

  // ---- descriptors (host-built, uploaded before capture)
  const char *why = nullptr;
  std::vector<int> class_total(classes.size(), 0);
  for (size_t c = 0; c < classes.size(); ++c) {
    std::vector<Fp64GroupProb> hd(members[c].size());
    int begin = 0;
    for (size_t k = 0; k < members[c].size(); ++k) {
      const F64Item &it = f64[members[c][k]];
      const double *Ause = it.stage_a ? reinterpret_cast<double *>(base + it.offA) : it.A;
      const int64_t ldA = it.stage_a ? it.la : it.lda;
      const double *Bs = reinterpret_cast<double *>(base + it.offB);
      Fp64Launch L = fp64_launch(it.t, Ause, ldA, Bs, it.lb, it.B, it.ldb, it.tile);
      if (it.exact >= 0) L.gate = gates + it.exact;
      if (int rc = fp64_group_prob(L, it.tile, &hd[k], &why)) return fail(rc, why ? why : "FP64 descriptor");
      hd[k].tile_begin = begin;
      begin += hd[k].tile_count;
    }
    class_total[c] = begin;
    g->fp64_tiles += begin;
    e = cudaMemcpy(base + off_desc[c], hd.data(), hd.size() * sizeof(Fp64GroupProb), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return cuda_fail(e, "FP64 descriptors");
    if (int rc = fp64_group_prepare(classes[c], UVATRMM_ENGINE_DFMA)) return fail(rc, "FP64 kernel attributes");
  }
  // Staging copies: first those of the small kernel's own problems, which run
  // beside the waves, then the rest, behind them.
  std::vector<CopyJob> copies;
  int64_t copy_blocks[2] = {0, 0};
  size_t copies_first = 0;
  for (int part = 0; part < 2; ++part) {
    auto add_copy = [&](const double *src, int64_t lds, size_t off, int64_t ldd, int64_t rows, int64_t cols,
                        int gate) {
      CopyJob j{src, reinterpret_cast<double *>(base + off), lds, ldd, rows, rows * cols,
                gate >= 0 ? gates + gate : nullptr, copy_blocks[part]};
      copy_blocks[part] += (j.total + kCopyPerBlock - 1) / kCopyPerBlock;
      copies.push_back(j);
    };
    for (auto &it : f64) {
      if ((it.small && it.exact < 0) != (part == 0)) continue;
      const int64_t ka = it.t.side == CblasLeft ? it.t.m : it.t.n;
      add_copy(it.B, it.ldb, it.offB, it.lb, it.t.m, it.t.n, it.exact);
      if (it.stage_a) add_copy(it.A, it.lda, it.offA, it.la, ka, ka, it.exact);
    }
    if (part == 0) copies_first = copies.size();
  }
  if (std::max(copy_blocks[0], copy_blocks[1]) > INT32_MAX)
    return fail(UVATRMM_EINVAL, "group too large for one staging launch");
  if (!copies.empty()) {
    e = cudaMemcpy(base + off_copy, copies.data(), copies.size() * sizeof(CopyJob), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return cuda_fail(e, "staging jobs");
  }
  SmallList smalls[2];  // the small kernel's own problems; those it stands behind the lossless route for
  for (auto &it : f64) {
    if (!it.small) continue;
    SmallProduct p =
        small_trmm(it.t, it.A, it.lda, reinterpret_cast<double *>(base + it.offB), it.lb, it.B, it.ldb, 0.0);
    p.part = reinterpret_cast<double *>(base + it.offPart);
    if (it.exact >= 0) p.gate = gates + it.exact;
    smalls[it.exact >= 0].add(p, it.exact >= 0 ? kGatedUnits : 1);
    // (Counted as the tile kernel's tiles, which are its outputs' measure.)
    g->fp64_tiles += (it.t.m + 63) / 64 * ((it.t.n + 63) / 64);
  }
  SmallJob *dsmall[2] = {reinterpret_cast<SmallJob *>(base + off_small), nullptr};
  dsmall[1] = dsmall[0] + smalls[0].jobs.size();
  for (int k = 0; k < 2; ++k) {
    if (smalls[k].jobs.empty()) continue;
    e = cudaMemcpy(dsmall[k], smalls[k].jobs.data(), smalls[k].jobs.size() * sizeof(SmallJob),
                   cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return cuda_fail(e, "small FP64 jobs");
    if (int rc = small_group_prepare()) return fail(rc, "small kernel attributes");
  }
  std::vector<int> wave_total(waves.size(), 0);
  std::vector<OzWaveTables> wave_tab(waves.size());
  for (size_t w = 0; w < waves.size(); ++w) {
    std::vector<OzGroupProb> hd(waves[w].size());
    std::vector<OzWaveItem> items(waves[w].size());
    int begin = 0;
    for (size_t k = 0; k < waves[w].size(); ++k) {
      const OzItem &it = oz[waves[w][k]];
      const OzPlan &pl = it.plan;
      OzWaveItem &wi = items[k];
      ozaki_operands(it.t, it.A, it.lda, it.B, it.ldb, wi.L, wi.R);
      wi.sb = oz_scale_buf(base + off_wave + it.offE, pl.Mp, pl.Np, pl.K);
      wi.plan = pl;
      wi.LR = reinterpret_cast<uint16_t *>(base + off_wave + it.offP);
      wi.RR = wi.LR + (int64_t)pl.n_moduli * pl.Mp * pl.Kp;
      wi.res = reinterpret_cast<uint16_t *>(base + off_wave + it.offR);
      wi.alpha = it.t.alpha;
      wi.C = it.B;
      wi.ldc = it.ldb;
      wi.ctl = it.ctl >= 0 ? gates + it.ctl : nullptr;
      OzGemmLaunch L;
      L.ctl = wi.ctl;
      L.LR = reinterpret_cast<uint16_t *>(base + off_wave + it.offP);
      L.RR = L.LR + (int64_t)pl.n_moduli * pl.Mp * pl.Kp;
      L.res = reinterpret_cast<uint16_t *>(base + off_wave + it.offR);
      L.Mp = pl.Mp; L.Np = pl.Np; L.Kp = pl.Kp; L.M = pl.M; L.N = pl.N; L.K = pl.K;
      L.l0 = 0; L.l1 = pl.n_moduli;
      L.n_moduli = pl.n_moduli;
      L.tri_left = it.t.side == CblasLeft;
      L.tri_lower = (it.t.uplo == CblasLower) != (it.t.trans != 0);
      L.raster_group = it.raster;
      L.status = h->dctl + 1;
      L.num_sms = h->num_sms;
      if (int rc = oz_group_prob(L, &hd[k], &why)) return fail(rc, why ? why : "Ozaki descriptor");
      hd[k].tile_begin = begin;
      begin += hd[k].tile_count;
    }
    wave_total[w] = begin;
    g->oz_tiles += begin;
    e = cudaMemcpy(base + off_wdesc[w], hd.data(), hd.size() * sizeof(OzGroupProb), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return cuda_fail(e, "Ozaki descriptors");
    if (int rc = oz_wave_tables(items.data(), (int)items.size(), base + off_wtab[w], &wave_tab[w]))
      return fail(rc, "Ozaki wave job tables");
  }
  if (!waves.empty())
    if (int rc = oz_gemm_prepare()) return fail(rc, "residue GEMM attributes");
  g->waves = (int)waves.size();

  // ---- capture
  cudaStream_t st = h->stream;
  bool own_stream = false;
  if (!st) {  // the legacy default stream cannot be captured
    if ((e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking)) != cudaSuccess)
      return cuda_fail(e, "capture stream");
    own_stream = true;
  }
  e = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal);
  if (e != cudaSuccess) {
    if (own_stream) cudaStreamDestroy(st);
    return cuda_fail(e, "cudaStreamBeginCapture");
  }
  int rc = UVATRMM_OK;
  auto stage = [&](int part, cudaStream_t on) {
    if (rc != UVATRMM_OK || !copy_blocks[part]) return;
    const size_t first = part ? copies_first : 0, n = part ? copies.size() - copies_first : copies_first;
    stage_wave_kernel<<<(unsigned)copy_blocks[part], 256, 0, on>>>(
        reinterpret_cast<const CopyJob *>(base + off_copy) + first, (int)n);
    if (cudaGetLastError() != cudaSuccess) rc = UVATRMM_EDEVICE;
    g->launches += 1;
  };
  auto small = [&](int part, cudaStream_t on) {
    if (rc != UVATRMM_OK || smalls[part].jobs.empty()) return;
    rc = launch_small_group(dsmall[part], smalls[part], on);
    g->launches += smalls[part].reduce_blocks ? 2 : 1;
  };
  // The small kernel's own problems run beside the waves: it is bound by the
  // FP64 pipe, which the waves leave alone.
  cudaStream_t side = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;
  const bool beside = !smalls[0].jobs.empty() && !waves.empty();
  if (beside) {
    if ((e = cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking)) == cudaSuccess)
      e = cudaEventCreateWithFlags(&fork, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&join, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventRecord(fork, st);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(side, fork, 0);
    if (e != cudaSuccess) rc = UVATRMM_EDEVICE;
    stage(0, side);
    small(0, side);
    if (rc == UVATRMM_OK && cudaEventRecord(join, side) != cudaSuccess) rc = UVATRMM_EDEVICE;
  }
  for (size_t z = 0; z < zeros.size() && rc == UVATRMM_OK; ++z)
    if (cudaMemset2DAsync(zeros[z].first, zero_ld[z] * 8, 0, zeros[z].second.m * 8, zeros[z].second.n, st) !=
        cudaSuccess)
      rc = UVATRMM_EDEVICE;
  // Per wave: grouped scales + residues (2 launches), one grouped residue
  // GEMM, one grouped reassembly.
  for (size_t w = 0; w < waves.size() && rc == UVATRMM_OK; ++w) {
    rc = oz_wave_prep(wave_tab[w], st);
    if (rc == UVATRMM_OK)
      rc = launch_oz_gemm_group(reinterpret_cast<OzGroupProb *>(base + off_wdesc[w]), (int)waves[w].size(),
                                wave_total[w], h->dctl + 1, h->num_sms, st, &why);
    if (rc == UVATRMM_OK) rc = oz_wave_reassemble(wave_tab[w], st);
    g->launches += 4;
  }
  if (!beside) {
    stage(0, st);
    small(0, st);
  }
  stage(1, st);
  small(1, st);
  for (size_t c = 0; c < classes.size() && rc == UVATRMM_OK; ++c) {
    rc = launch_trmm_fp64_group(reinterpret_cast<Fp64GroupProb *>(base + off_desc[c]), (int)members[c].size(),
                                class_total[c], classes[c], UVATRMM_ENGINE_DFMA, ctl + (int)c, h->dctl + 1,
                                h->num_sms, st, &why);
    g->launches += 1;
  }
  if (beside && join && cudaStreamWaitEvent(st, join, 0) != cudaSuccess && rc == UVATRMM_OK) rc = UVATRMM_EDEVICE;
  cudaGraph_t graph = nullptr;
  e = cudaStreamEndCapture(st, &graph);
  if (side) cudaStreamDestroy(side);
  if (fork) cudaEventDestroy(fork);
  if (join) cudaEventDestroy(join);
  if (own_stream) cudaStreamDestroy(st);
  if (rc != UVATRMM_OK) {
    if (graph) cudaGraphDestroy(graph);
    return fail(rc, why ? why : "capturing the group failed");
  }
  if (e != cudaSuccess) return cuda_fail(e, "cudaStreamEndCapture");
  g->graph = graph;
  e = cudaGraphInstantiate(&g->exec, graph, 0);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGraphInstantiate");
  return UVATRMM_OK;
}

}  // namespace
}  // namespace uvt

using namespace uvt;

extern "C" {

UVATRMM_API int uvatrmm_group_create(uvatrmm_handle_t h, const uvatrmm_trmm_problem *problems, int count,
                                    uvatrmm_group_t *group) {
  if (!group) return fail(UVATRMM_EINVAL, "group pointer is NULL");
  *group = nullptr;
  if (!(h = resolve(h))) return uvatrmm_last_status();
  if (count < 0 || (count > 0 && !problems)) return fail(UVATRMM_EINVAL, "invalid problem list");
  std::lock_guard<std::mutex> lk(h->mu);
  auto *g = new uvatrmm_group_st();
  g->h = h;
  int rc = build(g, problems, count, true);
  if (rc != UVATRMM_OK) {
    destroy_group(g);
    return rc;
  }
  *group = g;
  h->groups++;
  return ok();
}

UVATRMM_API int uvatrmm_group_run(uvatrmm_group_t g) {
  if (!g) return fail(UVATRMM_EINVAL, "group is NULL");
  std::lock_guard<std::mutex> lk(g->h->mu);
  cudaError_t e = cudaGraphLaunch(g->exec, g->h->stream);
  return e == cudaSuccess ? ok() : cuda_fail(e, "cudaGraphLaunch");
}

UVATRMM_API int uvatrmm_group_stats(uvatrmm_group_t g, double *flops, int *launches, int64_t *fp64_tiles,
                                   int64_t *ozaki_tiles, int *ozaki_waves, int64_t *arena_bytes) {
  if (!g) return fail(UVATRMM_EINVAL, "group is NULL");
  if (flops) *flops = g->flops;
  if (launches) *launches = g->launches;
  if (fp64_tiles) *fp64_tiles = g->fp64_tiles;
  if (ozaki_tiles) *ozaki_tiles = g->oz_tiles;
  if (ozaki_waves) *ozaki_waves = g->waves;
  if (arena_bytes) *arena_bytes = (int64_t)g->arena_bytes;
  return ok();
}

UVATRMM_API int uvatrmm_group_destroy(uvatrmm_group_t g) {
  if (!g) return ok();
  {
    std::lock_guard<std::mutex> lk(g->h->mu);
    cudaStreamSynchronize(g->h->stream);
    g->h->groups--;
  }
  destroy_group(g);
  return ok();
}

}  // extern "C"
