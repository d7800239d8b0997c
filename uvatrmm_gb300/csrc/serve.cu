// Request loop with continuous batching (see the serving section of uvatrmm.h).
//
// One server thread owns the device work:
//   admit  - FIFO: the head request is admitted when a slot is free and the
//            pool (one cudaMalloc of the HBM budget, first-fit) has room for
//            its working set; host-mode operands are copied in on a copy
//            stream; FP64 requests large enough for the lossless integer
//            route have their operands scaled there, and once the decision
//            is back on the host they are Ozaki work (with the moduli they
//            need: the rest of their planes goes back to the pool) or, where
//            it says no, FP64 tiles;
//   tick   - one grouped launch per kind over tile ranges taken from every
//            active request (Ozaki slicing of newly admitted requests, the
//            residue GEMM, Ozaki reassembly of requests whose last GEMM tiles
//            are in this tick, then the FP64 TRMM), alternating between two
//            compute streams with two ticks in flight, so one tick's tail
//            overlaps the next tick and the device never waits for the host;
//   retire - when a tick's Ozaki work completes, the Ozaki requests
//            reassembled in it are finished; when the whole tick completes,
//            its FP64 requests are (host mode: after their result's copy
//            back); their memory returns to the pool and waiters are woken.
#include <algorithm>
#include <chrono>
#include <condition_variable>
#include <cstring>
#include <deque>
#include <map>
#include <memory>
#include <string>
#include <thread>
#include <unordered_map>
#include <vector>

#include "api_internal.h"
#include "common.cuh"
#include "ozaki.cuh"
#include "trmm_fp64.cuh"

namespace {

using namespace uvt;

double now_s() {
  return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

size_t pool_round(size_t bytes) { return (bytes + 255) / 256 * 256; }

// First-fit allocator over [0, size) with 256-byte granularity.
class Pool {
 public:
  void init(size_t size) {
    size_ = size;
    free_.clear();
    free_[0] = size;
    used_ = peak_ = 0;
  }
  bool alloc(size_t bytes, size_t *off) {
    bytes = pool_round(bytes);
    for (auto it = free_.begin(); it != free_.end(); ++it) {
      if (it->second >= bytes) {
        *off = it->first;
        const size_t rest = it->second - bytes, at = it->first + bytes;
        free_.erase(it);
        if (rest) free_[at] = rest;
        used_ += bytes;
        peak_ = std::max(peak_, used_);
        return true;
      }
    }
    return false;
  }
  void release(size_t off, size_t bytes) {
    bytes = pool_round(bytes);
    used_ -= bytes;
    auto it = free_.emplace(off, bytes).first;
    auto nx = std::next(it);
    if (nx != free_.end() && it->first + it->second == nx->first) {
      it->second += nx->second;
      free_.erase(nx);
    }
    if (it != free_.begin()) {
      auto pv = std::prev(it);
      if (pv->first + pv->second == it->first) {
        pv->second += it->second;
        free_.erase(it);
      }
    }
  }
  size_t peak() const { return peak_; }

 private:
  size_t size_ = 0, used_ = 0, peak_ = 0;
  std::map<size_t, size_t> free_;
};

enum ReqState { PENDING, ACTIVE, DONE, FAILED, CANCELLED };

struct Req {
  int64_t id = 0;
  uvatrmm_trmm_problem p{};
  bool on_device = false;
  Trmm t{};
  double flops = 0.0;
  ReqState state = PENDING;
  int status = UVATRMM_OK;
  double t_submit = 0.0, t_done = 0.0;
  size_t bytes = 0, off = 0;
  // device view of the operands (user buffers or pool copies)
  const double *A = nullptr;
  int64_t lda = 0;
  double *Bin = nullptr;  // FP64 tiles: staged input copy; residues: the buffer sliced
  int64_t ldbin = 0;
  double *Cout = nullptr;  // where the result lands on the device
  int64_t ldc = 0;
  // copy-in (and the scaling of the lossless route) finished
  cudaEvent_t h2d = nullptr;
  bool h2d_pending = false;
  // Runs as residue GEMM tiles: the Ozaki tier, or the lossless route.
  bool oz = false;
  // Lossless route of an FP64 request: its decision is awaited (in pinned
  // slot ctl_slot), after which `oz` says whether it was taken.
  bool exact = false, deciding = false;
  int ctl_slot = -1;
  OzCtl *ctl = nullptr;
  size_t planes_at = 0;  // its planes' place in the pool block; given back from there on as the decision allows
  double *stage_b = nullptr;  // where B's copy goes if it becomes FP64 tiles
  int lane = 0;               // its copy stream
  cudaStream_t copy = nullptr;
  // FP64 tier: tiles, or (small) one launch unit of the small kernel
  Fp64GroupProb fd{};
  bool small = false;
  SmallProduct sp{};
  double *part = nullptr;  // its partial sums
  // Ozaki tier
  OzPlan plan{};
  OzGroupProb od{};
  OzScaleBuf sb{};
  uint16_t *LR = nullptr, *RR = nullptr;
  uint16_t *res = nullptr;
  bool prepped = false;
  // tile progress
  int total = 0, next = 0;
  double tile_cost = 0.0;  // work per tile (flops of its tier)
  int64_t last_tick = -1;
  bool copy_back = false;
  cudaEvent_t d2h = nullptr;
};

struct TickSlot {
  char *dev = nullptr;
  char *host = nullptr;  // pinned mirror
  cudaEvent_t done = nullptr;
  cudaEvent_t prepped = nullptr;  // this tick's Ozaki slicing finished
  cudaEvent_t gemm_done = nullptr;  // this tick's residue GEMM (and slicing) finished
  cudaEvent_t oz_done = nullptr;    // this tick's Ozaki work finished (before its FP64 launch)
  bool has_prep = false;
  bool oz_retired = false;          // finishing_oz already retired
  int64_t id = -1;
  std::vector<int64_t> finishing;     // FP64-tier requests whose last work is in this tick
  std::vector<int64_t> finishing_oz;  // Ozaki-tier requests reassembled in this tick
};

}  // namespace

struct uvatrmm_server_st {
  uvatrmm_handle_t h = nullptr;  // internal handle (status word, SM count)
  int device = 0;
  uvatrmm_server_config cfg{};
  // Ticks alternate between two compute streams, so one tick's tail overlaps
  // the next tick's start; cross-tick order comes from events.
  cudaStream_t cstream[2] = {nullptr, nullptr};
  // Copies in and out, and the scaling of FP64 requests for the lossless
  // route: a request keeps to one of these streams, so that the short
  // scalings of a burst run side by side.
  static constexpr int kCopyStreams = 4;
  cudaStream_t copy[kCopyStreams] = {};
  int *counters = nullptr;  // the scalings', kScaleTiles per copy stream
  char *arena = nullptr;
  Pool pool;
  // tick descriptor slots
  static constexpr int kSlots = 4;
  TickSlot slots[kSlots];
  size_t slot_bytes = 0;
  int64_t tick_counter = 0;
  bool route_ok = false;  // the creating handle's options leave the kernel family open
  OzCtl *ctl_host = nullptr;  // pinned, one per admitted request at most
  std::vector<int> ctl_free;
  std::deque<int64_t> inflight;  // tick ids in order
  // requests
  std::mutex mu;
  std::condition_variable cv_submit, cv_done;
  std::unordered_map<int64_t, std::unique_ptr<Req>> reqs;
  std::deque<int64_t> pending;
  std::vector<int64_t> active;
  int64_t next_id = 1;
  bool stop = false;
  std::thread worker;
  // stats
  std::vector<double> lat_ms;
  uvatrmm_server_stats st{};
};

namespace {

bool stages_a(const Req &r) {
  return !r.on_device || reinterpret_cast<uintptr_t>(r.p.A) % 16 || r.p.lda % 2;
}

// Scales, decision word, planes and product residues of `n` moduli.
struct OzBytes {
  size_t scale, ctl, planes, res;
};
OzBytes oz_bytes(const OzPlan &pl, int n, bool exact) {
  return {oz_scale_bytes(pl.Mp, pl.Np, pl.K), exact ? sizeof(OzCtl) : 0, (size_t)n * (pl.Mp + pl.Np) * pl.Kp * 2,
          (size_t)oz_res_planes(n) * pl.Mp * pl.Np * sizeof(uint16_t)};
}

// Partial sums of the small kernel, where the request may run on it.
size_t part_bytes(const Req &r) {
  if (!r.small && !(r.exact && small_behind_exact(r.t.m, r.t.n, r.plan.K, r.t.side == CblasLeft))) return 0;
  return small_part_bytes(small_trmm(r.t, nullptr, 0, nullptr, 0, nullptr, 0, 0.0));
}

size_t working_bytes(const Req &r) {
  const Trmm &t = r.t;
  const int64_t ka = t.side == CblasLeft ? t.m : t.n;
  size_t b = 0;
  auto add = [&](size_t x) { b += pool_round(x); };
  const bool tier_oz = r.p.tier == UVATRMM_TIER_OZAKI;
  if (stages_a(r)) add((size_t)round_up(ka, 16) * ka * 8);
  if (!tier_oz) {
    add((size_t)round_up(t.m, 16) * t.n * 8);            // staged input B
    if (!r.on_device) add((size_t)round_up(t.m, 16) * t.n * 8);  // output C
    add(part_bytes(r));
  } else if (!r.on_device) {
    add((size_t)round_up(t.m, 16) * t.n * 8);  // B copy, overwritten
  }
  if (tier_oz || r.exact) {
    const OzBytes o = oz_bytes(r.plan, r.plan.n_moduli, r.exact);
    add(o.scale);
    add(o.ctl);
    add(o.planes);
    add(o.res);
  }
  return b;
}

// The FP64 tile kernel's descriptor.
int setup_tiles(Req &r) {
  const Trmm &t = r.t;
  const int64_t ka = t.side == CblasLeft ? t.m : t.n;
  r.oz = false;
  if (r.small) {
    r.sp = small_trmm(t, r.A, r.lda, r.Bin, r.ldbin, r.Cout, r.ldc, 0.0);
    r.sp.part = r.part;
    r.total = 1;
    r.tile_cost = r.flops;
    return UVATRMM_OK;
  }
  Fp64Launch L;
  L.M = t.m;
  L.N = t.n;
  L.K = ka;
  L.alpha = t.alpha;
  L.C = r.Cout;
  L.ldc = r.ldc;
  L.unit = t.unit;
  L.tri_lower = (t.uplo == CblasLower) != (t.trans != 0);
  if (t.side == CblasLeft) {
    L.tri_left = true;
    L.xl = MatRef{r.A, ka, ka, r.lda};
    L.lft_kmajor = t.trans != 0;
    L.xr = MatRef{r.Bin, t.m, t.n, r.ldbin};
    L.rgt_kmajor = true;
  } else {
    L.tri_left = false;
    L.xl = MatRef{r.Bin, t.m, t.n, r.ldbin};
    L.lft_kmajor = false;
    L.xr = MatRef{r.A, ka, ka, r.lda};
    L.rgt_kmajor = t.trans == 0;
  }
  L.engine = UVATRMM_ENGINE_DFMA;
  L.schedule = UVATRMM_SCHED_DYNAMIC;
  L.shape = UVATRMM_SHAPE_TRAPEZOID;
  L.tile = 64;
  const char *why = nullptr;
  if (int rc = fp64_group_prob(L, 64, &r.fd, &why)) return rc;
  r.total = r.fd.tile_count;
  r.tile_cost = r.flops / std::max(1, r.total);
  return UVATRMM_OK;
}

// Lays the planes and product residues of plan.n_moduli moduli out from
// `planes` on and builds the residue GEMM's descriptor.
int setup_residues(uvatrmm_server_t s, Req &r, char *planes) {
  const Trmm &t = r.t;
  const OzPlan &pl = r.plan;
  r.LR = reinterpret_cast<uint16_t *>(planes);
  r.res = reinterpret_cast<uint16_t *>(planes + pool_round(oz_bytes(pl, pl.n_moduli, r.exact).planes));
  OzGemmLaunch L;
  L.LR = r.LR;
  L.RR = r.RR = r.LR + (int64_t)pl.n_moduli * pl.Mp * pl.Kp;
  L.res = r.res;
  L.Mp = pl.Mp; L.Np = pl.Np; L.Kp = pl.Kp; L.M = pl.M; L.N = pl.N; L.K = pl.K;
  L.l0 = 0;
  L.l1 = pl.n_moduli;
  L.n_moduli = pl.n_moduli;
  L.tri_left = t.side == CblasLeft;
  L.tri_lower = (t.uplo == CblasLower) != (t.trans != 0);
  L.raster_group = 0;
  L.status = s->h->dctl + 1;
  L.num_sms = s->h->num_sms;
  const char *why = nullptr;
  if (int rc = oz_group_prob(L, &r.od, &why)) return rc;
  r.oz = true;
  r.total = r.od.tile_count;
  r.tile_cost = (double)pl.n_moduli * 2.0 * pl.Mp * pl.Np * (pl.Kp / 2 + 64) / std::max(1, r.total);
  return UVATRMM_OK;
}

// Lays out the request's pool block and builds its descriptors.
int setup(uvatrmm_server_t s, Req &r) {
  const Trmm &t = r.t;
  const int64_t ka = t.side == CblasLeft ? t.m : t.n;
  char *base = s->arena + r.off;
  size_t cur = 0;
  auto take = [&](size_t x) {
    char *p = base + cur;
    cur += pool_round(x);
    return p;
  };
  const bool tier_oz = r.p.tier == UVATRMM_TIER_OZAKI;
  const int64_t la = round_up(ka, 16), lb = round_up(t.m, 16);
  r.lane = (int)(r.id % uvatrmm_server_st::kCopyStreams);
  r.copy = s->copy[r.lane];
  const cudaMemcpyKind kind = r.on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
  if (stages_a(r)) {
    double *dA = reinterpret_cast<double *>(take((size_t)la * ka * 8));
    if (cudaMemcpy2DAsync(dA, la * 8, r.p.A, r.p.lda * 8, ka * 8, ka, kind, r.copy) != cudaSuccess)
      return UVATRMM_EDEVICE;
    r.A = dA;
    r.lda = la;
    r.h2d_pending = true;
  } else {
    r.A = r.p.A;
    r.lda = r.p.lda;
  }
  // Residue work on device operands reads B where it lies; everything else
  // has its own copy.
  double *stage = nullptr;
  if (!tier_oz || !r.on_device) stage = reinterpret_cast<double *>(take((size_t)lb * t.n * 8));
  if (r.on_device && (tier_oz || r.exact)) {
    r.Bin = r.p.B;
    r.ldbin = r.p.ldb;
  } else {
    r.Bin = stage;
    r.ldbin = lb;
    if (cudaMemcpy2DAsync(r.Bin, lb * 8, r.p.B, r.p.ldb * 8, t.m * 8, t.n, kind, r.copy) != cudaSuccess)
      return UVATRMM_EDEVICE;
    r.h2d_pending = true;
  }
  if (const size_t pb = part_bytes(r)) r.part = reinterpret_cast<double *>(take(pb));
  if (r.on_device) {
    r.Cout = r.p.B;
    r.ldc = r.p.ldb;
  } else {
    r.Cout = tier_oz ? r.Bin : reinterpret_cast<double *>(take((size_t)lb * t.n * 8));
    r.ldc = lb;
    r.copy_back = true;
  }
  if (tier_oz || r.exact) {
    const OzPlan &pl = r.plan;
    const OzBytes o = oz_bytes(pl, pl.n_moduli, r.exact);
    r.sb = oz_scale_buf(take(o.scale), pl.Mp, pl.Np, pl.K);
    r.ctl = r.exact ? reinterpret_cast<OzCtl *>(take(o.ctl)) : nullptr;
    r.planes_at = cur;
    take(o.planes);
    take(o.res);
  }
  if (r.exact) {
    // Scaled and decided behind the copies; the host reads the decision.
    OzOperand L, R;
    ozaki_operands(t, r.A, r.lda, r.Bin, r.ldbin, L, R);
    r.stage_b = stage;
    r.ctl_slot = s->ctl_free.back();
    s->ctl_free.pop_back();
    if (cudaMemcpyAsync(r.ctl, &kOzCtlInit, sizeof(OzCtl), cudaMemcpyHostToDevice, r.copy) != cudaSuccess ||
        oz_scales(L, R, r.sb, s->counters + r.lane * kScaleTiles, r.ctl, nullptr, r.copy) != UVATRMM_OK ||
        cudaMemcpyAsync(s->ctl_host + r.ctl_slot, r.ctl, sizeof(OzCtl), cudaMemcpyDeviceToHost, r.copy) !=
            cudaSuccess)
      return UVATRMM_EDEVICE;
    r.h2d_pending = r.deciding = true;
  } else if (int rc = tier_oz ? setup_residues(s, r, base + r.planes_at) : setup_tiles(r)) {
    return rc;
  }
  if (r.h2d_pending) {
    if (cudaEventCreateWithFlags(&r.h2d, cudaEventDisableTiming) != cudaSuccess) return UVATRMM_EDEVICE;
    cudaEventRecord(r.h2d, r.copy);
  }
  return cur <= r.bytes ? UVATRMM_OK : UVATRMM_EINVAL;
}

// The decision of an FP64 request's scaling has arrived.
int decided(uvatrmm_server_t s, Req &r) {
  r.deciding = r.h2d_pending = false;  // everything on the copy stream before it is done too
  const OzCtl c = s->ctl_host[r.ctl_slot];
  s->ctl_free.push_back(r.ctl_slot);
  r.ctl_slot = -1;
  const bool go = c.go && c.n <= r.plan.n_moduli;
  size_t keep = r.planes_at;
  if (go) {
    r.plan.n_moduli = c.n;
    const OzBytes o = oz_bytes(r.plan, c.n, true);
    keep += pool_round(o.planes) + pool_round(o.res);
  }
  {
    std::lock_guard<std::mutex> lk(s->mu);
    if (keep < r.bytes) s->pool.release(r.off + keep, r.bytes - keep);
    r.bytes = keep;
  }
  if (go) return setup_residues(s, r, s->arena + r.off + r.planes_at);
  r.small = small_behind_exact(r.t.m, r.t.n, r.plan.K, r.t.side == CblasLeft);
  if (r.Bin != r.stage_b) {
    const int64_t lb = round_up(r.t.m, 16);
    if (cudaMemcpy2DAsync(r.stage_b, lb * 8, r.Bin, r.ldbin * 8, r.t.m * 8, r.t.n, cudaMemcpyDeviceToDevice,
                          r.copy) != cudaSuccess)
      return UVATRMM_EDEVICE;
    r.Bin = r.stage_b;
    r.ldbin = lb;
    r.h2d_pending = true;
    cudaEventRecord(r.h2d, r.copy);
  }
  return setup_tiles(r);
}

void finish(uvatrmm_server_t s, Req &r, int status) {
  r.state = status == UVATRMM_OK ? DONE : FAILED;
  r.status = status;
  r.t_done = now_s();
  // (What was enqueued for a request that fails may still use its memory.)
  if (status != UVATRMM_OK && r.copy) cudaStreamSynchronize(r.copy);
  if (r.bytes) s->pool.release(r.off, r.bytes);
  r.bytes = 0;
  if (r.ctl_slot >= 0) s->ctl_free.push_back(r.ctl_slot);
  r.ctl_slot = -1;
  if (r.h2d) cudaEventDestroy(r.h2d);
  if (r.d2h) cudaEventDestroy(r.d2h);
  r.h2d = r.d2h = nullptr;
  if (status == UVATRMM_OK) {
    s->st.completed++;
    s->st.served_flops += r.flops;
    s->lat_ms.push_back((r.t_done - r.t_submit) * 1e3);
    s->st.last_done_s = std::max(s->st.last_done_s, r.t_done);
  } else {
    s->st.failed++;
  }
}

// Bytes an area of a tick slot takes (descriptors start at multiples of 256).
size_t slot_area(size_t bytes) { return pool_round(bytes); }

// Builds and enqueues one tick; returns false when there was nothing to do.
bool launch_tick(uvatrmm_server_t s, std::vector<Req *> &act) {
  const int64_t id = s->tick_counter;
  TickSlot &slot = s->slots[id % uvatrmm_server_st::kSlots];
  // the slot's previous tick must be retired (inflight holds at most 2 < kSlots)
  std::vector<Req *> prep, reas;
  std::vector<Fp64GroupProb> fdesc;
  std::vector<OzGroupProb> odesc;
  std::vector<Req *> touched;
  double f_budget = s->cfg.tick_fp64_gflop * 1e9, o_budget = s->cfg.tick_ozaki_gflop * 1e9;
  SmallList sdesc;
  int f_begin = 0, o_begin = 0;
  // Order: the oldest request of each tier first, with at most a quarter of
  // the tier's tick (so nothing starves), then shortest remaining work first
  // (small requests are not stuck behind large ones).
  std::vector<Req *> order;
  std::vector<Req *> rest;
  Req *oldest[2] = {nullptr, nullptr};
  for (Req *r : act)
    if (!r->deciding && r->next < r->total) {
      const int k = r->oz;
      if (!oldest[k]) oldest[k] = r;
      else rest.push_back(r);
    }
  std::stable_sort(rest.begin(), rest.end(), [](const Req *a, const Req *b) {
    return (a->total - a->next) * a->tile_cost < (b->total - b->next) * b->tile_cost;
  });
  for (Req *r : oldest)
    if (r) order.push_back(r);
  order.insert(order.end(), rest.begin(), rest.end());
  // Tiles per request: first the shares above; then the tick is made
  // work-conserving -- budget nobody else could use goes to the requests in
  // the same order (the oldest first), so a request running with little
  // company is not held to a quarter of the device.
  std::vector<int> takes(order.size(), 0);
  int n_oz = 0, n_f64 = 0;
  for (size_t i = 0; i < order.size(); ++i) {
    Req *r = order[i];
    const bool oz = r->oz;
    double &budget = oz ? o_budget : f_budget;
    if (budget <= 0) continue;
    if ((oz ? n_oz : n_f64) >= s->cfg.max_active) continue;
    const double share = r == oldest[oz ? 1 : 0] ? 0.25 * (oz ? s->cfg.tick_ozaki_gflop : s->cfg.tick_fp64_gflop) * 1e9
                                                 : budget;
    const int take = (int)std::min<double>(r->total - r->next, std::max(1.0, std::ceil(share / r->tile_cost)));
    budget -= take * r->tile_cost;
    takes[i] = take;
    (oz ? n_oz : n_f64)++;
  }
  for (size_t i = 0; i < order.size(); ++i) {
    Req *r = order[i];
    if (!takes[i]) continue;
    double &budget = r->oz ? o_budget : f_budget;
    const int more = (int)std::min<double>(r->total - r->next - takes[i], std::floor(budget / r->tile_cost));
    if (more <= 0) continue;
    takes[i] += more;
    budget -= more * r->tile_cost;
  }
  for (size_t i = 0; i < order.size(); ++i) {
    Req *r = order[i];
    const int take = takes[i];
    if (!take) continue;
    const bool oz = r->oz;
    if (oz) {
      if (!r->prepped) {
        prep.push_back(r);
        r->prepped = true;
      }
      OzGroupProb d = r->od;
      d.tile_begin = o_begin;
      d.tile_count = take;
      d.tile_offset = r->next;
      o_begin += take;
      odesc.push_back(d);
    } else if (r->small) {
      sdesc.add(r->sp, 1);
    } else {
      Fp64GroupProb d = r->fd;
      d.tile_begin = f_begin;
      d.tile_count = take;
      d.tile_offset = r->next;
      f_begin += take;
      fdesc.push_back(d);
    }
    r->next += take;
    touched.push_back(r);
    if (r->next >= r->total) {
      if (oz) reas.push_back(r);
      r->last_tick = id;
    }
  }
  if (touched.empty()) return false;
  cudaStream_t cs = s->cstream[id & 1];
  const TickSlot *prev = id > 0 ? &s->slots[(id - 1) % uvatrmm_server_st::kSlots] : nullptr;
  // Wait for the staging copies of the requests in this tick.
  for (Req *r : touched)
    if (r->h2d_pending) {
      cudaStreamWaitEvent(cs, r->h2d, 0);
      r->h2d_pending = false;
    }
  // Descriptor image -> pinned slot -> device slot.
  OzWaveTables tprep{}, treas{};
  std::vector<char> img_prep, img_reas;
  auto items = [&](const std::vector<Req *> &v) {
    std::vector<OzWaveItem> it(v.size());
    for (size_t k = 0; k < v.size(); ++k) {
      Req &r = *v[k];
      ozaki_operands(r.t, r.A, r.lda, r.Bin, r.ldbin, it[k].L, it[k].R);
      it[k].sb = r.sb;
      it[k].plan = r.plan;
      it[k].LR = r.LR;
      it[k].RR = r.RR;
      it[k].res = r.res;
      it[k].alpha = r.t.alpha;
      it[k].C = r.Cout;
      it[k].ldc = r.ldc;
      it[k].ctl = r.ctl;
      it[k].scaled = r.exact;
    }
    return it;
  };
  // Only what the tick uses is copied.
  const size_t off_f64 = 0, off_small = slot_area(fdesc.size() * sizeof(Fp64GroupProb));
  const size_t off_oz = off_small + slot_area(sdesc.jobs.size() * sizeof(SmallJob));
  const size_t off_prep = off_oz + slot_area(odesc.size() * sizeof(OzGroupProb));
  const size_t off_reas = off_prep + (prep.empty() ? 0 : slot_area(oz_wave_table_bytes((int)prep.size())));
  const size_t used = off_reas + (reas.empty() ? 0 : slot_area(oz_wave_table_bytes((int)reas.size())));
  if (!prep.empty()) {
    auto it = items(prep);
    oz_wave_image(it.data(), (int)it.size(), slot.dev + off_prep, img_prep, &tprep);
  }
  if (!reas.empty()) {
    auto it = items(reas);
    oz_wave_image(it.data(), (int)it.size(), slot.dev + off_reas, img_reas, &treas);
  }
  memcpy(slot.host + off_f64, fdesc.data(), fdesc.size() * sizeof(Fp64GroupProb));
  memcpy(slot.host + off_small, sdesc.jobs.data(), sdesc.jobs.size() * sizeof(SmallJob));
  memcpy(slot.host + off_oz, odesc.data(), odesc.size() * sizeof(OzGroupProb));
  memcpy(slot.host + off_prep, img_prep.data(), img_prep.size());
  memcpy(slot.host + off_reas, img_reas.data(), img_reas.size());
  cudaMemcpyAsync(slot.dev, slot.host, used, cudaMemcpyHostToDevice, cs);
  const char *why = nullptr;
  int rc = UVATRMM_OK;
  if (!prep.empty()) {
    rc = oz_wave_prep(tprep, cs);
    cudaEventRecord(slot.prepped, cs);
  }
  slot.has_prep = !prep.empty();
  // Residue tiles of a request sliced in the previous tick (other stream).
  if (prev && prev->has_prep && !odesc.empty()) cudaStreamWaitEvent(cs, prev->prepped, 0);
  if (rc == UVATRMM_OK && !odesc.empty())
    rc = launch_oz_gemm_group(reinterpret_cast<OzGroupProb *>(slot.dev + off_oz), (int)odesc.size(), o_begin,
                              s->h->dctl + 1, s->h->num_sms, cs, &why);
  cudaEventRecord(slot.gemm_done, cs);
  // The tick's Ozaki work comes before its FP64 tiles, so Ozaki requests that
  // finish here retire on oz_done without waiting for those tiles.
  if (rc == UVATRMM_OK && !reas.empty()) {
    // Earlier residue tiles of these requests ran in previous ticks: the one
    // before this (other stream) up to its residue GEMM; older ticks retired.
    if (prev) cudaStreamWaitEvent(cs, prev->gemm_done, 0);
    rc = oz_wave_reassemble(treas, cs);
  }
  cudaEventRecord(slot.oz_done, cs);
  if (rc == UVATRMM_OK)
    rc = launch_small_group(reinterpret_cast<const SmallJob *>(slot.dev + off_small), sdesc, cs);
  if (rc == UVATRMM_OK && !fdesc.empty())
    rc = launch_trmm_fp64_group(reinterpret_cast<Fp64GroupProb *>(slot.dev + off_f64), (int)fdesc.size(),
                                f_begin, 64, UVATRMM_ENGINE_DFMA, s->h->dctl + 2 + (int)(id % 2), s->h->dctl + 1,
                                s->h->num_sms, cs, &why);
  // A tick retires only after the previous one, so completion is in order.
  if (prev) cudaStreamWaitEvent(cs, prev->done, 0);
  cudaEventRecord(slot.done, cs);
  slot.id = id;
  slot.finishing.clear();
  slot.finishing_oz.clear();
  slot.oz_retired = false;
  for (Req *r : touched)
    if (r->last_tick == id) {
      const bool oz = r->oz;
      (oz ? slot.finishing_oz : slot.finishing).push_back(r->id);
      if (r->copy_back) {
        cudaEventCreateWithFlags(&r->d2h, cudaEventDisableTiming);
        cudaStreamWaitEvent(r->copy, oz ? slot.oz_done : slot.done, 0);
        cudaMemcpy2DAsync(r->p.B, r->p.ldb * 8, r->Cout, r->ldc * 8, r->t.m * 8, r->t.n, cudaMemcpyDeviceToHost,
                          r->copy);
        cudaEventRecord(r->d2h, r->copy);
      }
    }
  if (rc != UVATRMM_OK)
    for (Req *r : touched) r->status = rc;
  s->inflight.push_back(id);
  s->tick_counter++;
  s->st.ticks++;
  return true;
}

void worker(uvatrmm_server_t s) {
  cudaSetDevice(s->device);
  std::vector<Req *> act;
  std::vector<int64_t> done_wait;  // host-mode requests waiting for their copy back
  while (true) {
    bool did = false;
    {
      std::unique_lock<std::mutex> lk(s->mu);
      // admit (FIFO)
      while (!s->pending.empty() && (int)s->active.size() < s->cfg.max_active) {
        Req &r = *s->reqs[s->pending.front()];
        if (r.state == CANCELLED) {
          s->pending.pop_front();
          continue;
        }
        size_t off;
        if (!s->pool.alloc(r.bytes, &off)) break;
        r.off = off;
        s->pending.pop_front();
        r.state = ACTIVE;
        int rc = setup(s, r);
        if (rc != UVATRMM_OK) {
          finish(s, r, rc);
          s->cv_done.notify_all();
          continue;
        }
        s->active.push_back(r.id);
        did = true;
      }
      s->st.peak_bytes = (int64_t)s->pool.peak();
      act.clear();
      for (int64_t id : s->active) act.push_back(s->reqs[id].get());
      if (s->stop && s->pending.empty() && s->active.empty() && s->inflight.empty() && done_wait.empty()) break;
    }
    // Decisions of the lossless route that have arrived.
    bool awaiting = false;
    for (size_t k = 0; k < act.size();) {
      Req &r = *act[k];
      const cudaError_t q = r.deciding ? cudaEventQuery(r.h2d) : cudaSuccess;
      if (q == cudaErrorNotReady) awaiting = true;
      if (r.deciding && q != cudaErrorNotReady) {
        const int rc = q == cudaSuccess ? decided(s, r) : UVATRMM_EDEVICE;
        did = true;
        if (rc != UVATRMM_OK) {
          std::lock_guard<std::mutex> lk(s->mu);
          s->active.erase(std::find(s->active.begin(), s->active.end(), r.id));
          finish(s, r, rc);
          s->cv_done.notify_all();
          act.erase(act.begin() + k);
          continue;
        }
      }
      ++k;
    }
    // launch while fewer than two ticks are in flight
    if (s->inflight.size() < 2 && launch_tick(s, act)) did = true;
    // Retire: the Ozaki requests of any tick in flight once its Ozaki work
    // is done; the oldest tick (with its FP64 requests) once it is done.
    auto retire = [&](const std::vector<int64_t> &ids, cudaError_t q) {
      std::lock_guard<std::mutex> lk(s->mu);
      for (int64_t rid : ids) {
        Req &r = *s->reqs[rid];
        s->active.erase(std::find(s->active.begin(), s->active.end(), rid));
        if (r.d2h) done_wait.push_back(rid);
        else finish(s, r, q == cudaSuccess ? r.status : UVATRMM_EDEVICE);
      }
      s->cv_done.notify_all();
    };
    for (int64_t tid : s->inflight) {
      TickSlot &slot = s->slots[tid % uvatrmm_server_st::kSlots];
      if (slot.oz_retired) continue;
      const cudaError_t q = cudaEventQuery(slot.oz_done);
      if (q == cudaErrorNotReady) continue;
      slot.oz_retired = true;
      if (!slot.finishing_oz.empty()) {
        retire(slot.finishing_oz, q);
        did = true;
      }
    }
    if (!s->inflight.empty()) {
      TickSlot &slot = s->slots[s->inflight.front() % uvatrmm_server_st::kSlots];
      cudaError_t q = cudaEventQuery(slot.done);
      if (q != cudaErrorNotReady) {
        s->inflight.pop_front();
        if (!slot.oz_retired) {
          slot.oz_retired = true;
          retire(slot.finishing_oz, q);
        }
        retire(slot.finishing, q);
        did = true;
      }
    }
    if (!done_wait.empty()) {
      std::lock_guard<std::mutex> lk(s->mu);
      for (size_t k = 0; k < done_wait.size();) {
        Req &r = *s->reqs[done_wait[k]];
        cudaError_t q = cudaEventQuery(r.d2h);
        if (q != cudaErrorNotReady) {
          finish(s, r, q == cudaSuccess ? r.status : UVATRMM_EDEVICE);
          done_wait.erase(done_wait.begin() + k);
          did = true;
        } else {
          ++k;
        }
      }
      s->cv_done.notify_all();
    }
    if (!did && !awaiting) {
      std::unique_lock<std::mutex> lk(s->mu);
      s->cv_submit.wait_for(lk, std::chrono::microseconds(50));
    }
  }
}

}  // namespace

using namespace uvt;

extern "C" {

UVATRMM_API int uvatrmm_server_create(uvatrmm_handle_t h, const uvatrmm_server_config *cfg, uvatrmm_server_t *out) {
  if (!out) return fail(UVATRMM_EINVAL, "server pointer is NULL");
  *out = nullptr;
  if (!(h = resolve(h))) return uvatrmm_last_status();
  auto *s = new uvatrmm_server_st();
  s->cfg.hbm_budget_bytes = (int64_t)120e9;
  s->cfg.max_active = 512;
  s->cfg.tick_fp64_gflop = 12.0;
  s->cfg.tick_ozaki_gflop = 3000.0;
  if (cfg) {
    if (cfg->hbm_budget_bytes > 0) s->cfg.hbm_budget_bytes = cfg->hbm_budget_bytes;
    if (cfg->max_active > 0) s->cfg.max_active = cfg->max_active;
    if (cfg->tick_fp64_gflop > 0) s->cfg.tick_fp64_gflop = cfg->tick_fp64_gflop;
    if (cfg->tick_ozaki_gflop > 0) s->cfg.tick_ozaki_gflop = cfg->tick_ozaki_gflop;
  }
  s->device = h->device;
  s->route_ok = route_free(h, h->schedule, h->shape);
  uvatrmm_handle_t ih = nullptr;
  int rc = uvatrmm_create(&ih);
  if (rc != UVATRMM_OK) {
    delete s;
    return rc;
  }
  s->h = ih;
  cudaError_t e = cudaStreamCreateWithFlags(&s->cstream[0], cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&s->cstream[1], cudaStreamNonBlocking);
  for (auto &c : s->copy)
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&c, cudaStreamNonBlocking);
  const size_t counter_bytes = uvatrmm_server_st::kCopyStreams * kScaleTiles * sizeof(int);
  if (e == cudaSuccess) e = cudaMalloc(&s->counters, counter_bytes);
  if (e == cudaSuccess) e = cudaMemset(s->counters, 0, counter_bytes);
  if (e == cudaSuccess) e = cudaMalloc(&s->arena, (size_t)s->cfg.hbm_budget_bytes);
  // tick slots: FP64, small and Ozaki descriptors, two wave tables, packed
  const size_t na = (size_t)s->cfg.max_active;
  s->slot_bytes = slot_area(na * sizeof(Fp64GroupProb)) + slot_area(na * sizeof(SmallJob)) +
                  slot_area(na * sizeof(OzGroupProb)) + 2 * slot_area(oz_wave_table_bytes((int)na));
  for (auto &sl : s->slots) {
    if (e == cudaSuccess) e = cudaMalloc(&sl.dev, s->slot_bytes);
    if (e == cudaSuccess) e = cudaMallocHost(&sl.host, s->slot_bytes);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&sl.done, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&sl.prepped, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&sl.gemm_done, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&sl.oz_done, cudaEventDisableTiming);
  }
  if (e == cudaSuccess) e = cudaMallocHost(&s->ctl_host, na * sizeof(OzCtl));
  for (int k = 0; k < (int)na; ++k) s->ctl_free.push_back(k);
  if (e == cudaSuccess && (fp64_group_prepare(64, UVATRMM_ENGINE_DFMA) || oz_gemm_prepare() || small_group_prepare())) e = cudaErrorUnknown;
  if (e != cudaSuccess) {
    const int code = cuda_fail(e, "server setup");
    uvatrmm_server_destroy(s);
    return code;
  }
  s->pool.init((size_t)s->cfg.hbm_budget_bytes);
  s->worker = std::thread(worker, s);
  *out = s;
  return ok();
}

UVATRMM_API int uvatrmm_server_submit(uvatrmm_server_t s, const uvatrmm_trmm_problem *p, int operands_on_device,
                                     int64_t *id) {
  if (!s || !p || !id) return fail(UVATRMM_EINVAL, "invalid arguments");
  if (int bad = check_args(p->layout, p->side, p->uplo, p->transa, p->diag, p->m, p->n, p->lda, p->ldb))
    return fail(UVATRMM_EINVAL, "parameter " + std::to_string(bad) + " had an illegal value");
  if (p->tier != UVATRMM_TIER_FP64 && p->tier != UVATRMM_TIER_OZAKI) return fail(UVATRMM_EINVAL, "unknown tier");
  if (p->tier == UVATRMM_TIER_OZAKI && p->moduli != 0 && (p->moduli < 2 || p->moduli > kMaxModuli))
    return fail(UVATRMM_EINVAL, "moduli out of range");
  auto r = std::make_unique<Req>();
  r->p = *p;
  r->on_device = operands_on_device != 0;
  r->t = normalise(p->layout, p->side, p->uplo, p->transa, p->diag, p->m, p->n, p->alpha);
  const Trmm &t = r->t;
  r->flops = t.side == CblasLeft ? (double)t.m * t.m * t.n : (double)t.n * t.n * t.m;
  OzPlan &pl = r->plan;
  pl.M = t.m;
  pl.N = t.n;
  pl.K = t.side == CblasLeft ? t.m : t.n;
  pl.Mp = oz_pad_rows(pl.M);
  pl.Np = oz_pad_cols(pl.N);
  pl.Kp = round_up(pl.K, 64);
  if (p->tier == UVATRMM_TIER_OZAKI) {
    pl.n_moduli = p->moduli ? p->moduli : ozaki_auto_moduli(pl.K);
    pl.bits = ozaki_bits(pl.n_moduli, pl.K);
  } else {
    pl.n_moduli = kCrtModuli;
    pl.bits = 0;
    if (s->route_ok && t.m && t.n && t.alpha != 0.0) {
      const Route route = pick_route(t.m, t.n, pl.K, true, t.side == CblasLeft);
      r->exact = route == Route::kExact;
      r->small = route == Route::kSmall;
    }
  }
  if (t.m == 0 || t.n == 0 || t.alpha == 0.0) {
    // Nothing for the device to multiply: served at once.
    if (t.alpha == 0.0 && t.m && t.n) {
      if (r->on_device) {
        cudaMemset2D(p->B, p->ldb * 8, 0, t.m * 8, t.n);
      } else {
        for (int64_t j = 0; j < t.n; ++j) memset(p->B + j * p->ldb, 0, (size_t)t.m * 8);
      }
    }
    std::lock_guard<std::mutex> lk(s->mu);
    r->id = s->next_id++;
    r->t_submit = now_s();
    if (s->st.submitted == 0) s->st.first_submit_s = r->t_submit;
    s->st.submitted++;
    *id = r->id;
    Req &rr = *r;
    s->reqs[rr.id] = std::move(r);
    finish(s, rr, UVATRMM_OK);
    s->cv_done.notify_all();
    return ok();
  }
  // The lossless route takes at most an eighth of the budget per request, so
  // that it does not narrow how many are admitted at once by much: planes for
  // as many moduli as that holds (which depends on the request alone, so that
  // its result does, too), until the decision tells how many are needed.
  r->bytes = working_bytes(*r);
  while (r->exact && (int64_t)r->bytes > s->cfg.hbm_budget_bytes / 8) {
    r->exact = --pl.n_moduli >= 2;
    r->bytes = working_bytes(*r);
  }
  std::lock_guard<std::mutex> lk(s->mu);
  if (s->stop) return fail(UVATRMM_EINVAL, "server is stopping");
  if ((int64_t)r->bytes > s->cfg.hbm_budget_bytes) {
    s->st.refused++;
    return fail(UVATRMM_EBUSY, "request needs " + std::to_string(r->bytes) + " bytes, more than the HBM budget");
  }
  r->id = s->next_id++;
  r->t_submit = now_s();
  if (s->st.submitted == 0) s->st.first_submit_s = r->t_submit;
  s->st.submitted++;
  *id = r->id;
  s->pending.push_back(r->id);
  s->reqs[r->id] = std::move(r);
  s->cv_submit.notify_one();
  return ok();
}

UVATRMM_API int uvatrmm_server_wait(uvatrmm_server_t s, int64_t id, double timeout_s) {
  if (!s) return fail(UVATRMM_EINVAL, "server is NULL");
  std::unique_lock<std::mutex> lk(s->mu);
  auto it = s->reqs.find(id);
  if (it == s->reqs.end()) return fail(UVATRMM_EINVAL, "unknown request id");
  Req &r = *it->second;
  auto finished = [&] { return r.state == DONE || r.state == FAILED || r.state == CANCELLED; };
  if (timeout_s < 0) s->cv_done.wait(lk, finished);
  else if (!s->cv_done.wait_for(lk, std::chrono::duration<double>(timeout_s), finished))
    return fail(UVATRMM_ENOTREADY, "request still in flight");
  if (r.state == CANCELLED) return fail(UVATRMM_EINVAL, "request was cancelled");
  if (r.state == FAILED) return fail(r.status, "request failed");
  return ok();
}

UVATRMM_API int uvatrmm_server_cancel(uvatrmm_server_t s, int64_t id) {
  if (!s) return fail(UVATRMM_EINVAL, "server is NULL");
  std::lock_guard<std::mutex> lk(s->mu);
  auto it = s->reqs.find(id);
  if (it == s->reqs.end()) return fail(UVATRMM_EINVAL, "unknown request id");
  Req &r = *it->second;
  if (r.state != PENDING) return fail(UVATRMM_EBUSY, "request already admitted");
  r.state = CANCELLED;
  s->pending.erase(std::find(s->pending.begin(), s->pending.end(), id));
  s->st.cancelled++;
  s->cv_done.notify_all();
  return ok();
}

UVATRMM_API int uvatrmm_server_latency(uvatrmm_server_t s, int64_t id, double *ms) {
  if (!s || !ms) return fail(UVATRMM_EINVAL, "invalid arguments");
  std::lock_guard<std::mutex> lk(s->mu);
  auto it = s->reqs.find(id);
  if (it == s->reqs.end()) return fail(UVATRMM_EINVAL, "unknown request id");
  const Req &r = *it->second;
  if (r.state != DONE) return fail(r.state == FAILED ? r.status : UVATRMM_ENOTREADY, "request not completed");
  *ms = (r.t_done - r.t_submit) * 1e3;
  return ok();
}

UVATRMM_API int uvatrmm_server_get_stats(uvatrmm_server_t s, uvatrmm_server_stats *out) {
  if (!s || !out) return fail(UVATRMM_EINVAL, "invalid arguments");
  std::lock_guard<std::mutex> lk(s->mu);
  *out = s->st;
  std::vector<double> v = s->lat_ms;
  if (!v.empty()) {
    std::sort(v.begin(), v.end());
    auto pct = [&](double q) { return v[std::min(v.size() - 1, (size_t)(q * (v.size() - 1) + 0.5))]; };
    out->p50_ms = pct(0.5);
    out->p99_ms = pct(0.99);
    out->max_ms = v.back();
    double sum = 0;
    for (double x : v) sum += x;
    out->mean_ms = sum / v.size();
  }
  out->peak_bytes = (int64_t)s->pool.peak();
  return ok();
}

UVATRMM_API int uvatrmm_server_destroy(uvatrmm_server_t s) {
  if (!s) return ok();
  {
    std::lock_guard<std::mutex> lk(s->mu);
    s->stop = true;
    s->cv_submit.notify_all();
  }
  if (s->worker.joinable()) s->worker.join();
  for (auto cs : s->cstream)
    if (cs) cudaStreamSynchronize(cs);
  for (auto c : s->copy)
    if (c) cudaStreamSynchronize(c);
  for (auto &sl : s->slots) {
    if (sl.dev) cudaFree(sl.dev);
    if (sl.host) cudaFreeHost(sl.host);
    if (sl.done) cudaEventDestroy(sl.done);
    if (sl.prepped) cudaEventDestroy(sl.prepped);
    if (sl.gemm_done) cudaEventDestroy(sl.gemm_done);
    if (sl.oz_done) cudaEventDestroy(sl.oz_done);
  }
  if (s->ctl_host) cudaFreeHost(s->ctl_host);
  if (s->arena) cudaFree(s->arena);
  for (auto cs : s->cstream)
    if (cs) cudaStreamDestroy(cs);
  for (auto c : s->copy)
    if (c) cudaStreamDestroy(c);
  if (s->counters) cudaFree(s->counters);
  if (s->h) uvatrmm_destroy(s->h);
  delete s;
  return ok();
}

}  // extern "C"
