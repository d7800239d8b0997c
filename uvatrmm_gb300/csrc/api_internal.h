// Internal host-side pieces shared by the C-ABI translation units.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <mutex>
#include <string>
#include <vector>

#include "uvatrmm.h"

// Offsets in the handle's control block (dctl), and its size: the lossless
// route's decision word, and the scaling's counters (16384 ints).
constexpr size_t kHandleCtlOffset = 256, kHandleCountersOffset = 512,
                 kHandleSlotsOffset = kHandleCountersOffset + 16384 * sizeof(int),
                 kHandleCtlBytes = kHandleSlotsOffset + 1024 * sizeof(unsigned long long);

struct uvatrmm_handle_st {
  int device = 0;
  int num_sms = 0;
  cudaStream_t stream = nullptr;
  int engine = UVATRMM_ENGINE_DFMA;
  bool engine_set = false;  // UVATRMM_OPT_ENGINE was set: FP64 calls stay on that engine
  int schedule = UVATRMM_SCHED_DYNAMIC;
  int shape = UVATRMM_SHAPE_TRAPEZOID;
  int tile = 0;
  int64_t ozaki_scratch_mb = 49152;  // residue-plane budget per pass (MiB)
  bool autotune = true;
  int oz_raster = 0;  // residue-GEMM raster group of single Ozaki calls (0 = default)
  uint32_t expiry_test_polls = 0;  // UVATRMM_OPT_WAIT_EXPIRY_TEST (0 = off)
  uint32_t exchange_expiry_polls = 0;  // UVATRMM_OPT_EXCHANGE_EXPIRY_TEST (0 = off)
  bool oz_err_host = false;        // UVATRMM_OPT_OZAKI_ERR_HOST
  // Grow-only device workspace slots: 0-2 plain-path and GEMM staging,
  // 3 reductions and the small kernel's partial sums, 4 Ozaki scales, 5 Ozaki residue planes, 6 Ozaki product
  // residues, 7 Ozaki error-estimate scratch and the block-cyclic pointer
  // tables.  Calls on a handle are serialised by `mu` and a slot's contents
  // live only within one call (a slot that grows first drains the stream).
  static constexpr int kSlots = 8;
  void *ws[kSlots] = {};
  size_t ws_cap[kSlots] = {};
  // Slots whose block was handed out during a stream capture, and such blocks
  // that were outgrown: kept until the handle goes, as a graph may use them.
  bool ws_captured[kSlots] = {};
  std::vector<void *> ws_kept;
  // What keeps a default handle when its thread ends: groups alive on it, or
  // calls on it that were captured.
  std::atomic<int> groups{0};
  bool captured = false;
  // [0] tile counter, [1] kernel status word, [2], [3] the server's tile
  // counters; the lossless route's OzCtl at kHandleCtlOffset, the scaling's
  // counters at kHandleCountersOffset, its blocks' words at kHandleSlotsOffset.
  int *dctl = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  // Per-stage GPU timing of the last Ozaki call (UVATRMM_OPT_STAGE_TIMING):
  // events bracket scaling, each pass's slicing and GEMM, and reassembly.
  bool stage_timing = false;
  static constexpr int kStageEvents = 48;
  cudaEvent_t sev[kStageEvents] = {};
  int n_sev = 0;
  int sev_kind[kStageEvents] = {};  // stage the interval ending at this event belongs to
  bool host_direct = false;  // kernels can address the host's pageable memory at its full rate
  // Host staging for host operands outside uvatrmm_host_alloc memory: two
  // page-locked huge-page buffers used alternately (host_mem.cu).
  size_t hstage_bytes = (size_t)256 << 20;  // chunk size (UVATRMM_OPT_HOST_STAGE_KB)
  void *hstage[2] = {};
  size_t hstage_cap = 0;
  cudaEvent_t hstage_ev[2] = {};
  std::mutex mu;
};

namespace uvt {

// Thread-local error reporting.
int fail(int status, const std::string &msg);
int ok();
int cuda_fail(cudaError_t e, const char *what);

// Returns the handle to use (the argument, or the calling thread's default
// handle on the current device); nullptr and an error set on failure.
uvatrmm_handle_t resolve(uvatrmm_handle_t h);

// Ensures workspace slot `slot` holds at least `bytes`; returns its pointer or nullptr.
void *workspace(uvatrmm_handle_t h, int slot, size_t bytes);
// True while the handle's stream is being captured into a graph.
bool stream_captures(uvatrmm_handle_t h);

// Host <-> device 2-D copy (`width` bytes x `height` lines) for the host
// entry points, ordered on h->stream.  Host memory from uvatrmm_host_alloc
// is copied directly; other host memory goes through the handle's staging
// buffers, packed by several CPU threads while the previous chunk's DMA
// runs.  A device-to-host copy has landed in `dst` when this returns.
cudaError_t host_copy2d(uvatrmm_handle_t h, void *dst, size_t dpitch, const void *src, size_t spitch, size_t width,
                        size_t height, cudaMemcpyKind kind);
// Host-to-device copy of the referenced triangle of the ka x ka
// column-major A (lower: rows j..ka-1 of column j; upper: rows 0..j), in
// blocks of kTriCopyCols columns, each block the rectangle over its part of
// the triangle.  The device copy's other entries are left as they were: the
// kernels never use the unreferenced triangle's values.
constexpr int64_t kTriCopyCols = 256;
cudaError_t copy_triangle_h2d(uvatrmm_handle_t h, double *dA, int64_t la, const double *A, int64_t lda, int64_t ka,
                              bool lower);
// `rc` of a host entry point that gives up after its copies were enqueued: the
// caller may free its buffers once this returns.
inline int drained(uvatrmm_handle_t h, int rc) {
  cudaStreamSynchronize(h->stream);
  return rc;
}
// True when [p, p + bytes) lies inside one uvatrmm_host_alloc region.
bool host_alloc_contains(const void *p, size_t bytes);
// Frees the handle's staging buffers and events.
void release_host_staging(uvatrmm_handle_t h);

// Reads and clears the kernel status word (synchronising the stream).
int collect_status(uvatrmm_handle_t h);

inline int64_t round_up(int64_t x, int64_t m) { return (x + m - 1) / m * m; }

// Column-major normalised TRMM description (CBLAS row-major calls are
// turned into the column-major call on the transposed matrices).
struct Trmm {
  int side, uplo, trans, unit;  // CBLAS enum values; trans/unit as 0/1
  int64_t m, n;                 // B is m x n
  double alpha;
};
int check_args(int layout, int side, int uplo, int transa, int diag, int64_t m, int64_t n, int64_t lda,
               int64_t ldb);
Trmm normalise(int layout, int side, int uplo, int transa, int diag, int64_t m, int64_t n, double alpha);

// FP64 TRMM on device buffers (stages misaligned operands, and B when in
// place, through workspace slots 0 and 1).  `plain`: on the tile kernel even
// where the lossless route would be taken.  `begin` (may be null) is recorded
// once the workspace is there, ahead of the work.
int device_trmm(uvatrmm_handle_t h, int layout, int side, int uplo, int transa, int diag, int64_t m, int64_t n,
                double alpha, const double *dA, int64_t lda, const double *dB, int64_t ldb, double *dC,
                int64_t ldc, bool in_place, int schedule, int shape, double beta = 0.0, bool plain = false,
                cudaEvent_t begin = nullptr);

// A small product for trmm_small.cu: out[r, v] = alpha * sum_k T[r, k] X[k, v]
// + beta * out[r, v] with T R x K (triangular, R = K, or dense).
struct SmallProduct {
  const double *T, *X;
  double *C;
  int64_t ldt;                   // T[r, k] = t_kcontig ? T[k + r ldt] : T[r + k ldt]
  int64_t k_stride, v_stride;    // X[k, v]
  int64_t ck_stride, cv_stride;  // out[r, v]
  int R, K, V;
  double alpha, beta;
  bool t_kcontig, tri, lower, unit;
  int kc;        // split: k per chunk (small_chunk()), 0 unsplit
  double *part;  // split: partial sums, small_part_bytes()
  const struct OzCtl *gate;  // lossless route in front: nothing to do where it computed the result
  int *counter;              // with `gate` in a launch of its own: zeroed by the route's scaling
};
constexpr int kSmallMaxK = 2048;  // of an unsplit product (its vectors lie in shared memory)
int small_chunk(int64_t R, int64_t V, int64_t K, bool tri);
size_t small_part_bytes(const SmallProduct &p);
// Its estimated time in us (a huge number where it cannot run), and whether
// it can run in place (X = out) without a copy of X.
double small_us(int64_t R, int64_t V, int64_t K, bool tri);
bool small_in_place(const SmallProduct &p);
int launch_small(const SmallProduct &p, bool in_place, cudaStream_t st);
// Many small products in two launches (the second adds partial sums).
struct SmallJob {
  SmallProduct p;
  int block_begin, reduce_begin;
  int units;  // (row block, vector group, chunk) triples per block
};
constexpr int kGatedUnits = 16;  // of jobs that mostly have nothing to do: fewer blocks to pass over
struct SmallList {
  std::vector<SmallJob> jobs;
  int blocks = 0, reduce_blocks = 0, max_len = 0;
  void add(SmallProduct p, int units);
};
int small_group_prepare();
// `jobs`: the list's jobs on the device.
int launch_small_group(const SmallJob *jobs, const SmallList &list, cudaStream_t st);
SmallProduct small_trmm(const Trmm &t, const double *A, int64_t lda, const double *B, int64_t ldb, double *C,
                        int64_t ldc, double beta);
// Gives a split product its partial sums' workspace; where there is none (no
// memory, or a stream capture before it was ever needed) unsplits it.  False:
// too long for one chunk, the tile kernel has to take it.
bool small_scratch(uvatrmm_handle_t h, SmallProduct *p);

struct OzOperand;
struct OzCtl;
inline OzCtl *handle_ctl(uvatrmm_handle_t h) {
  return reinterpret_cast<OzCtl *>(reinterpret_cast<char *>(h->dctl) + kHandleCtlOffset);
}
inline unsigned long long *fused_slots(uvatrmm_handle_t h) {
  return reinterpret_cast<unsigned long long *>(reinterpret_cast<char *>(h->dctl) + kHandleSlotsOffset);
}
inline int *scale_counters(uvatrmm_handle_t h) {
  return reinterpret_cast<int *>(reinterpret_cast<char *>(h->dctl) + kHandleCountersOffset);
}
// Kernel family for an M x N x K product (`tri`: one operand triangular) of
// a single call on a handle whose options leave the choice open.
enum class Route { kTile, kSmall, kExact };
Route pick_route(int64_t M, int64_t N, int64_t K, bool tri, bool tri_left, bool in_place = false, int64_t staged = 0);
// Behind the lossless route of a TRMM: the small kernel instead of the tile
// kernel where it is faster (the same bits where it is not split along K).
bool small_behind_exact(int64_t M, int64_t N, int64_t K, bool tri_left);
// True when no option pins the handle's FP64 calls to the tile kernel, nor
// the schedule and shape of this call.
inline bool route_free(uvatrmm_handle_t h, int schedule, int shape) {
  return !h->engine_set && !h->tile && !h->expiry_test_polls && h->schedule == UVATRMM_SCHED_DYNAMIC &&
         h->shape == UVATRMM_SHAPE_TRAPEZOID && schedule == UVATRMM_SCHED_DYNAMIC && shape == UVATRMM_SHAPE_TRAPEZOID;
}
// Enqueues C := alpha * Lft * Rgt + beta * C by the lossless route and gives
// the decision word by which the FP64 tile kernel and its staging copies
// behind it must be gated (they run where it says that the route did not).
// *gate = nullptr when the route is not possible (no room for its scratch):
// nothing has been enqueued then.  `stage`: where such a kernel needs a copy
// of C as it was (in place), which the route's last kernel then makes.
int exact_product(uvatrmm_handle_t h, const OzOperand &L, const OzOperand &R, bool tri_none, bool tri_left,
                  bool tri_lower, double alpha, double beta, double *C, int64_t ldc, const OzCtl **gate,
                  double *stage = nullptr, int64_t lds = 0);
// Takes the route's scratch for such a product ahead of the call.
void exact_reserve(uvatrmm_handle_t h, int64_t M, int64_t N, int64_t K, bool by_cols);
// Copies a column-major rows x cols block; with `gate`, only where the
// lossless route did not compute the result.
cudaError_t stage_copy(uvatrmm_handle_t h, double *dst, int64_t ldd, const double *src, int64_t lds, int64_t rows,
                       int64_t cols, const OzCtl *gate);
// The two operands of a normalised TRMM as the integer kernels see them.
void ozaki_operands(const Trmm &t, const double *dA, int64_t lda, const double *dB, int64_t ldb, OzOperand &L,
                    OzOperand &R);

// Ozaki emulated TRMM on device buffers, in place on dB (ozaki_api.cu).
int ozaki_device(uvatrmm_handle_t h, int layout, int side, int uplo, int transa, int diag, int64_t m, int64_t n,
                 double alpha, const double *dA, int64_t lda, double *dB, int64_t ldb, int moduli, double *relerr,
                 int *bits_out);

// Relative Frobenius error of S sampled result vectors `got` against a
// compensated FP64 host computation from op(A) (host memory, column-major
// view of the normalised call) and the S sampled input vectors `b` (both
// stored vector after vector, m entries each for side Left, n for side
// Right); ozaki_err.cu.
double host_ref_relerr(const Trmm &t, const double *A, int64_t lda, int S, const double *b, const double *got);

// Autotuner (tune.cu): tuned tile edge (FP64) or raster group (Ozaki) for a
// problem shape; measures and caches a missing bucket when h->autotune.
int tune_choice(uvatrmm_handle_t h, int tier, int side, int64_t m, int64_t n, int *choice);

// C := beta * C over a column-major rows x cols device block (extras.cu).
int scale_device(uvatrmm_handle_t h, double *C, int64_t ldc, int64_t rows, int64_t cols, double beta);

// ||X - R||_F / ||R||_F over column-major device blocks.
int rel_frobenius(uvatrmm_handle_t h, int64_t rows, int64_t cols, const double *X, int64_t ldx, const double *R,
                  int64_t ldr, double *rel);

}  // namespace uvt
