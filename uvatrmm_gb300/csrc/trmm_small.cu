// Small FP64 products: one launch, one output per thread.
//
// The FP64 pipe bounds every FP64 product here (2 FMAs per clock per SM, so
// one warp FMA holds an SM quarter's pipe for 64 clocks), and a 64 x 64 tile
// keeps one SM busy for 0.99 us per k while the others idle.  Small products
// are therefore spread as thin as they go: a block of four warps takes 32
// rows of the left matrix T and four vectors, each warp one vector, each lane
// one output, so a single warp per SM quarter already saturates its pipe and
// there are enough of them from 64 x 64 on.  Operands need no register
// tiles: 64 clocks per FMA leave room for its two shared-memory reads.
//
// Unsplit, every output sums its products in increasing k from zero, as the
// tile kernel does, so both give the same bits.  A lone warp's dependent FMAs
// take 0.07 us per k, so where there are too few outputs for the chip K is
// split into chunks of kc, each block sums one chunk, and a second launch adds
// an output's partial sums in the chunks' order.  kc depends on the problem's
// sizes alone: a call, a group and the server give the same bits, unless the
// partial sums' workspace is not to be had (a first call that is captured, or
// no memory): then the product runs unsplit, or on the tile kernel.
//
// In place unsplit, the blocks of one vector group (all rows, up to 8 x 32) form a
// cluster: they read the vectors, meet at the cluster's barrier, and only
// then overwrite them, which saves the staging copy's launch.
//
// Measured against the tile kernel (side L, out of place, per call): 64 x 64
// 9.3 against 51 us, 128 x 128 12.8 / 133, 256 x 256 32 / 287, 1000 x 1
// 12.8 / 280 (unsplit 76), 4000 x 1 34 / 1122; from about 300 x 300 on the
// lossless route is faster than both.
#include <algorithm>
#include <cmath>

#include "api_internal.h"
#include "common.cuh"
#include "ozaki.cuh"

namespace uvt {
namespace {

constexpr int kRows = 32, kVecs = 4, kChunk = 32, kThreads = 32 * kVecs;
constexpr int kMaxCluster = 8;

__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// Row block bx, vector group by: out[r, v] = alpha * sum_k T[r, k] X[k, v] (+ beta * out[r, v]);
// split, the sum over chunk bz into part[bz][v][r].
template <bool CLUSTER>
__device__ __forceinline__ void small_body(const SmallProduct &p, int bx, int by, int bz, double *vs) {
  __shared__ double ts[2][kChunk][kRows + 1];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int r0 = bx * kRows, v0 = by * kVecs;
  // k range of this row block, from a chunk boundary on.
  int k0 = 0, k1 = p.K;
  if (p.tri) {
    if (p.lower) k1 = min(p.K, r0 + kRows);
    else k0 = r0;
  }
  const int len = p.kc ? p.kc : p.K;  // of a vector in shared memory
  if (p.kc) {
    k0 = max(k0, bz * p.kc);
    k1 = min(k1, (bz + 1) * p.kc);
    if (k0 >= k1) return;
  }
  // T[r0.., k..k+32): eight elements per thread, consecutive threads along
  // the stored matrix's contiguous dimension; outside the triangle and the
  // matrix nothing is read.
  double t[8];
  auto load = [&](int k) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int a = lane, b = warp + 4 * q;  // contiguous, other
      const int r = r0 + (p.t_kcontig ? b : a), kk = k + (p.t_kcontig ? a : b);
      const bool in = r < p.R && kk < p.K && (!p.tri || (p.lower ? kk <= r : kk >= r));
      double x = 0.0;
      if (in) x = p.tri && p.unit && kk == r ? 1.0 : p.T[p.t_kcontig ? kk + (int64_t)r * p.ldt : r + (int64_t)kk * p.ldt];
      t[q] = x;
    }
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int a = lane, b = warp + 4 * q;
      if (p.t_kcontig) ts[buf][a][b] = t[q];
      else ts[buf][b][a] = t[q];
    }
  };
  load(k0);
  // The vectors' part [k0, k1) (all of them are read here or in the cluster's
  // other blocks before anything is overwritten).
  const int span = k1 - k0;
  for (int i = tid; i < span * kVecs; i += kThreads) {
    const int v = p.v_stride == 1 ? i % kVecs : i / span, k = k0 + (p.v_stride == 1 ? i / kVecs : i % span);
    vs[v * len + k - k0] = v0 + v < p.V ? p.X[(int64_t)k * p.k_stride + (int64_t)(v0 + v) * p.v_stride] : 0.0;
  }
  if (CLUSTER) cluster_arrive();
  store(0);
  __syncthreads();
  const double *vec = vs + warp * len - k0;
  const int r = r0 + lane;
  const bool mine = v0 + warp < p.V;  // this warp has a vector (idle FMAs would hold the pipe)
  double acc = 0.0;
  int buf = 0;
  for (int k = k0; k < k1; k += kChunk, buf ^= 1) {
    const bool more = k + kChunk < k1;
    if (more) load(k + kChunk);
    const int n = min(kChunk, k1 - k);
    if (mine) {
      if (p.tri && k + kChunk > r0 && k < r0 + kRows) {
        // On the diagonal: a zero outside the triangle is not multiplied, so
        // that an infinity or NaN there does not reach the row.
#pragma unroll 4
        for (int i = 0; i < n; ++i)
          if (p.lower ? k + i <= r : k + i >= r) acc = fma(ts[buf][i][lane], vec[k + i], acc);
      } else if (n == kChunk) {
#pragma unroll 8
        for (int i = 0; i < kChunk; ++i) acc = fma(ts[buf][i][lane], vec[k + i], acc);
      } else {
        for (int i = 0; i < n; ++i) acc = fma(ts[buf][i][lane], vec[k + i], acc);
      }
    }
    if (more) store(buf ^ 1);
    __syncthreads();
  }
  if (CLUSTER) cluster_wait();
  if (r < p.R && mine && p.kc) {
    p.part[((int64_t)bz * p.V + v0 + warp) * p.R + r] = acc;
  } else if (r < p.R && mine) {
    double *c = p.C + (int64_t)r * p.ck_stride + (int64_t)(v0 + warp) * p.cv_stride;
    *c = p.beta != 0.0 ? fma(p.beta, *c, p.alpha * acc) : p.alpha * acc;
  }
}

// The row blocks of a vector group are rotated from group to group: blocks go
// to SMs in turn, and an SM that always got the triangle's longest rows would
// finish last (m = n = 256: 41 -> 36 us).
__device__ __forceinline__ int rotated(int x, int y, int nx) { return (x + y) % nx; }

template <bool CLUSTER>
__global__ void __launch_bounds__(kThreads) trmm_small_kernel(const __grid_constant__ SmallProduct p) {
  extern __shared__ double vs[];  // [vector][k]
  small_body<CLUSTER>(p, rotated((int)blockIdx.x, (int)(blockIdx.y + blockIdx.z), (int)gridDim.x), (int)blockIdx.y,
                      (int)blockIdx.z, vs);
}

// Behind the lossless route: mostly there is nothing to do, so few blocks
// (m = n = 1000: 9.9 us for 8000 that return at once).  They take their units
// from the call's counter: dealt out in turns, those of the blocks that are not
// resident at first (1216 of seven per SM, fewer by shared memory from K = 500
// on) ran last on a chip otherwise idle (768 x 2564: 1626 -> 1367 us, 65 x 30730 402 -> 325).
constexpr int kGatedBlocks = 1216;
__global__ void __launch_bounds__(kThreads) trmm_small_gated_kernel(const __grid_constant__ SmallProduct p) {
  extern __shared__ double vs[];
  __shared__ int next;
  chain_wait();
  if (p.gate->go) return;
  const int nx = (p.R + kRows - 1) / kRows, ny = (p.V + kVecs - 1) / kVecs;
  const int units = nx * ny * (p.kc ? (p.K + p.kc - 1) / p.kc : 1);
  for (;;) {
    if (threadIdx.x == 0) next = atomicAdd(p.counter, 1);
    __syncthreads();
    const int i = next;
    if (i >= units) return;
    const int y = i / nx % ny, z = i / nx / ny;
    small_body<false>(p, rotated(i % nx, y + z, nx), y, z, vs);
    __syncthreads();  // the unit has read its vectors
  }
}

int splits_of(const SmallProduct &p) { return p.kc ? (p.K + p.kc - 1) / p.kc : 1; }

// The partial sums of outputs [256 b, 256 b + 256) of a split product, in the chunks' order.
__device__ __forceinline__ void reduce_body(const SmallProduct &p, int b) {
  const int64_t i = (int64_t)b * 256 + threadIdx.x;
  if (i >= (int64_t)p.R * p.V) return;
  const int v = (int)(i / p.R), r = (int)(i - (int64_t)v * p.R), r0 = r / kRows * kRows;
  int c0 = 0, c1 = (p.K + p.kc - 1) / p.kc;  // the chunks this row block has
  if (p.tri) {
    if (p.lower) c1 = (min(p.K, r0 + kRows) + p.kc - 1) / p.kc;
    else c0 = r0 / p.kc;
  }
  double acc = 0.0;
#pragma unroll 4
  for (int c = c0; c < c1; ++c) acc += p.part[((int64_t)c * p.V + v) * p.R + r];
  double *out = p.C + (int64_t)r * p.ck_stride + (int64_t)v * p.cv_stride;
  *out = p.beta != 0.0 ? fma(p.beta, *out, p.alpha * acc) : p.alpha * acc;
}

__global__ void __launch_bounds__(256) trmm_small_reduce_kernel(const __grid_constant__ SmallProduct p) {
  chain_wait();
  if (p.gate && p.gate->go) return;
  reduce_body(p, (int)blockIdx.x);
}

// Many small products in one launch (none of them in place): block b belongs
// to the job whose range [block_begin, next job's) holds it.
__device__ __forceinline__ int find_small(const SmallJob *jobs, int n, int b, bool reduce) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if ((reduce ? jobs[mid].reduce_begin : jobs[mid].block_begin) <= b) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

__global__ void __launch_bounds__(kThreads) trmm_small_group_kernel(const SmallJob *jobs, int n) {
  extern __shared__ double vs[];
  const int b = (int)blockIdx.x, j = find_small(jobs, n, b, false);
  const SmallProduct p = jobs[j].p;
  if (p.gate && p.gate->go) return;
  const int nx = (p.R + kRows - 1) / kRows, ny = (p.V + kVecs - 1) / kVecs, units = jobs[j].units;
  const int nz = p.kc ? (p.K + p.kc - 1) / p.kc : 1;
  const int first = (b - jobs[j].block_begin) * units;
  for (int i = first; i < min(first + units, nx * ny * nz); ++i) {
    if (i > first) __syncthreads();  // the unit before has read its vectors
    const int y = i / nx % ny, z = i / nx / ny;
    small_body<false>(p, rotated(i % nx, y + z, nx), y, z, vs);
  }
}

__global__ void __launch_bounds__(256) trmm_small_reduce_group_kernel(const SmallJob *jobs, int n) {
  const int b = (int)blockIdx.x, j = find_small(jobs, n, b, true);
  const SmallProduct &p = jobs[j].p;
  if (!p.kc || (p.gate && p.gate->go)) return;
  reduce_body(p, b - jobs[j].reduce_begin);
}

}  // namespace

int small_chunk(int64_t R, int64_t V, int64_t K, bool tri) {
  // Chunks for four warps per SM quarter, of 64 to 1024 k; none where one
  // chunk would hold nearly all of K, or the partial sums take over 8 MB.
  const double warps = std::ceil(R / 32.0) * (double)V;
  const double kc = (double)K * (tri ? std::min(1.0, 0.5 * (1 + 32.0 / R)) : 1.0) * warps / 2432;
  const int64_t c = (std::max<int64_t>(64, std::min<int64_t>(1024, (int64_t)kc)) + 31) / 32 * 32;
  if (c * 4 >= K * 3 || (double)((K + c - 1) / c) * V * R * 8 > 8e6) return 0;
  return (int)c;
}

double small_us(int64_t R, int64_t V, int64_t K, bool tri) {
  const int kc = small_chunk(R, V, K, tri);
  // (65535: the grid's y and z.)
  if ((!kc && K > kSmallMaxK) || R > (1 << 20) || V > 65535 * kVecs || (kc && (K + kc - 1) / kc > 65535)) return 1e30;
  // Launch (two when split); then a lone warp's dependent FMAs (0.07 us per k
  // of its chunk), or 64 clocks of an SM quarter's pipe per warp FMA at five
  // sixths and the uneven end, or the matrix's bytes.
  const double warps = std::ceil(R / 32.0) * (double)V, k = (double)K, frac = tri ? 0.5 * (1 + 32.0 / R) : 1.0;
  const double fmas = warps * k * std::min(1.0, frac) / 608;
  const double bytes_us = 8.0 * R * k * std::min(1.0, frac) / 4e6;
  if (kc) return 9 + std::max(std::max(0.070 * kc, 0.037 * fmas + 0.04 * kc), bytes_us);
  return 5 + std::max(0.070 * k, 0.037 * fmas + 0.04 * k);
}

bool small_in_place(const SmallProduct &p) { return p.kc || p.R <= kMaxCluster * kRows; }

size_t small_part_bytes(const SmallProduct &p) {
  return p.kc ? (size_t)splits_of(p) * p.V * p.R * sizeof(double) : 0;
}

int launch_small(const SmallProduct &p, bool in_place, cudaStream_t st) {
  if ((!p.kc && p.K > kSmallMaxK) || p.K < 1 || (in_place && !small_in_place(p))) return UVATRMM_EINVAL;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((p.R + kRows - 1) / kRows), (unsigned)((p.V + kVecs - 1) / kVecs),
                     (unsigned)splits_of(p));
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = (size_t)(p.kc ? p.kc : p.K) * kVecs * sizeof(double);
  cfg.stream = st;
  const bool cluster = in_place && !p.kc && cfg.gridDim.x > 1;
  static const bool ready =
      cudaFuncSetAttribute(trmm_small_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           kSmallMaxK * kVecs * (int)sizeof(double)) == cudaSuccess &&
      cudaFuncSetAttribute(trmm_small_gated_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           kSmallMaxK * kVecs * (int)sizeof(double)) == cudaSuccess;
  if (!ready || cfg.gridDim.y > 65535u || cfg.gridDim.z > 65535u) return UVATRMM_EDEVICE;
  cudaError_t e;
  if (cluster) {
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = cfg.gridDim.x;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, trmm_small_kernel<true>, p);
  } else if (p.gate) {
    const int64_t units = (int64_t)cfg.gridDim.x * cfg.gridDim.y * cfg.gridDim.z;
    e = launch_chained(trmm_small_gated_kernel, dim3((unsigned)std::min<int64_t>(units, kGatedBlocks)), cfg.blockDim,
                       cfg.dynamicSmemBytes, st, p);
  } else {
    e = cudaLaunchKernelEx(&cfg, trmm_small_kernel<false>, p);
  }
  if (e == cudaSuccess && p.kc)
    e = launch_chained(trmm_small_reduce_kernel, dim3((unsigned)(((int64_t)p.R * p.V + 255) / 256)), dim3(256), 0, st,
                       p);
  return e == cudaSuccess ? UVATRMM_OK : UVATRMM_EDEVICE;
}

int small_blocks(const SmallJob &j) {
  const int units = (j.p.R + kRows - 1) / kRows * ((j.p.V + kVecs - 1) / kVecs) * splits_of(j.p);
  return (units + j.units - 1) / j.units;
}
int small_reduce_blocks(const SmallJob &j) { return j.p.kc ? (int)(((int64_t)j.p.R * j.p.V + 255) / 256) : 0; }

int small_group_prepare() {
  static const bool ready =
      cudaFuncSetAttribute(trmm_small_group_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           kSmallMaxK * kVecs * (int)sizeof(double)) == cudaSuccess;
  return ready ? UVATRMM_OK : UVATRMM_EDEVICE;
}

void SmallList::add(SmallProduct p, int units) {
  SmallJob j{p, blocks, reduce_blocks, units};
  blocks += small_blocks(j);
  reduce_blocks += small_reduce_blocks(j);
  max_len = std::max(max_len, p.kc ? p.kc : p.K);
  jobs.push_back(j);
}

int launch_small_group(const SmallJob *jobs, const SmallList &list, cudaStream_t st) {
  const int n = (int)list.jobs.size();
  if (n == 0) return UVATRMM_OK;
  if (int rc = small_group_prepare()) return rc;
  trmm_small_group_kernel<<<list.blocks, kThreads, (size_t)list.max_len * kVecs * sizeof(double), st>>>(jobs, n);
  if (list.reduce_blocks) trmm_small_reduce_group_kernel<<<list.reduce_blocks, 256, 0, st>>>(jobs, n);
  return cudaGetLastError() == cudaSuccess ? UVATRMM_OK : UVATRMM_EDEVICE;
}

SmallProduct small_trmm(const Trmm &t, const double *A, int64_t lda, const double *B, int64_t ldb, double *C,
                        int64_t ldc, double beta) {
  const bool lower = (t.uplo == CblasLower) != (t.trans != 0), left = t.side == CblasLeft;
  SmallProduct p{};
  p.T = A;
  p.ldt = lda;
  p.X = B;
  p.C = C;
  p.K = p.R = (int)(left ? t.m : t.n);
  p.V = (int)(left ? t.n : t.m);
  p.kc = small_chunk(p.R, p.V, p.K, true);
  p.alpha = t.alpha;
  p.beta = beta;
  p.tri = true;
  p.unit = t.unit;
  // Left: T = op(A), vectors are B's columns.  Right: T = op(A)^T, B's rows.
  p.lower = left ? lower : !lower;
  p.t_kcontig = left == (t.trans != 0);
  p.k_stride = left ? 1 : ldb;
  p.v_stride = left ? ldb : 1;
  p.ck_stride = left ? 1 : ldc;
  p.cv_stride = left ? ldc : 1;
  return p;
}

}  // namespace uvt
