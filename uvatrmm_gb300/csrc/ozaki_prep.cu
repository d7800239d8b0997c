// Ozaki path, memory-bound stages: per-row/column power-of-two scales, the
// residue planes (slicing), and the CRT reassembly to FP64.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "api_internal.h"
#include "common.cuh"
#include "ozaki.cuh"

namespace uvt {
namespace {

// ---------------------------------------------------------------- element access
__device__ __forceinline__ double load_elem(const OzOperand &op, int64_t p, int64_t k) {
  if (p >= op.P || k >= op.K) return 0.0;
  if (op.tri) {
    const int64_t r = op.p_is_row ? p : k, c = op.p_is_row ? k : p;
    if (r == c) return op.unit ? 1.0 : (op.kcontig ? op.X[k + p * op.ld] : op.X[p + k * op.ld]);
    if (op.lower ? (c > r) : (c < r)) return 0.0;
  }
  return op.kcontig ? op.X[k + p * op.ld] : op.X[p + k * op.ld];
}

// Triangular operand: its nonzeros lie at k <= p (else at k >= p).
__device__ __forceinline__ bool tri_k_le_p(const OzOperand &op) { return op.p_is_row == op.lower; }

// ilogb(|v|) + 1 for v != 0 (so |v| < 2^result), from the bits of |v|.
__device__ __forceinline__ int exp_above(uint64_t b) {
  const int be = (int)(b >> 52);
  if (be) return be - 1023 + 1;
  return b ? (63 - __clzll((long long)b)) - 1074 + 1 : kExpNone;  // subnormal: |v| = b * 2^-1074
}

// Minus the exponent of the lowest set bit of v != 0, from the bits of |v|.
__device__ __forceinline__ int neg_low_bit(uint64_t b) {
  const uint32_t lo = (uint32_t)b, hi = (uint32_t)(b >> 32);
  const int be = (int)(hi >> 20);
  const uint32_t mh = (hi & 0xFFFFFu) | (be ? 0x100000u : 0u);
  const int tz = lo ? __ffs((int)lo) - 1 : 31 + __ffs((int)mh);
  return 1075 - max(be, 1) - tz;
}

// The largest exponent and, SPAN, the lowest set bit of the entries seen.  Per
// entry the 64-bit maximum of |v| is that of its upper word (the lower words'
// union serves where all of those are zero), and where no lower word of the
// N entries is zero, as in most data, the lowest bit is in it: ten integer
// instructions instead of some twenty, which bound the scaling (ALU pipe 65 %
// busy at m = n = 4096: 56 -> 45 us).
template <bool SPAN>
struct Extent {
  uint32_t hi = 0, lo = 0;
  int nl = kExpNone;

  template <int N>
  __device__ __forceinline__ void take(const double (&v)[N]) {
    uint32_t least = 0xFFFFFFFFu;
#pragma unroll
    for (int q = 0; q < N; ++q) {
      const uint32_t l = (uint32_t)__double2loint(v[q]);
      hi = max(hi, (uint32_t)__double2hiint(v[q]) & 0x7FFFFFFFu);
      lo |= l;
      least = min(least, l);
    }
    if (!SPAN) return;
    if (least) {
#pragma unroll
      for (int q = 0; q < N; ++q) {
        const int be = (int)(((uint32_t)__double2hiint(v[q]) & 0x7FFFFFFFu) >> 20);
        nl = max(nl, 1075 - max(be, 1) - __clz((int)__brev((uint32_t)__double2loint(v[q]))));
      }
    } else {
#pragma unroll
      for (int q = 0; q < N; ++q) {
        const uint64_t b = (uint64_t)__double_as_longlong(v[q]) & 0x7FFFFFFFFFFFFFFFull;
        if (b) nl = max(nl, neg_low_bit(b));
      }
    }
  }
  __device__ __forceinline__ int exponent() const { return exp_above(((uint64_t)hi << 32) | (hi ? 0u : lo)); }
};

// ---------------------------------------------------------------- scales
// Tiles of 32 (p) x 64 (k) per 256-thread block in the slicing; the scaling
// takes the same 32 rows over a range of k.
constexpr int TP = 32, TK = 64;
static_assert(kOzBlock % TP == 0 && kOzBlock % TK == 0, "a residue tile lies in one K-range block");
constexpr int kScaleChunk = 64;  // k per step of a scaling block: eight loads in flight per thread

struct ScaleJob {
  OzOperand op;
  int *e;              // result per row
  int *pe, *pn;        // per split and row: partial maxima (splits > 1)
  int *cnt;            // per row tile: splits finished; zero between launches
  int side;            // 0: Lft, 1: Rgt
  int tiles, splits;   // row tiles; K splits of kps each
  int64_t kps, pstride;
  OzCtl *ctl;          // lossless route
  int ctl_blocks;      // row tiles of both operands
  int klog;            // 1024 log2 K, rounded up
  int *zero;
  int64_t block_begin;  // grouped launches
};

// floor(1024 log2 M) of the first n moduli's product (one less, to be safe
// from the rounding of this computation).
struct Log2Table {
  int v[kCrtModuli + 1];
};
constexpr Log2Table make_log2_table() {
  Log2Table t{};
  double m = 1.0;  // M / 2^e in [1, 2)
  int e = 0;
  for (int n = 1; n <= kCrtModuli; ++n) {
    m *= kModuli[n - 1];
    while (m >= 2.0) {
      m /= 2.0;
      ++e;
    }
    double f = m;
    int frac = 0;
    for (int i = 0; i < 10; ++i) {
      f *= f;
      frac *= 2;
      if (f >= 2.0) {
        f /= 2.0;
        ++frac;
      }
    }
    t.v[n] = 1024 * e + frac - 1;
  }
  return t;
}
__constant__ Log2Table kLog2M = make_log2_table();
// K * 2^(bits) <= 0.47 M in these units: 1024 log2(1 / 0.47), rounded up.
constexpr int kMargin = 1116;

// The route's decision from the operands' spans and lowest bits, by a warp
// (lane l looks at sets of l + 1 moduli).
__device__ __forceinline__ void decide(int span0, int span1, int nl0, int nl1, bool bad, int klog, int &go, int &n,
                                       int &b0, int &b1) {
  b0 = max(span0, 1);
  b1 = max(span1, 1);
  // Every exact result is a multiple of 2^(low0 + low1): at -1074 or above
  // none is rounded twice on its way to a subnormal.
  const bool fine = nl0 == kExpNone || nl1 == kExpNone || nl0 + nl1 <= 1074;
  const int need = 1024 * (b0 + b1) + klog + kMargin, ln = threadIdx.x & 31;
  const unsigned enough = __ballot_sync(0xffffffffu, ln >= 1 && ln < kCrtModuli && kLog2M.v[ln + 1] >= need);
  n = enough ? __ffs(enough) : kCrtModuli;
  go = !bad && fine && b0 <= kMaxBits && b1 <= kMaxBits && enough != 0;
}
static_assert(kCrtModuli == 32, "a lane per set");

// Rows [32 bx, 32 bx + 32) of the operand over k in [by kps, (by + 1) kps).
// Bound by the latency of its loads (small operands) or by HBM (large ones):
// every thread has eight loads in flight at four blocks per SM, and small
// operands are split along K until there are blocks for every SM.  m = n =
// 512: 20 -> 10.6 us, 4096: 71 -> 54 us against four loads in flight, 2048 k
// per block and no K splits (then 45 us, see Extent).
template <bool SPAN>
__device__ __forceinline__ void scale_body(const ScaleJob &J, int64_t bx, int64_t by) {
  __shared__ int red[TP], redn[TP];
  __shared__ int last;
  const OzOperand &op = J.op;
  const int tid = threadIdx.x, w = tid >> 5, ln = tid & 31;
  const int64_t p0 = bx * TP;
  const int64_t kb = by * J.kps, ke = min(op.K, kb + J.kps);
  const bool k_le_p = tri_k_le_p(op);
  const int off = op.unit ? 1 : 0;  // a unit diagonal is not read
  if (tid < TP) red[tid] = redn[tid] = kExpNone;
  __syncthreads();
  // Row p's own k range, and the range of k that any of the tile's rows has.
  auto row_range = [&](int64_t p, int64_t &lo, int64_t &hi) {
    lo = kb;
    hi = p < op.P ? ke : kb;
    if (op.tri) {
      if (k_le_p) hi = min(hi, p + 1 - off);
      else lo = max(lo, p + off);
    }
  };
  int64_t k0 = kb, k1 = ke;
  if (op.tri) {
    if (k_le_p) k1 = min(k1, p0 + TP);
    else k0 = max(k0, p0);
  }
  const bool plain = !op.tri && p0 + TP <= op.P;
  if (op.kcontig) {
    // Warp w takes rows p0 + w, p0 + w + 8, ...; its lanes stride over k.
    Extent<SPAN> x4[4];
    for (int64_t k = k0 + ln; k < k1 + ln; k += kScaleChunk) {
      double v[4][2];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int64_t p = p0 + w + 8 * r;
        const double *x = op.X + p * op.ld + k;
        if (plain && k - ln + kScaleChunk <= k1) {
#pragma unroll
          for (int q = 0; q < 2; ++q) v[r][q] = x[32 * q];
        } else {
          int64_t lo, hi;
          row_range(p, lo, hi);
#pragma unroll
          for (int q = 0; q < 2; ++q) v[r][q] = k + 32 * q >= lo && k + 32 * q < hi ? x[32 * q] : 0.0;
        }
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) x4[r].take(v[r]);
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int e = __reduce_max_sync(0xffffffffu, x4[r].exponent());
      const int n = SPAN ? __reduce_max_sync(0xffffffffu, x4[r].nl) : 0;
      if (ln == 0) {
        red[w + 8 * r] = e;
        redn[w + 8 * r] = n;
      }
    }
  } else {
    const int64_t p = p0 + ln;
    Extent<SPAN> ext;
    int64_t lo, hi;
    row_range(p, lo, hi);
    for (int64_t k = k0 + w; k < k1; k += kScaleChunk) {
      const double *x = op.X + p + k * op.ld;
      double v[8];
      if (plain && k - w + kScaleChunk <= k1) {
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = x[8 * q * op.ld];
      } else {
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = k + 8 * q >= lo && k + 8 * q < hi ? x[8 * q * op.ld] : 0.0;
      }
      ext.take(v);
    }
    const int e = ext.exponent();
    if (e != kExpNone) atomicMax(&red[ln], e);
    if (SPAN && ext.nl != kExpNone) atomicMax(&redn[ln], ext.nl);
  }
  __syncthreads();
  const bool row = tid < TP && p0 + tid < op.P;
  // A unit diagonal's one.
  if (row && op.tri && op.unit && p0 + tid >= kb && p0 + tid < ke) {
    red[tid] = max(red[tid], 1);
    redn[tid] = max(redn[tid], 0);
  }
  int e = row ? red[tid] : kExpNone, n = row ? redn[tid] : kExpNone;
  if (J.splits > 1) {
    // The last split of this tile to arrive combines the partial maxima.
    if (row) {
      J.pe[by * J.pstride + p0 + tid] = e;
      if (SPAN) J.pn[by * J.pstride + p0 + tid] = n;
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) {
      last = atomicAdd(&J.cnt[bx], 1) == J.splits - 1;
      if (last) J.cnt[bx] = 0;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (row)
      for (int q = 0; q < J.splits; ++q) {
        e = max(e, __ldcg(&J.pe[q * J.pstride + p0 + tid]));
        if (SPAN) n = max(n, __ldcg(&J.pn[q * J.pstride + p0 + tid]));
      }
  }
  if (row) J.e[p0 + tid] = e;
  if (!SPAN || tid >= 32) return;
  const int span = __reduce_max_sync(0xffffffffu, e == kExpNone ? kExpNone : e + n);
  const int low = __reduce_max_sync(0xffffffffu, e == kExpNone ? kExpNone : n);
  const int top = __reduce_max_sync(0xffffffffu, e);
  bool all = false;
  if (tid == 0) {
    if (span != kExpNone) {
      atomicMax(&J.ctl->span[J.side], span);
      atomicMax(&J.ctl->nlow[J.side], low);
    }
    if (top > 1024) atomicOr(&J.ctl->bad, 1);  // infinity or NaN
    __threadfence();
    all = atomicAdd(&J.ctl->done, 1u) == (unsigned)J.ctl_blocks - 1;
  }
  if (!__any_sync(0xffffffffu, all)) return;
  // The last tile's warp decides.
  __threadfence();
  volatile OzCtl *c = J.ctl;
  int go, nm, b0, b1;
  decide(c->span[0], c->span[1], c->nlow[0], c->nlow[1], c->bad != 0, J.klog, go, nm, b0, b1);
  __syncwarp();
  if (tid) return;
  c->go = go;
  c->n = nm;
  c->bits[0] = b0;
  c->bits[1] = b1;
  c->span[0] = c->span[1] = c->nlow[0] = c->nlow[1] = kExpNone;
  c->bad = 0;
  c->done = 0u;
  if (J.zero) *J.zero = 0;
}

// Both operands of one call: blocks [0, tiles * splits) are Lft's.
template <bool SPAN>
__global__ void __launch_bounds__(256, 4) scale_kernel(const __grid_constant__ ScaleJob L,
                                                    const __grid_constant__ ScaleJob R) {
  chain_wait();
  const int64_t nl = (int64_t)L.tiles * L.splits;
  const int64_t b = blockIdx.x;
  if (b < nl) scale_body<SPAN>(L, b % L.tiles, b / L.tiles);
  else scale_body<SPAN>(R, (b - nl) % R.tiles, (b - nl) / R.tiles);
}

// ---------------------------------------------------------------- residues
constexpr uint32_t pow2mod(int e, uint32_t m) {
  uint32_t r = 1 % m;
  for (int i = 0; i < e; ++i) r = (r * 2) % m;
  return r;
}

// All residues go through the FP32 pipe.  The signed integer x is cut into ND
// digits d_i of W bits, balanced into [-2^(W-1), 2^(W-1)) by one added bias,
// so x is congruent to s = sum_i d_i c_i modulo m with c_i = 2^(W i) mod m
// balanced into [-m/2, m/2]: |s| <= ND 2^(W-1) 181 < 2^23, exact in fp32.
// r = s - m * rint(s / m), rounding by the 1.5 * 2^23 constant in one fma, is
// congruent to x: the quotient's error, at most |s/m| 2^-24 <= ND 2^(W-2)
// 2^-24 (0.00098 to 0.00122 for the forms below), is below
// the gap 1/(2m) >= 0.00137 between s/m and a half-integer for the odd
// moduli, and the even modulus 362 only has the tie +-181 either way, so
// |r| <= 181 as the residue GEMM's exactness bound requires.
// Balanced digits carry 14 bits where plain ones in the same bounds carry
// 11: four digits (six FP32 operations per residue) instead of six (eight).
template <int ND_, int W_>
struct Digits {
  static constexpr int ND = ND_, W = W_;
  static constexpr int kBits = ND * W - 2;  // |x| < 2^kBits, so that x plus the bias stays below 2^(ND W)
  static_assert(ND * (1 << (W - 1)) * 181 < (1 << 23), "the digit sum is exact in fp32");
  static_assert((double)ND * (1 << (W - 2)) / 16777216.0 < 0.5 / 363, "the quotient rounds to the nearest integer");
};
using Narrow = Digits<4, 14>;  // |x| < 2^54: automatic counts, and FP64 entries of one binade
using Middle = Digits<5, 14>;  // |x| < 2^68
using Wide7 = Digits<7, 13>;   // |x| < 2^89: full mantissas over a common range
using Wide8 = Digits<8, 13>;   // |x| < 2^102
using Wide = Digits<10, 13>;   // the last digit holds the 11 bits left of 128: |x| < 2^126
static_assert(kMaxBits <= 126, "the digits cover the widest integers");

// c_i for modulus m, balanced.
constexpr float digit_coeff(int bit, int m) {
  const int r = (int)pow2mod(bit, (uint32_t)m);
  return (float)(r > m / 2 ? r - m : r);
}

// Bits of digit i (the last one of Wide is cut off at bit 128).
template <class D>
constexpr int digit_width(int i) {
  return D::W * (i + 1) <= 128 ? D::W : 128 - D::W * i;
}

template <class D>
constexpr unsigned __int128 digit_bias() {
  unsigned __int128 b = 0;
  for (int i = 0; i < D::ND; ++i) b |= (unsigned __int128)1 << (D::W * i + digit_width<D>(i) - 1);
  return b;
}

// A digit of `w` bits with its bias taken off.
__device__ __forceinline__ float digit_float(uint32_t v, int w) {
  return __uint_as_float(0x4B000000u | (v & ((1u << w) - 1))) - (8388608.0f + (float)(1 << (w - 1)));
}

// Digits of the signed integer with magnitude x and sign bit `neg`.
template <class D>
__device__ __forceinline__ void digits(uint64_t x, bool neg, float (&d)[D::ND]) {
  static_assert(D::ND * D::W <= 64, "");
  const uint64_t t = (neg ? 0 - x : x) + (uint64_t)digit_bias<D>();
  const uint32_t lo = (uint32_t)t, hi = (uint32_t)(t >> 32);
#pragma unroll
  for (int i = 0; i < D::ND; ++i) {
    const int at = D::W * i;
    d[i] = digit_float(at >= 32 ? hi >> (at - 32) : at + D::W <= 32 ? lo >> at : __funnelshift_r(lo, hi, at), D::W);
  }
}
template <class D>
__device__ __forceinline__ void digits(unsigned __int128 x, bool neg, float (&d)[D::ND]) {
  const unsigned __int128 t = (neg ? 0 - x : x) + digit_bias<D>();
  const uint32_t w[5] = {(uint32_t)t, (uint32_t)(t >> 32), (uint32_t)(t >> 64), (uint32_t)(t >> 96), 0u};
#pragma unroll
  for (int i = 0; i < D::ND; ++i) {
    const int at = D::W * i;
    d[i] = digit_float(__funnelshift_r(w[at / 32], w[at / 32 + 1], at % 32), digit_width<D>(i));
  }
}

// The moduli's constants, read by a loop counter that is the same in all
// lanes: m, 1/m and the digits' coefficients of both digit widths.
struct ResidueConst {
  float m, inv, c14[4], c13[10];
};
struct ResidueTable {
  ResidueConst l[kCrtModuli];
};
constexpr ResidueTable make_residue_table() {
  ResidueTable t{};
  for (int l = 0; l < kCrtModuli; ++l) {
    const int m = kModuli[l];
    t.l[l].m = (float)m;
    t.l[l].inv = 1.0f / (float)m;
    for (int i = 0; i < 4; ++i) t.l[l].c14[i] = digit_coeff(14 * (i + 1), m);
    for (int i = 0; i < 10; ++i) t.l[l].c13[i] = digit_coeff(13 * (i + 1), m);
  }
  return t;
}
__constant__ ResidueTable kRes = make_residue_table();

// Residues of the NK entries with digits d (NK / 4 rows of four consecutive k,
// `row` apart in a plane), moduli [l0, l1), an 8-byte store per row and
// plane.  A loop, not an unrolled list of the moduli: that overran the
// instruction cache, and the constants are loaded once for all NK entries
// (m = n = 4096, both operands: 183 -> 180 us, and less code to fetch in
// short launches).
template <class D, int NK>
__device__ __forceinline__ void store_residues(const float (&d)[NK][D::ND], int l0, int l1, uint16_t *out,
                                               int64_t plane, int64_t row) {
#pragma unroll 1
  for (int l = l0; l < l1; ++l, out += plane) {
    const ResidueConst &rc = kRes.l[l];
    uint32_t r[NK];
#pragma unroll
    for (int q = 0; q < NK; ++q) {
      float s = d[q][0];
#pragma unroll
      for (int i = 1; i < D::ND; ++i) s = fmaf(d[q][i], D::W == 14 ? rc.c14[(i - 1) & 3] : rc.c13[i - 1], s);
      const float n = fmaf(s, rc.inv, 12582912.0f) - 12582912.0f;
      r[q] = __float_as_uint(fmaf(-n, rc.m, s));  // |residue| <= 181: exact in the upper 16 bits
    }
#pragma unroll
    for (int h = 0; h < NK / 4; ++h)
      *reinterpret_cast<uint2 *>(out + h * row) =
          make_uint2(__byte_perm(r[4 * h], r[4 * h + 1], 0x7632), __byte_perm(r[4 * h + 2], r[4 * h + 3], 0x7632));
  }
}

// |v| scaled to `bits` bits under its row's exponent ep: rint(|v| 2^(bits - ep)).
__device__ __forceinline__ void scaled_parts(double v, int bits, int ep, uint64_t &mant, int &s) {
  const uint64_t b = (uint64_t)__double_as_longlong(v);
  const int be = (int)((b >> 52) & 0x7FF);
  mant = (b & ((1ull << 52) - 1)) | (be ? 1ull << 52 : 0ull);
  s = max(be, 1) - 1075 + bits - ep;  // scaled integer = mant * 2^s < 2^bits
}
__device__ __forceinline__ uint64_t scaled63(double v, int bits, int ep) {
  uint64_t mant;
  int s;
  scaled_parts(v, bits, ep, mant, s);
  // bits <= 63, so s <= 10 for normal entries: shift right by 11 - s >= 1 of
  // the mantissa at the top of the word, rounding half up.  (A subnormal's
  // unnormalised mantissa may need s > 10: its upper bits are zero.)
  // (A row without nonzeros has ep = kExpNone: its shift counts mean nothing.)
  if (s > 10) return mant << (s & 63);
  const int r = 10 - s;
  const uint64_t z = (unsigned)r < 64u ? (mant << 11) >> r : 0;
  return (z >> 1) + (z & 1);
}
__device__ __forceinline__ unsigned __int128 scaled128(double v, int bits, int ep) {
  uint64_t mant;
  int s;
  scaled_parts(v, bits, ep, mant, s);
  if (s >= 0) return (unsigned __int128)mant << (s & 127);
  return s > -64 ? (mant + (1ull << (-s - 1))) >> (-s) : 0;
}

struct ResidueJob {
  OzOperand op;
  const int *e;
  int side;  // 0: Lft, 1: Rgt
  int bits, l0, l1;
  int64_t Pp, Kp, gx;
  uint16_t *R;
  const OzCtl *ctl;     // lossless route: bits and moduli count from here
  int64_t blocks;       // gx * row tiles
  int64_t block_begin;  // grouped launches
};

// x >> n, 0 for n > 63 (the instruction's own clamp: C++ leaves it undefined).
__device__ __forceinline__ uint64_t shr_clamp(uint64_t x, uint32_t n) {
  uint64_t r;
  asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(n));
  return r;
}

// Digits of rint(v 2^(bits - ep)) for |v| 2^(bits - ep) < 2^54 and no
// subnormal v: the mantissa at the top of a word, shifted down by its
// exponent's distance (zeros shift to nothing), rounded half up, given its
// sign and the bias in one addition.  `far` = 1085 - bits + ep.
template <class D>
__device__ __forceinline__ void digits_normal(double v, int far, float (&d)[D::ND]) {
  static_assert(D::ND * D::W <= 64, "");
  const uint32_t hi = (uint32_t)__double2hiint(v), lo = (uint32_t)__double2loint(v);
  const uint32_t be = (hi >> 20) & 0x7FFu;
  const uint64_t m = ((uint64_t)(__funnelshift_l(lo, hi, 11) | 0x80000000u) << 32) | (lo << 11);
  const uint64_t x = (shr_clamp(m, (uint32_t)far - be) + 1) >> 1;
  const uint32_t neg = (uint32_t)((int32_t)hi >> 31);
  const uint64_t n64 = ((uint64_t)neg << 32) | neg;
  const uint64_t t = (x ^ n64) + ((uint64_t)digit_bias<D>() + (neg & 1u));
  const uint32_t tl = (uint32_t)t, th = (uint32_t)(t >> 32);
#pragma unroll
  for (int i = 0; i < D::ND; ++i) {
    const int at = D::W * i;
    d[i] = digit_float(at >= 32 ? th >> (at - 32) : at + D::W <= 32 ? tl >> at : __funnelshift_r(tl, th, at), D::W);
  }
}

// Digits of one entry, |v| 2^(bits - ep) < 2^kBits.
template <class D>
__device__ __forceinline__ void entry_digits(double v, int bits, int ep, float (&d)[D::ND]) {
  // (Zeros, and rows of them, come out as zero: their mantissa is.)
  const bool neg = __double2hiint(v) < 0;
  if constexpr (D::ND * D::W <= 64) digits<D>(scaled63(v, bits, ep), neg, d);
  else digits<D>(scaled128(v, bits, ep), neg, d);
}

// The same for the narrow form, out of line for the rare entries that need it.
__device__ __noinline__ float4 narrow_entry(double v, int bits, int ep) {
  float d[Narrow::ND];
  entry_digits<Narrow>(v, bits, ep, d);
  return make_float4(d[0], d[1], d[2], d[3]);
}

// Digits of the thread's eight entries (two rows of four consecutive k): the
// common form (rows whose exponent keeps every entry clear of subnormals), or
// else the general one.
__device__ __forceinline__ void narrow_digits(const double (&v)[2][4], int bits, const int (&ep)[2],
                                              float (&d)[8][Narrow::ND]) {
  const int far[2] = {1085 - bits + ep[0], 1085 - bits + ep[1]};
  bool fast = far[0] >= 66 && far[1] >= 66;  // a zero (exponent field 0) then shifts out wholly
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const uint32_t h2 = (uint32_t)__double2hiint(v[q >> 2][q & 3]) << 1;
    fast = fast && (h2 >= 0x00200000u || (h2 | (uint32_t)__double2loint(v[q >> 2][q & 3])) == 0u);
  }
  if (fast) {
#pragma unroll
    for (int q = 0; q < 8; ++q) digits_normal<Narrow>(v[q >> 2][q & 3], far[q >> 2], d[q]);
  } else {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const float4 f = narrow_entry(v[q >> 2][q & 3], bits, ep[q >> 2]);
      d[q][0] = f.x;
      d[q][1] = f.y;
      d[q][2] = f.z;
      d[q][3] = f.w;
    }
  }
}

// Wider integers: a row of four at a time.
template <class D>
__device__ __forceinline__ void wide_rows(const double (&v)[2][4], int bits, const int (&ep)[2], int l0, int l1,
                                          uint16_t *R, int64_t plane, int64_t half) {
#pragma unroll 1
  for (int h = 0; h < 2; ++h) {
    float d[4][D::ND];
#pragma unroll
    for (int q = 0; q < 4; ++q) entry_digits<D>(h ? v[1][q] : v[0][q], bits, h ? ep[1] : ep[0], d[q]);
    store_residues<D, 4>(d, l0, l1, R + h * half, plane, half);
  }
}

// Residues of the thread's eight entries (rows `half` apart in a plane) by the
// fewest digits that hold their bits.
__device__ __forceinline__ void slice_rows(const double (&v)[2][4], int bits, const int (&ep)[2], int l0, int l1,
                                           uint16_t *R, int64_t plane, int64_t half) {
  if (bits <= Narrow::kBits) {
    float d[8][Narrow::ND];
    narrow_digits(v, bits, ep, d);
    store_residues<Narrow, 8>(d, l0, l1, R, plane, half);
  } else if (bits <= Middle::kBits) {
    float d[8][Middle::ND];
#pragma unroll
    for (int q = 0; q < 8; ++q) entry_digits<Middle>(v[q >> 2][q & 3], bits, ep[q >> 2], d[q]);
    store_residues<Middle, 8>(d, l0, l1, R, plane, half);
  } else if (bits <= Wide7::kBits) {
    wide_rows<Wide7>(v, bits, ep, l0, l1, R, plane, half);
  } else if (bits <= Wide8::kBits) {
    wide_rows<Wide8>(v, bits, ep, l0, l1, R, plane, half);
  } else {
    wide_rows<Wide>(v, bits, ep, l0, l1, R, plane, half);
  }
}

// The 32 (p) x 64 (k) residue tile (bx = k tile, by = p tile).
__device__ __forceinline__ void residue_body(const ResidueJob &J, int64_t bx, int64_t by) {
  __shared__ double tile[TP][TK + 1];
  const OzOperand &op = J.op;
  const int tid = threadIdx.x;
  const int64_t p0 = by * TP, k0 = bx * TK;
  if (op.tri) {
    // The residue GEMM never reads this tile when its K slab is outside the
    // range of the kOzBlock-row block holding it (see kOzBlock).
    const int64_t b = p0 / kOzBlock * kOzBlock;
    if (tri_k_le_p(op) ? k0 >= b + kOzBlock : k0 + TK <= b) return;
  }
  // Each thread takes four consecutive k of rows tid/16 and tid/16 + 16; the
  // eight loads of all threads are in flight together.
  const int64_t plane = J.Pp * J.Kp;
  const int pa = tid >> 4, kk0 = (tid & 15) * 4;
  const int ep[2] = {J.e[p0 + pa], J.e[p0 + pa + TP / 2]};
  // Entries that need no test: a tile inside the matrix and off the diagonal.
  const bool inside = p0 + TP <= op.P && k0 + TK <= op.K &&
                      (!op.tri || (tri_k_le_p(op) ? k0 + TK <= p0 : k0 >= p0 + TP));
  double v[2][4];
  if (op.kcontig) {
    if (inside) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const double *x = op.X + (p0 + pa + h * (TP / 2)) * op.ld + k0 + kk0;
#pragma unroll
        for (int q = 0; q < 4; ++q) v[h][q] = x[q];
      }
    } else {
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int q = 0; q < 4; ++q) v[h][q] = load_elem(op, p0 + pa + h * (TP / 2), k0 + kk0 + q);
    }
  } else {
    const int pp = tid & 31, kk = tid >> 5;
    double t[8];
    if (inside) {
      const double *x = op.X + p0 + pp + (k0 + kk) * op.ld;
#pragma unroll
      for (int q = 0; q < 8; ++q) t[q] = x[8 * q * op.ld];
    } else {
#pragma unroll
      for (int q = 0; q < 8; ++q) t[q] = load_elem(op, p0 + pp, k0 + kk + 8 * q);
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) tile[pp][kk + 8 * q] = t[q];
    __syncthreads();
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int q = 0; q < 4; ++q) v[h][q] = tile[pa + h * (TP / 2)][kk0 + q];
  }
  const int l0 = J.l0;
  int bits = J.bits, l1 = J.l1;
  if (J.ctl) {
    if (!J.ctl->go) return;
    bits = J.ctl->bits[J.side];
    l1 = min(l1, J.ctl->n);
    if (l1 <= l0) return;
  }
  // The same in every lane, and known to be: bounds and plane addresses of
  // the loop over the moduli then run on the uniform datapath.
  bits = __reduce_max_sync(0xffffffffu, bits);
  l1 = __reduce_max_sync(0xffffffffu, l1);
  slice_rows(v, bits, ep, l0, l1, J.R + (p0 + pa) * J.Kp + k0 + kk0, plane, (TP / 2) * J.Kp);
}

// Bound by the planes' writes: a plain fill of HBM runs at 4.0 TB/s (a copy at
// 6.8), and m = n = 4096 writes 0.65 GB, 16384 x 256 4.3 GB in 1.1 ms (where the
// planes fit L2, instruction issue bounds it: six FP32 instructions and a
// quarter of a store per residue).  Eight entries per thread, whose loads are
// in flight together, at three blocks per SM (78 registers): 262 -> 172 us for
// both operands of m = n = 4096 against four entries, six digits and the list
// of moduli unrolled.  Packed fp32 halves the issue slots and changes nothing.
// LATER: a pass other than the first, whose blocks take several tiles.
template <bool LATER>
__global__ void __launch_bounds__(256, 3) residue_kernel(const __grid_constant__ ResidueJob L,
                                                         const __grid_constant__ ResidueJob R) {
  chain_wait();
  // A pass over further moduli than the operands need.  (The first pass reads
  // the decision behind the operands' loads, not ahead of them.)
  if (LATER && L.ctl && (!L.ctl->go || L.l0 >= L.ctl->n)) return;
  int64_t b = blockIdx.x;
  do {
    if (b < L.blocks) residue_body(L, b % L.gx, b / L.gx);
    else residue_body(R, (b - L.blocks) % R.gx, (b - L.blocks) / R.gx);
    b += gridDim.x;
    if (LATER) __syncthreads();  // (the tile in shared memory)
  } while (LATER && b < L.blocks + R.blocks);
}

// ---------------------------------------------------------------- scales and residues at once
// Small operands: a block holds eight whole rows in shared memory, finds their
// scales and, once all blocks have (SPAN: the decision needs every row), cuts
// them into residues.  That reads the operands once and takes one launch and
// one exchange between all blocks (which are resident together: a cooperative
// launch) where the two kernels take a second round of loads and a chain of
// partial maxima and counters.  Latency bounds both: 512 x 512 takes 14 us
// instead of 9 + 10 (calls: 38.2 -> 35.4 us; 300 x 300 37.1 -> 32.6, emulated
// tier 512 x 512 30.3 -> 23.5, which needs no exchange).
constexpr int FR = 8;    // rows per block
constexpr int NT = 512;  // threads; 16 warps have an SM's slicing well in flight
// Polls of the wait for the other blocks, as of every wait here: blocks whose
// SM another stream's long kernel still holds start that much later.
constexpr uint32_t kFusedSpin = kSpinLimit;
constexpr unsigned kLostBlock = 1u << 16;  // OzCtl::done counts blocks below this, blocks whose wait ran out above
static_assert(kFusedSlots < (int)kLostBlock, "");

struct FusedJob {
  ScaleJob L, R;  // tiles: blocks of FR rows
  ResidueJob rL, rR;
  unsigned long long *slots;  // one word per block
  int *status;
  unsigned expiry_polls;  // tests: the last block first waits this long for a word that nothing writes
};

// What a block tells the others: the launch's number, whether its rows hold a
// non-finite entry, their lowest bit and their span (0: all zeros).
__device__ __forceinline__ unsigned long long slot_word(unsigned gen, int span, int low, bool bad) {
  const unsigned v = span == kExpNone ? 0u : ((unsigned)(low + 1024) << 12) | (unsigned)span;
  return ((unsigned long long)gen << 32) | (bad ? 0x80000000u : 0u) | v;
}

template <bool SPAN>
__global__ void __launch_bounds__(NT, 1) fused_kernel(const __grid_constant__ FusedJob F) {
  extern __shared__ __align__(16) double rows[];  // [FR][ld], k from kb on
  __shared__ int red[FR], redn[FR], all[6], dec[4];  // (all[5]: a wait of this block ran out)
  __shared__ unsigned gen;  // this launch's number
  unsigned arrived = 0;
  chain_wait();
  const int nleft = F.L.tiles, nblocks = nleft + F.R.tiles;
  const bool left = (int)blockIdx.x < nleft;
  const ScaleJob &S = left ? F.L : F.R;
  const ResidueJob &J = left ? F.rL : F.rR;
  const OzOperand &op = J.op;
  const int tid = threadIdx.x, w = tid >> 5, ln = tid & 31;
  const int b = (int)blockIdx.x - (left ? 0 : nleft);
  const int64_t p0 = (int64_t)b * FR;
  const int K = (int)op.K, Kp = (int)J.Kp, ld = Kp + 2;
  const bool k_le_p = tri_k_le_p(op);
  // The k that the residue GEMM reads of these rows (see kOzBlock).
  int kb = 0, ke = Kp;
  if (op.tri) {
    const int blk = (int)(p0 / kOzBlock) * kOzBlock;
    if (k_le_p) ke = min(ke, blk + kOzBlock);
    else kb = blk;
  }
  if (tid < FR) red[tid] = redn[tid] = kExpNone;
  if (SPAN && tid < 6) all[tid] = tid < 4 ? kExpNone : 0;
  if (SPAN && tid == 0) gen = *(volatile unsigned *)&S.ctl->gen + 1;
  {
    // All of the rows' loads are in flight at once; a warp reads along k, or
    // eight rows by four k.  Nothing outside the triangle is read.
    const int pp = op.kcontig ? w / (NT / 256) : ln & 7;
    const int k1 = op.kcontig ? 32 * (w % (NT / 256)) + ln : 4 * w + (ln >> 3);
    const int64_t p = p0 + pp;
    int lo = 0, hi = p < op.P ? K : 0;
    if (op.tri) {
      if (k_le_p) hi = min(hi, (int)p + (op.unit ? 0 : 1));
      else lo = (int)p + (op.unit ? 1 : 0);
    }
    const double *x = op.X + (op.kcontig ? p * op.ld + kb + k1 : p + (kb + k1) * op.ld);
    const int64_t step = op.kcontig ? NT / 8 : NT / 8 * op.ld;
    uint32_t dst = smem_u32(rows + pp * ld + k1);
    for (int k = kb + k1; k < ke; k += NT / 8, x += step, dst += NT) {
      const bool in = k >= lo && k < hi;
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(in ? x : op.X), "r"(in ? 8 : 0)
                   : "memory");
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  }
  __syncthreads();
  {
    const int r = w / (NT / 256);
    Extent<SPAN> ext;
    double *x = rows + r * ld;
#pragma unroll 4
    for (int k = kb + 32 * (w % (NT / 256)) + ln; k < ke; k += NT / 8) {
      double v[1] = {x[k - kb]};
      if (op.tri && op.unit && k == p0 + r && k < K) x[k - kb] = v[0] = 1.0;
      ext.take(v);
    }
    const int e = __reduce_max_sync(0xffffffffu, ext.exponent());
    const int nl = SPAN ? __reduce_max_sync(0xffffffffu, ext.nl) : 0;
    if (ln == 0) {
      atomicMax(&red[r], e);
      if (SPAN) atomicMax(&redn[r], nl);
    }
  }
  __syncthreads();
  if (tid < FR && p0 + tid < op.P) S.e[p0 + tid] = red[tid];
  if (SPAN) {
    if (w == 0) {
      const int e = ln < FR ? red[ln] : kExpNone, n = ln < FR ? redn[ln] : kExpNone;
      const int span = __reduce_max_sync(0xffffffffu, e == kExpNone ? kExpNone : e + n);
      const int low = __reduce_max_sync(0xffffffffu, e == kExpNone ? kExpNone : n);
      const int top = __reduce_max_sync(0xffffffffu, e);
      if (ln == 0)
        *(volatile unsigned long long *)(F.slots + blockIdx.x) = slot_word(gen, span, low, top > 1024);
    }
    // Every block reads every block's word.
    int span[2] = {kExpNone, kExpNone}, low[2] = {kExpNone, kExpNone}, bad = 0;
    bool lost = false;
    auto word = [&](int i, uint32_t polls) {
      unsigned long long v;
      uint32_t it = 0;
      do v = *(volatile unsigned long long *)(F.slots + i);
      while ((unsigned)(v >> 32) != gen && ++it < polls);
      lost = lost || it >= polls;
      return v;
    };
    if (F.expiry_polls && (int)blockIdx.x == nblocks - 1 && tid == 0) word(kFusedSlots - 1, F.expiry_polls);
    for (int i = tid; i < nblocks; i += NT) {
      const unsigned long long v = word(i, kFusedSpin);
      const int s = (int)(v & 0xFFFu), side = i >= nleft;
      if (s) {
        span[side] = max(span[side], s);
        low[side] = max(low[side], (int)((v >> 12) & 0xFFFu) - 1024);
      }
      bad |= (int)((v >> 31) & 1u);
    }
    if (span[0] != kExpNone) atomicMax(&all[0], span[0]);
    if (span[1] != kExpNone) atomicMax(&all[1], span[1]);
    if (low[0] != kExpNone) atomicMax(&all[2], low[0]);
    if (low[1] != kExpNone) atomicMax(&all[3], low[1]);
    if (bad) atomicMax(&all[4], 1);
    if (lost) {
      record_error(F.status, KERR_WAIT_TIMEOUT);
      atomicMax(&all[5], 1);
    }
    __syncthreads();
    // The last block to get here publishes (when its last warp, which has the
    // least to cut, is done: nothing waits for this atomic): the launch's
    // number, as every block has read the one before, and the decision, a no
    // where any block's wait ran out, as that block has cut no residues.
    if (tid == NT - 32) arrived = atomicAdd(&S.ctl->done, all[5] ? kLostBlock + 1u : 1u);
    if (w == 0) {
      int go, n, b0, b1;
      decide(all[0], all[1], all[2], all[3], all[4] != 0, S.klog, go, n, b0, b1);
      if (ln == 0) {
        dec[0] = go && !all[5] ? n : 0;
        dec[1] = n;
        dec[2] = b0;
        dec[3] = b1;
      }
    }
    __syncthreads();
  }
  const int l1 = __reduce_max_sync(0xffffffffu, SPAN ? dec[0] : J.l1);
  const int bits = __reduce_max_sync(0xffffffffu, SPAN ? dec[left ? 2 : 3] : J.bits);
  if (l1 == 0) ke = kb;
  const int64_t plane = J.Pp * J.Kp;
  const int r = tid / (NT / 4);
  int ep[2] = {red[r], red[r + FR / 2]};
  ep[0] = ep[0] == kExpNone ? 0 : ep[0];  // (rows of zeros then take the common form)
  ep[1] = ep[1] == kExpNone ? 0 : ep[1];
  for (int k = kb + 4 * (tid % (NT / 4)); k < ke; k += NT) {
    double v[2][4];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const double2 *x = reinterpret_cast<const double2 *>(rows + (r + h * (FR / 2)) * ld + k - kb);
      const double2 a = x[0], c = x[1];
      v[h][0] = a.x;
      v[h][1] = a.y;
      v[h][2] = c.x;
      v[h][3] = c.y;
    }
    slice_rows(v, bits, ep, 0, l1, J.R + (p0 + r) * J.Kp + k, plane, (FR / 2) * J.Kp);
  }
  if (SPAN && tid == NT - 32 && (arrived & (kLostBlock - 1)) == (unsigned)nblocks - 1) {
    const bool whole = arrived < kLostBlock;
    S.ctl->go = dec[0] != 0 && whole;
    S.ctl->n = dec[1];
    S.ctl->bits[0] = dec[2];
    S.ctl->bits[1] = dec[3];
    S.ctl->gen = gen;
    S.ctl->done = 0u;
    if (S.zero) *S.zero = 0;
  }
}

// ---------------------------------------------------------------- reassembly
// The residue GEMM stores y_l + 256 with y_l a balanced residue of u_l C'
// modulo m_l, so with P_l = M/m_l the sum S = sum_l (y_l + 256) P_l + c, c =
// -256 sum_l P_l mod M, is congruent to C' modulo M; every term is positive
// and S/M < 64.  With |C'| <= K 2^(bits) <= 0.47 M, C' = S - k M for
// k = rint(S/M), and any estimate of S/M within 0.03 gives that k.  C' is
// formed in L 32-bit limbs (least significant first) in two's complement,
// M < 2^(32L), so limbs above L never matter.
constexpr int kLimbs = 9;  // L for 32 moduli (M < 2^263)
// Three residues are joined before the wide sums: with m_a m_b m_c = m,
// y_a (M/m_a) + y_b (M/m_b) + y_c (M/m_c) = t (M/m) for t = y_a m_b m_c +
// y_b m_a m_c + y_c m_a m_b < 3 * 439 * 363^2 < 2^28, so a 15-modulus element
// of four limbs takes 20 wide multiply-adds instead of 60.
constexpr int kGroups = (kCrtModuli + 2) / 3;
constexpr int kLimbRow = (kLimbs + 3) / 4 * 4;

// One CRT set: the weights of the residues in their groups, P_g = M/m of
// every group, -M, the limb count L (smallest >= 2 with M < 2^(32L)), and
// the k estimate's shift and scale: S >> (32(L-2) + 14 + shift), at most 2^23,
// times `scale` is S/M.
struct alignas(16) CrtSet {
  uint32_t w[kGroups][4];             // (16-byte rows: one shared load each)
  uint32_t P[kGroups][kLimbRow];
  uint32_t Mneg[kLimbRow];  // 2^(32L) - M in L limbs
  uint32_t c[kLimbRow];     // -256 sum_l P_l mod M
  float scale;
  int shift;
  int limbs, groups;
  int up;  // M, P and c are multiplied by 2^up (sets below 2^32)
};
struct CrtTable {
  CrtSet s[kCrtModuli + 1];
};
constexpr CrtTable make_crt_table() {
  CrtTable t{};
  for (int n = 2; n <= kCrtModuli; ++n) {
    CrtSet &s = t.s[n];
    uint32_t w[kLimbs] = {1};
    for (int l = 0; l < n; ++l) {
      uint64_t c = 0;
      for (int i = 0; i < kLimbs; ++i) {
        c += (uint64_t)w[i] * (uint32_t)kModuli[l];
        w[i] = (uint32_t)c;
        c >>= 32;
      }
    }
    int top = 0;
    for (int i = 0; i < kLimbs; ++i)
      if (w[i]) top = i;
    if (top == 0) {  // everything one limb up: the k estimate wants a limb below the top one
      w[1] = w[0];
      w[0] = 0;
      top = 1;
      s.up = 32;
    }
    s.limbs = top + 1;
    uint64_t c = 1;
    for (int i = 0; i < s.limbs; ++i) {
      c += (uint32_t)~w[i];
      s.Mneg[i] = (uint32_t)c;
      c >>= 32;
    }
    uint32_t sum[kLimbs + 1] = {};  // sum_l 256 P_l, then M minus its residue
    s.groups = (n + 2) / 3;
    for (int g = 0; g < s.groups; ++g) {
      uint32_t m = 1;
      for (int l = 3 * g; l < 3 * g + 3 && l < n; ++l) m *= (uint32_t)kModuli[l];
      for (int l = 3 * g; l < 3 * g + 3; ++l) s.w[g][l - 3 * g] = l < n ? m / (uint32_t)kModuli[l] : 0u;
      uint64_t r = 0;
      for (int i = kLimbs - 1; i >= 0; --i) {
        r = (r << 32) | w[i];
        s.P[g][i] = (uint32_t)(r / m);
        r %= m;
      }
      const uint64_t wsum = (uint64_t)kResidueBias * (s.w[g][0] + s.w[g][1] + s.w[g][2]);
      uint64_t cy = 0;
      for (int i = 0; i <= kLimbs; ++i) {
        cy += (i < kLimbs ? wsum * s.P[g][i] : 0) + sum[i];
        sum[i] = (uint32_t)cy;
        cy >>= 32;
      }
    }
    for (bool more = true; more;) {  // sum := sum - M while that is not negative
      uint32_t d[kLimbs + 1] = {};
      int64_t bw = 0;
      for (int i = 0; i <= kLimbs; ++i) {
        bw += (int64_t)sum[i] - (i < kLimbs ? w[i] : 0u);
        d[i] = (uint32_t)bw;
        bw >>= 32;
      }
      more = bw >= 0;
      if (more)
        for (int i = 0; i <= kLimbs; ++i) sum[i] = d[i];
    }
    int64_t bw = 0;
    for (int i = 0; i < kLimbs; ++i) {
      bw += (int64_t)w[i] - sum[i];
      s.c[i] = (uint32_t)bw;
      bw >>= 32;
    }
    // M / 2^(32(L-1)) from its three top limbs, and floor(log2 M) - 32(L-1).
    const int L = s.limbs;
    double m = (double)w[L - 1] + (double)w[L - 2] / 4294967296.0;
    if (L >= 3) m += (double)w[L - 3] / 4294967296.0 / 4294967296.0;
    int lg = 0;
    while ((w[L - 1] >> lg) > 1) ++lg;
    // 16 bits of M are kept below its top one: 32 + lg - 16 above limb L - 2's
    // unit are dropped, 14 of them first.
    s.shift = lg + 2;
    double unit = 1.0;  // 2^(14 + shift - 32) in units of limb L - 1
    for (int i = 0; i < 18 - s.shift; ++i) unit /= 2.0;
    for (int i = 0; i < s.shift - 18; ++i) unit *= 2.0;
    s.scale = (float)(unit / m);
  }
  return t;
}
__constant__ CrtTable kCrt = make_crt_table();
// What the k estimate leaves out of S is inside the 0.03: the limb sums
// below its two (each under groups * 3 * 439 * 363^2 * 2^32) are under M / 50,
// and the two shifts drop less than two units, M / 2^15.
constexpr bool estimate_holds() {
  const CrtTable t = make_crt_table();
  for (int n = 2; n <= kCrtModuli; ++n) {
    // 2^(32(L-2)) / M: the unit is 2^(14 + shift) of limb L - 2's.
    double below = t.s[n].scale;
    for (int i = 0; i < 14 + t.s[n].shift; ++i) below /= 2.0;
    if (t.s[n].limbs >= 3 && 1.001 * t.s[n].groups * 3 * 439 * 363 * 363 * below > 0.02) return false;
    if (t.s[n].scale * 8388608.0 < 64.0) return false;  // S/M < 64 stays below 2^23 units
  }
  return true;
}
static_assert(estimate_holds(), "the k estimate ignores too much");
// The (groups, limbs) pairs that crt_body unrolls are all there are.
constexpr bool kinds_covered() {
  const CrtTable t = make_crt_table();
  const int kinds[][2] = {{1, 2}, {2, 2}, {3, 2}, {3, 3}, {4, 3}, {4, 4},  {5, 4},  {6, 5},
                          {7, 5}, {7, 6}, {8, 6}, {8, 7}, {9, 7}, {10, 8}, {11, 8}, {11, 9}};
  for (int n = 2; n <= kCrtModuli; ++n) {
    bool found = false;
    for (const auto &k : kinds) found = found || (t.s[n].groups == k[0] && t.s[n].limbs == k[1]);
    if (!found) return false;
  }
  return true;
}
static_assert(kinds_covered(), "a CRT set has no unrolled reassembly");

// The integer X (L limbs, two's complement) times 2^e_scale, rounded once
// where the result is a normal double: the general form, for results whose
// top limbs are zero, zeros, and results outside the normal range.  Out of
// line: an FP64 instruction holds its narrow pipe even where its predicate
// is off, and the rare cases' selects cost every element.
__device__ __noinline__ double crt_general(uint4 lo4, uint4 hi4, uint32_t x8, int L, int e_scale) {
  uint32_t X[9] = {lo4.x, lo4.y, lo4.z, lo4.w, hi4.x, hi4.y, hi4.z, hi4.w, x8};
  const bool neg = (X[L - 1] >> 31) != 0;
  if (neg) {
    uint32_t c = 1;
    for (int k = 0; k < L; ++k) {
      X[k] = ~X[k] + c;
      c = c && X[k] == 0u;
    }
  }
  int t = L - 1;
  while (t >= 0 && X[t] == 0u) --t;
  if (t < 0) return 0.0;
  const int lz = __clz((int)X[t]);
  const uint32_t x1 = t >= 1 ? X[t - 1] : 0u, x0 = t >= 2 ? X[t - 2] : 0u;
  uint64_t top = ((uint64_t)__funnelshift_l(x1, X[t], lz) << 32) | __funnelshift_l(x0, x1, lz);
  bool sticky = (x0 << lz) != 0u;
  for (int k = 0; k < t - 2; ++k) sticky = sticky || X[k];
  top |= sticky ? 1ull : 0ull;
  const int k2 = 32 * (t - 1) - lz + e_scale;  // top * 2^k2
  uint64_t m = top >> 11;
  const uint32_t rem = (uint32_t)top & 0x7FFu;
  if (rem + ((uint32_t)m & 1u) > 0x400u) ++m;
  const int e = k2 + 63 + 1023;  // biased exponent of the leading bit
  double d;
  if (e + (int)(m >> 53) >= 1 && e + (int)(m >> 53) <= 2046)
    d = __longlong_as_double((long long)(((uint64_t)(uint32_t)(e - 1) << 52) + m));
  else
    d = ldexp(__ull2double_rn(top), k2);
  return neg ? -d : d;
}

// L limbs of a table row, by 16-byte shared loads.
template <int L>
__device__ __forceinline__ void limb_row(const uint32_t (&row)[kLimbRow], uint32_t (&x)[L]) {
#pragma unroll
  for (int k = 0; k < L; k += 4) {
    const uint4 q = *reinterpret_cast<const uint4 *>(&row[k]);
    x[k] = q.x;
    if (k + 1 < L) x[k + 1 < L ? k + 1 : 0] = q.y;
    if (k + 2 < L) x[k + 2 < L ? k + 2 : 0] = q.z;
    if (k + 3 < L) x[k + 3 < L ? k + 3 : 0] = q.w;
  }
}

// One C value (before alpha) from its limb sums.
template <int L>
__device__ __forceinline__ double crt_value(const CrtSet &cc, const uint64_t (&acc)[L], int e_scale) {
  // k = rint(S/M) from the two top limb sums (see estimate_holds), by fp32
  // additions of 2^23 instead of conversions: those of 64-bit integers run on
  // the narrow FP64 pipe.
  const uint64_t z = ((acc[L - 2] >> 14) + (acc[L - 1] << 18)) >> cc.shift;
  const float u = __uint_as_float(0x4B000000u | (uint32_t)z) - 8388608.0f;
  const uint32_t kq = __float_as_uint(fmaf(u, cc.scale, 8388608.0f)) & 0x7FFFFFu;
  // X = S + k (-M) in two's complement, then sign and magnitude.
  uint32_t X[L], Mneg[L];
  limb_row<L>(cc.Mneg, Mneg);
  uint64_t c = 0;
#pragma unroll
  for (int k = 0; k < L; ++k) {
    c = acc[k] + (uint64_t)kq * Mneg[k] + (c >> 32);
    X[k] = (uint32_t)c;
  }
  if constexpr (L >= 4) {
    // |X| = X, or ~X + 1: a window of three limbs from the top nonzero one on
    // (the top or the next), the limbs under it only saying whether the + 1
    // reaches it and whether anything is left under it.
    const uint32_t neg = (uint32_t)((int32_t)X[L - 1] >> 31);
    uint32_t low = 0;
#pragma unroll
    for (int k = 0; k < L - 4; ++k) low |= X[k];
    uint32_t w2 = X[L - 1] ^ neg, w1 = X[L - 2] ^ neg, w0 = X[L - 3] ^ neg;
    const bool down = w2 == 0u;
    w2 = down ? w1 : w2;
    w1 = down ? w0 : w1;
    w0 = down ? X[L - 4] ^ neg : w0;
    low = down ? low : low | X[L - 4];
    if (w2 + 1u > 1u) {  // neither zero nor all ones
      uint64_t t = (uint64_t)w0 + (low == 0u ? neg & 1u : 0u);
      w0 = (uint32_t)t;
      t = (uint64_t)w1 + (t >> 32);
      w1 = (uint32_t)t;
      w2 += (uint32_t)(t >> 32);
      // The 64 bits from the leading one on, the lowest a sticky bit, rounded
      // to 53 (ties to even); a carry out of them is the next power of two,
      // and adding the mantissa to the exponent field does that.
      const int lz = __clz((int)w2);
      const uint32_t th = __funnelshift_l(w1, w2, lz);
      const uint32_t tl = __funnelshift_l(w0, w1, lz) | ((low | (w0 << lz)) ? 1u : 0u);
      uint64_t m = (((uint64_t)th << 32) | tl) >> 11;
      m += (tl & 0x7FFu) + ((uint32_t)m & 1u) > 0x400u ? 1u : 0u;
      const int e = (down ? 32 * (L - 3) : 32 * (L - 2)) - lz + e_scale + 63 + 1022;  // biased exponent - 1
      if ((unsigned)e < 2045u)
        return __hiloint2double((int)((((uint32_t)e << 20) + (uint32_t)(m >> 32)) | (neg & 0x80000000u)),
                                (int)(uint32_t)m);
    }
  }
  const auto x = [&](int k) { return k < L ? X[k < L ? k : 0] : 0u; };
  return crt_general(make_uint4(x(0), x(1), x(2), x(3)), make_uint4(x(4), x(5), x(6), x(7)), x(8), L, e_scale);
}

// One row of two consecutive columns per thread: one 4-byte load per residue
// plane.  A block takes `chunks` runs of 256 such outputs, so that the
// decision word, the CRT set (staged in shared memory: its index is not known
// to be uniform) and the block's start are paid once for several, and a
// thread's planes are in flight together.  Bound by instruction issue and by
// HBM alike (2 B per modulus and column in, 8 B out): 267 -> 153 us at m = n =
// 4096 (62 % of the copy rate), with no FP64-pipe instruction on the common
// path, the loops unrolled for the set's size, and four blocks per SM (64
// registers, a few spilled: 170 -> 153 us against three).
struct CrtJob {
  const uint16_t *res;
  int64_t Mp, plane, M, N;
  const int *e_row, *e_col;
  int n, bits2;        // moduli, bits of both operands together
  double alpha, beta;
  int scaled;           // not (alpha == 1, beta == 0)
  double *C;
  int64_t ldc;
  const OzCtl *ctl;     // lossless route: n and bits2 from here
  double *stage;        // where the route did not compute C, a copy of it goes here (null: none)
  int64_t lds;
  int chunks;
  int64_t blocks;       // chunks * 256 outputs (rows of column pairs) each
  int64_t block_begin;  // grouped launches
};

// v := alpha * v + beta * c (two columns, ldc apart).  Out of line: a
// predicated-off FP64 instruction still holds the narrow FP64 pipe.
__device__ __noinline__ double2 scale_pair(double2 v, double alpha, double beta, const double *c, int64_t ldc,
                                           bool both) {
  v.x *= alpha;
  v.y *= alpha;
  if (beta != 0.0) {
    v.x = fma(beta, c[0], v.x);
    if (both) v.y = fma(beta, c[ldc], v.y);
  }
  return v;
}

// Row i of the columns with exponents ec (kExpNone: zero), for a CRT set of
// G groups and L limbs (both unrolled: G is 5 and L 4 for 13 to 15 moduli);
// `at`: its place in a residue plane, in bytes from `base`.  The last group's
// planes beyond n are allocated, not written, and have weight zero.
template <int L, int G>
__device__ __forceinline__ double2 crt_pair(const CrtJob &J, const CrtSet &cc, const char *base, uint32_t at,
                                            int bits2, int er, int2 ec) {
  uint64_t acc[2][L];
  {
    uint32_t c[L];
    limb_row<L>(cc.c, c);
#pragma unroll
    for (int k = 0; k < L; ++k) acc[0][k] = acc[1][k] = c[k];
  }
  const char *p = base + at;
  const int64_t step = J.plane * 2;
  constexpr int B = G <= 6 ? G : (G + 1) / 2;  // groups whose planes are in flight together
#pragma unroll
  for (int g0 = 0; g0 < G; g0 += B) {
    uint32_t w[3 * B];
#pragma unroll
    for (int u = 0; u < 3 * B; ++u, p += step)
      if (g0 + u / 3 < G) w[u] = *reinterpret_cast<const uint32_t *>(p);
#pragma unroll
    for (int h = 0; h < B; ++h) {
      if (g0 + h < G) {
        const uint4 wt = *reinterpret_cast<const uint4 *>(cc.w[g0 + h]);
        uint32_t P[L];
        limb_row<L>(cc.P[g0 + h], P);
        const uint32_t t0 =
            (w[3 * h] & 0xFFFFu) * wt.x + (w[3 * h + 1] & 0xFFFFu) * wt.y + (w[3 * h + 2] & 0xFFFFu) * wt.z;
        const uint32_t t1 = (w[3 * h] >> 16) * wt.x + (w[3 * h + 1] >> 16) * wt.y + (w[3 * h + 2] >> 16) * wt.z;
#pragma unroll
        for (int k = 0; k < L; ++k) {
          acc[0][k] += (uint64_t)t0 * P[k];
          acc[1][k] += (uint64_t)t1 * P[k];
        }
      }
    }
  }
  double2 v = make_double2(0.0, 0.0);
  if (er != kExpNone && ec.x != kExpNone) v.x = crt_value<L>(cc, acc[0], er + ec.x - bits2);
  if (er != kExpNone && ec.y != kExpNone) v.y = crt_value<L>(cc, acc[1], er + ec.y - bits2);
  return v;
}

// C to `stage`: what the FP64 kernel behind the route reads in place of an
// operand that it overwrites.
__device__ __forceinline__ void stage_outputs(const CrtJob &J) {
  for (int64_t j = blockIdx.x; j < J.N; j += gridDim.x)
    for (int64_t i = threadIdx.x; i < J.M; i += 256) J.stage[i + j * J.lds] = J.C[i + j * J.ldc];
}

// Block b of job J.
__device__ __forceinline__ void crt_body(const CrtJob &J, int64_t b) {
  __shared__ CrtSet cc;
  int n = J.n, bits2 = J.bits2;
  if (J.ctl) {
    if (!J.ctl->go) return;
    n = J.ctl->n;
    bits2 = J.ctl->bits[0] + J.ctl->bits[1];
  }
  n = __reduce_max_sync(0xffffffffu, n);  // known to be uniform: the planes' addresses are then, too
  for (int i = threadIdx.x; i < (int)(sizeof(CrtSet) / 4); i += 256)
    reinterpret_cast<uint32_t *>(&cc)[i] = reinterpret_cast<const uint32_t *>(&kCrt.s[n])[i];
  __syncthreads();
  const int64_t flat = b * J.chunks * 256;
  const int64_t p0 = flat / J.M;  // first column pair of the block
  const uint32_t per = (uint32_t)J.M;
  uint32_t g = (uint32_t)(flat - p0 * J.M) + threadIdx.x;
  const char *base = reinterpret_cast<const char *>(J.res) + p0 * J.Mp * 4;
  const int kind = __reduce_max_sync(0xffffffffu, 16 * cc.groups + cc.limbs);
  bits2 += cc.up;
#pragma unroll 1
  for (int ch = 0; ch < J.chunks; ++ch, g += 256) {
    const uint32_t dp = g / per, i = g - dp * per;
    const int64_t j = 2 * (p0 + dp);
    if (j >= J.N) return;
    const bool both = j + 1 < J.N;
    const uint32_t at = (dp * (uint32_t)J.Mp + i) * 4u;  // (a block's outputs: far under 2^32 bytes)
    const int er = J.e_row[i];
    const int2 ec = make_int2(J.e_col[j], both ? J.e_col[j + 1] : kExpNone);
    double2 v;
    switch (kind) {
#define UVT_CRT(G, L) \
  case 16 * G + L: v = crt_pair<L, G>(J, cc, base, at, bits2, er, ec); break;
      UVT_CRT(1, 2) UVT_CRT(2, 2) UVT_CRT(3, 2) UVT_CRT(3, 3) UVT_CRT(4, 3) UVT_CRT(4, 4) UVT_CRT(5, 4)
      UVT_CRT(6, 5) UVT_CRT(7, 5) UVT_CRT(7, 6) UVT_CRT(8, 6) UVT_CRT(8, 7) UVT_CRT(9, 7) UVT_CRT(10, 8)
      UVT_CRT(11, 8) UVT_CRT(11, 9)
#undef UVT_CRT
      default: v = make_double2(0.0, 0.0); break;
    }
    double *c = J.C + i + j * J.ldc;
    if (J.scaled) v = scale_pair(v, J.alpha, J.beta, c, J.ldc, both);
    c[0] = v.x;
    if (both) c[J.ldc] = v.y;
  }
}

__global__ void __launch_bounds__(256, 4) reassemble_kernel(const __grid_constant__ CrtJob J) {
  chain_wait();
  if (J.stage && !J.ctl->go) stage_outputs(J);
  else crt_body(J, blockIdx.x);
}

// ---------------------------------------------------------------- grouped (wave) kernels
// One launch per stage for all problems of a wave: block b belongs to the
// job whose [block_begin, block_begin + blocks) holds it.
template <class J>
__device__ __forceinline__ int find_job(const J *jobs, int n, int64_t b) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (jobs[mid].block_begin <= b) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

__device__ __forceinline__ int64_t flat_block() { return (int64_t)blockIdx.y * gridDim.x + blockIdx.x; }

__global__ void __launch_bounds__(256, 4) scale_wave_kernel(const ScaleJob *jobs, int n, int64_t total) {
  const int64_t b = flat_block();
  if (b >= total) return;
  const ScaleJob &J = jobs[find_job(jobs, n, b)];
  if (J.ctl) scale_body<true>(J, b - J.block_begin, 0);
  else scale_body<false>(J, b - J.block_begin, 0);
}

__global__ void __launch_bounds__(256, 3) residue_wave_kernel(const ResidueJob *jobs, int n, int64_t total) {
  const int64_t b = flat_block();
  if (b >= total) return;
  const ResidueJob &J = jobs[find_job(jobs, n, b)];
  const int64_t lb = b - J.block_begin;
  residue_body(J, lb % J.gx, lb / J.gx);
}

__global__ void __launch_bounds__(256, 4) reassemble_wave_kernel(const CrtJob *jobs, int n, int64_t total) {
  const int64_t b = flat_block();
  if (b >= total) return;
  const CrtJob &J = jobs[find_job(jobs, n, b)];
  crt_body(J, b - J.block_begin);
}

dim3 flat_grid(int64_t total) {
  const int64_t gx = std::min<int64_t>(total, 1 << 20);
  return dim3((unsigned)std::max<int64_t>(gx, 1), (unsigned)((total + gx - 1) / std::max<int64_t>(gx, 1)));
}

// log2 of the first n moduli's product.
double log2_modulus_product(int n) {
  double v = 0.0;
  for (int l = 0; l < n; ++l) v += std::log2((double)kModuli[l]);
  return v;
}

}  // namespace

int ozaki_bits(int n_moduli, int64_t K) {
  const double lm = log2_modulus_product(n_moduli);
  const double lk = std::log2((double)std::max<int64_t>(K, 1));
  int t = (int)std::floor((lm - lk - 2.0) / 2.0);
  return std::max(1, std::min(t, kMaxBits));
}

int ozaki_auto_moduli(int64_t K) {
  // 52 bits per scaled entry keep the result several times below a 1e-14
  // relative Frobenius error even for entries spread over 2^+-20 (measured:
  // 2.2e-16 at K = 32768 with 54 bits, 3.5e-15 with 50 bits).
  for (int n = 2; n <= kMaxModuli; ++n)
    if (ozaki_bits(n, K) >= 52) return n;
  return kMaxModuli;
}

namespace {
// K splits of a single call's scaling: blocks for two rounds of every SM at
// four each, but at least one chunk and at most 1024 k per split.
int64_t scale_split(int64_t tiles, int64_t K) {
  const int64_t want = (1216 + tiles - 1) / tiles;
  const int64_t kps = ((K + want - 1) / want + kScaleChunk - 1) / kScaleChunk * kScaleChunk;
  return std::max<int64_t>(kScaleChunk, std::min<int64_t>(kps, 1024));
}
}  // namespace

size_t oz_scale_bytes(int64_t Mp, int64_t Np, int64_t K) { return oz_scale_buf(nullptr, Mp, Np, K).bytes; }

OzScaleBuf oz_scale_buf(void *base, int64_t Mp, int64_t Np, int64_t K) {
  int *p = static_cast<int *>(base);
  const int64_t tiles = (Mp + Np) / TP, kps = scale_split(tiles, K);
  OzScaleBuf b;
  b.e_row = p;
  b.e_col = b.e_row + Mp;
  b.kps = kps;
  b.pstride = Mp + Np;
  b.part_e = b.e_col + Np;
  const int64_t parts = K > kps ? (K + kps - 1) / kps * (Mp + Np) : 0;
  b.part_n = b.part_e + parts;
  b.bytes = (size_t)(Mp + Np + 2 * parts) * sizeof(int);
  return b;
}

namespace {
ScaleJob scale_job(const OzOperand &op, int side, const OzScaleBuf &b, OzCtl *ctl, int64_t kps) {
  ScaleJob j;
  memset(&j, 0, sizeof(j));
  const int64_t at = side ? b.e_col - b.e_row : 0;
  j.op = op;
  j.e = b.e_row + at;
  j.pe = b.part_e + at;
  j.pn = b.part_n + at;
  j.pstride = b.pstride;
  j.side = side;
  j.tiles = (int)((op.P + TP - 1) / TP);
  j.splits = (int)((op.K + kps - 1) / kps);
  j.kps = kps;
  j.ctl = ctl;
  j.klog = (int)std::ceil(1024.0 * std::log2((double)std::max<int64_t>(op.K, 1)) + 1e-6);
  return j;
}
}  // namespace

int oz_scales(const OzOperand &L, const OzOperand &R, const OzScaleBuf &b, int *cnt, OzCtl *ctl, int *zero,
              cudaStream_t st) {
  if (L.P <= 0 || R.P <= 0 || L.K <= 0) return UVATRMM_EINVAL;
  ScaleJob jl = scale_job(L, 0, b, ctl, b.kps), jr = scale_job(R, 1, b, ctl, b.kps);
  if (jl.tiles + jr.tiles > kScaleTiles) {  // more row tiles than counters: no K splits
    jl.splits = jr.splits = 1;
    jl.kps = jr.kps = L.K;
  }
  jl.cnt = cnt;
  jr.cnt = cnt + jl.tiles;
  jl.ctl_blocks = jr.ctl_blocks = jl.tiles + jr.tiles;
  jl.zero = jr.zero = zero;
  const int64_t grid = (int64_t)jl.tiles * jl.splits + (int64_t)jr.tiles * jr.splits;
  if (grid > INT32_MAX) return UVATRMM_EINVAL;
  const cudaError_t e = launch_chained(ctl ? scale_kernel<true> : scale_kernel<false>, dim3((unsigned)grid), dim3(256),
                                       0, st, jl, jr);
  return e == cudaSuccess ? UVATRMM_OK : UVATRMM_EDEVICE;
}

namespace {
ResidueJob residue_job(const OzOperand &op, int side, const int *e, const OzPlan &plan, const OzCtl *ctl, int l0,
                       int l1, uint16_t *R) {
  ResidueJob j;
  memset(&j, 0, sizeof(j));
  j.op = op;
  j.e = e;
  j.side = side;
  j.bits = plan.bits;
  j.l0 = l0;
  j.l1 = l1;
  j.Pp = side ? plan.Np : plan.Mp;
  j.Kp = plan.Kp;
  j.gx = plan.Kp / TK;
  j.R = R;
  j.ctl = ctl;
  j.blocks = j.gx * ((op.P + TP - 1) / TP);
  return j;
}

CrtJob crt_job(const OzPlan &plan, const OzCtl *ctl, const uint16_t *res, const int *e_row, const int *e_col,
               double alpha, double beta, double *C, int64_t ldc, int64_t enough) {
  CrtJob c;
  memset(&c, 0, sizeof(c));
  c.res = res;
  c.Mp = plan.Mp;
  c.plane = plan.Mp * plan.Np;
  c.M = plan.M;
  c.N = plan.N;
  c.e_row = e_row;
  c.e_col = e_col;
  c.n = plan.n_moduli;
  c.bits2 = 2 * plan.bits;
  c.alpha = alpha;
  c.beta = beta;
  c.scaled = !(alpha == 1.0 && beta == 0.0);
  c.C = C;
  c.ldc = ldc;
  c.ctl = ctl;
  // Runs of 256 outputs per block: up to 16 once there are `enough` blocks.
  const int64_t runs = (plan.M * ((plan.N + 1) / 2) + 255) / 256;
  c.chunks = (int)std::max<int64_t>(1, std::min<int64_t>(16, runs / enough));
  c.blocks = (runs + c.chunks - 1) / c.chunks;
  return c;
}
}  // namespace

int oz_residues(const OzOperand &L, const OzOperand &R, const int *e_row, const int *e_col, const OzPlan &plan,
                const OzCtl *ctl, int l0, int l1, uint16_t *LR, uint16_t *RR, cudaStream_t st) {
  if (plan.Mp % TP || plan.Np % TP || plan.Kp % TK) return UVATRMM_EINVAL;
  const ResidueJob jl = residue_job(L, 0, e_row, plan, ctl, l0, l1, LR),
                   jr = residue_job(R, 1, e_col, plan, ctl, l0, l1, RR);
  const int64_t grid = jl.blocks + jr.blocks;
  if (grid > INT32_MAX) return UVATRMM_EINVAL;
  // A later pass often finds that its moduli are not needed: few blocks, which
  // then take several tiles each (16384 x 256: 136 us for 133120 empty ones).
  const bool later = ctl && l0 > 0;
  const cudaError_t e = launch_chained(later ? residue_kernel<true> : residue_kernel<false>,
                                       dim3((unsigned)(later ? std::min<int64_t>(grid, 8192) : grid)), dim3(256), 0,
                                       st, jl, jr);
  return e == cudaSuccess ? UVATRMM_OK : UVATRMM_EDEVICE;
}

int oz_prep_once(const OzOperand &L, const OzOperand &R, const OzScaleBuf &b, const OzPlan &plan, OzCtl *ctl, int *zero,
                 unsigned long long *slots, uint16_t *LR, uint16_t *RR, int *status, int num_sms, unsigned expiry_polls,
                 cudaStream_t st, bool *taken) {
  *taken = false;
  // A row's line is 16-byte aligned, and eight rows' lines start in different
  // banks.
  const size_t smem = (size_t)FR * (plan.Kp + 2) * sizeof(double);
  const int64_t blocks = (L.P + FR - 1) / FR + (R.P + FR - 1) / FR;
  // A block per SM; beyond these K the rows of a block are too much for one SM
  // (us, one launch / two): lossless route 512 x 512 35.4 / 38.2, 576 x 576
  // 47.3 / 45.6, 1000 x 200 45.0 / 40.4 (wide entries 68 / 61); emulated tier,
  // 20 moduli, 1000 x 200 44.0 / 46.7, 1150 x 60 52.4 / 48.1.
  constexpr int kMaxK = 1024;
  if (blocks > std::min(num_sms, kFusedSlots - 1) || plan.Kp > (ctl ? 512 : kMaxK)) return UVATRMM_OK;
  FusedJob f;
  f.L = scale_job(L, 0, b, ctl, L.K);
  f.R = scale_job(R, 1, b, ctl, R.K);
  f.L.tiles = (int)((L.P + FR - 1) / FR);
  f.R.tiles = (int)((R.P + FR - 1) / FR);
  f.L.zero = f.R.zero = zero;
  f.rL = residue_job(L, 0, b.e_row, plan, ctl, 0, plan.n_moduli, LR);
  f.rR = residue_job(R, 1, b.e_col, plan, ctl, 0, plan.n_moduli, RR);
  f.slots = slots;
  f.status = status;
  f.expiry_polls = expiry_polls;
  auto kernel = ctl ? fused_kernel<true> : fused_kernel<false>;
  if (smem > (48 << 10) && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                FR * (kMaxK + 2) * (int)sizeof(double)) != cudaSuccess) {
    cudaGetLastError();
    return UVATRMM_OK;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2] = {};
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeCooperative;
  attr[1].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = ctl ? 2 : 1;
  // (Where fewer SMs are to be had than the device has, the two kernels run.)
  if (cudaLaunchKernelEx(&cfg, kernel, f) == cudaSuccess) *taken = true;
  else cudaGetLastError();
  return UVATRMM_OK;
}

size_t oz_wave_table_bytes(int nitems) {
  auto r = [](size_t b) { return (b + 255) / 256 * 256; };
  return r(2 * (size_t)nitems * sizeof(ScaleJob)) + r(2 * (size_t)nitems * sizeof(ResidueJob)) +
         r((size_t)nitems * sizeof(CrtJob));
}

int oz_wave_tables(const OzWaveItem *items, int n, void *dev, OzWaveTables *out) {
  std::vector<char> image;
  oz_wave_image(items, n, dev, image, out);
  return cudaMemcpy(dev, image.data(), image.size(), cudaMemcpyHostToDevice) == cudaSuccess ? UVATRMM_OK
                                                                                          : UVATRMM_EDEVICE;
}

void oz_wave_image(const OzWaveItem *items, int n, void *dev, std::vector<char> &image, OzWaveTables *out) {
  std::vector<ScaleJob> sj(2 * n);
  std::vector<ResidueJob> rj(2 * n);
  std::vector<CrtJob> cj(n);
  int64_t bs = 0, br = 0, bc = 0;
  for (int i = 0; i < n; ++i) {
    const OzWaveItem &it = items[i];
    const OzPlan &pl = it.plan;
    for (int s = 0; s < 2; ++s) {
      const OzOperand &op = s ? it.R : it.L;
      ScaleJob &j = sj[2 * i + s];
      j = scale_job(op, s, it.sb, it.ctl, std::max<int64_t>(op.K, 1));
      j.block_begin = bs;
      bs += it.scaled ? 0 : j.tiles;
      ResidueJob &r = rj[2 * i + s];
      r = residue_job(op, s, j.e, pl, it.ctl, 0, pl.n_moduli, s ? it.RR : it.LR);
      r.block_begin = br;
      br += r.blocks;
    }
    sj[2 * i].ctl_blocks = sj[2 * i + 1].ctl_blocks = sj[2 * i].tiles + sj[2 * i + 1].tiles;
    cj[i] = crt_job(pl, it.ctl, it.res, it.sb.e_row, it.sb.e_col, it.alpha, 0.0, it.C, it.ldc, 64);
    cj[i].block_begin = bc;
    bc += cj[i].blocks;
  }
  auto r = [](size_t b) { return (b + 255) / 256 * 256; };
  char *base = static_cast<char *>(dev);
  out->scale = base;
  out->resid = base + r(sj.size() * sizeof(ScaleJob));
  out->crt = static_cast<char *>(out->resid) + r(rj.size() * sizeof(ResidueJob));
  out->n_scale = out->n_resid = 2 * n;
  out->n_crt = n;
  out->b_scale = bs;
  out->b_resid = br;
  out->b_crt = bc;
  image.assign(oz_wave_table_bytes(n), 0);
  memcpy(image.data(), sj.data(), sj.size() * sizeof(ScaleJob));
  memcpy(image.data() + (static_cast<char *>(out->resid) - base), rj.data(), rj.size() * sizeof(ResidueJob));
  memcpy(image.data() + (static_cast<char *>(out->crt) - base), cj.data(), cj.size() * sizeof(CrtJob));
}

int oz_wave_prep(const OzWaveTables &t, cudaStream_t st) {
  if (t.b_scale > 0)
    scale_wave_kernel<<<flat_grid(t.b_scale), 256, 0, st>>>(static_cast<const ScaleJob *>(t.scale), t.n_scale,
                                                            t.b_scale);
  if (t.b_resid > 0)
    residue_wave_kernel<<<flat_grid(t.b_resid), 256, 0, st>>>(static_cast<const ResidueJob *>(t.resid), t.n_resid,
                                                              t.b_resid);
  return cudaGetLastError() == cudaSuccess ? UVATRMM_OK : UVATRMM_EDEVICE;
}

int oz_wave_reassemble(const OzWaveTables &t, cudaStream_t st) {
  if (t.b_crt > 0) {
    reassemble_wave_kernel<<<flat_grid(t.b_crt), 256, 0, st>>>(static_cast<const CrtJob *>(t.crt), t.n_crt,
                                                               t.b_crt);
  }
  return cudaGetLastError() == cudaSuccess ? UVATRMM_OK : UVATRMM_EDEVICE;
}

int oz_reassemble(const OzPlan &plan, const OzCtl *ctl, const uint16_t *res, const int *e_row, const int *e_col,
                  double alpha, double beta, double *C, int64_t ldc, double *stage, int64_t lds, cudaStream_t st) {
  if (plan.M <= 0 || plan.N <= 0) return UVATRMM_OK;
  if (plan.n_moduli < 2 || plan.n_moduli > kCrtModuli) return UVATRMM_EINVAL;
  CrtJob j = crt_job(plan, ctl, res, e_row, e_col, alpha, beta, C, ldc, 912);
  j.stage = stage;
  j.lds = lds;
  if (j.blocks > INT32_MAX) return UVATRMM_EINVAL;
  const cudaError_t e = launch_chained(reassemble_kernel, dim3((unsigned)j.blocks), dim3(256), 0, st, j);
  return e == cudaSuccess ? UVATRMM_OK : UVATRMM_EDEVICE;
}

}  // namespace uvt
