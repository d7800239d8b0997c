// Ozaki-style split-precision FP64 TRMM on GB300's bf16 tensor cores.
//
// The emulated product C = alpha * Lft * Rgt (the same canonical GEMM view as
// the plain path, one operand triangular) is computed exactly in integers and
// rounded once:
//   1. scaling  - each row p of Lft and column p of Rgt gets a power-of-two
//      scale so its entries become integers of at most t bits
//      (Lft'[i,k] = rint(Lft[i,k] * 2^(t - e_i)), likewise Rgt');
//   2. slicing  - every integer is cut into its residues modulo N pairwise
//      coprime moduli m_l <= 363; each residue, balanced into [-181, 181],
//      is exactly representable in bf16 (integers up to 256 are);
//   3. products - for every modulus, one bf16 x bf16 -> fp32 tcgen05 GEMM of
//      the residue matrices.  Products are at most 181^2 and every K chunk
//      of 512 is reduced modulo m_l in the fp32 accumulator (in TMEM) before
//      the next (512 * 181^2 + 184 < 2^24), so every accumulated value is an
//      integer below 2^24 and the accumulation is exact.  The kernel stores
//      y_l = u_l C' mod m_l, balanced, as 16-bit words, u_l = (M/m_l)^-1 mod
//      m_l (M = prod m_l);
//   4. reassembly - the Chinese remainder theorem rebuilds C' (|C'| < M/4, or
//      at most 0.47 M on the lossless route) per element as S - k M with
//      S = sum_l y_l (M/m_l) and k = rint(S/M), which is rounded once to FP64
//      and scaled back by 2^(e_i + d_j - 2t) * alpha.
// Moduli of about 8.4 bits (rather than 8 with m_l <= 256) give the 121 bits
// that 54-bit entries need at K = 32768 with 15 products instead of 16.
// N (the slice count) sets M and hence t; see ozaki_bits().
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

namespace uvt {

constexpr int kMaxModuli = 20;  // slices a caller of the emulated tier may ask for
constexpr int kCrtModuli = 32;  // slices the lossless route of the FP64 calls may use
// The residue GEMM's 16-bit words hold balanced residues plus this.
constexpr int kResidueBias = 256;
// Pairwise coprime, largest first (greedy from 363 down): 3*11^2, 2*181, 19^2,
// 359, 5*71, 353, 349, 347, 7^3, 337, 331, 317, 313, 311, 307, 13*23, 293,
// 17^2, 283, 281, then primes.
constexpr int kModuli[kCrtModuli] = {363, 362, 361, 359, 355, 353, 349, 347, 343, 337, 331, 317, 313, 311,
                                     307, 299, 293, 289, 283, 281, 277, 271, 269, 263, 257, 251, 241, 239,
                                     233, 229, 227, 223};

// u_l = (M/m_l)^-1 mod m_l for the first n moduli, M = prod_{j<n} m_j.
constexpr int crt_u(int n, int l) {
  const int m = kModuli[l];
  int prod = 1;
  for (int j = 0; j < n; ++j)
    if (j != l) prod = prod * (kModuli[j] % m) % m;
  // Extended Euclid: prod * u = 1 (mod m).
  int r0 = m, r1 = prod, t0 = 0, t1 = 1;
  while (r1) {
    const int q = r0 / r1, r2 = r0 - q * r1, t2 = t0 - q * t1;
    r0 = r1; r1 = r2; t0 = t1; t1 = t2;
  }
  return t0 < 0 ? t0 + m : t0;
}

// Exponent that means "no nonzero entry" (memset byte 0x80).
constexpr int kExpNone = (int)0x80808080;

// The lossless route of the FP64 calls: what the scaling launch finds out
// about a problem's operands, kept on the device.  A row of Lft (a column of
// Rgt) spans from the exponent of its largest entry down to the lowest set
// bit of any entry.  With integers as wide as the widest span no bit of any
// entry is lost, so the integer product is the exact product, and reassembly
// rounds it once: no result is further from the exact one than half a unit
// in its last place.  `go` says that this holds (every entry finite, the
// spans within the largest CRT set, no subnormal result); otherwise every
// later kernel of the route returns at once and the FP64 tile kernel behind
// it computes the call.
struct OzCtl {
  int go;       // 1: the integer route computes the result
  int n;        // moduli: the fewest with K * 2^(bits[0] + bits[1]) <= 0.47 M
  int bits[2];  // bits per scaled entry of Lft, of Rgt
  // Running values of the scaling launch; its last block resets them.
  int span[2];   // widest span
  int nlow[2];   // minus the exponent of the lowest set bit
  int bad;       // a non-finite entry was seen
  unsigned done;  // row tiles (fused kernel: blocks) that have arrived
  unsigned gen;   // launches of the fused kernel so far
};
constexpr OzCtl kOzCtlInit{0, 0, {0, 0}, {kExpNone, kExpNone}, {kExpNone, kExpNone}, 0, 0u, 0u};
constexpr int kMaxBits = 126;  // what the slicing's digits hold

// Bits t kept per scaled operand entry for n moduli and inner dimension K:
// the largest t with K * 2^(2t) < M / 4.
int ozaki_bits(int n_moduli, int64_t K);
// Slice count the automatic choice uses for inner dimension K (t >= 52).
int ozaki_auto_moduli(int64_t K);

// One operand of the emulated product as the residue kernels see it:
// P[p, k] = kcontig ? X[k + p*ld] : X[p + k*ld], p < P, k < K.
// `tri` = 0: dense; 1: this operand is op(A); then the triangle test uses
// (r, c) = p_is_row ? (p, k) : (k, p).
struct OzOperand {
  const double *X;
  int64_t ld;
  int64_t P, K;
  bool kcontig;
  bool tri, p_is_row, lower, unit;
};

struct OzPlan {
  int n_moduli;       // N (the largest N of the lossless route)
  int bits;           // t (emulated tier)
  int64_t M, N, K;    // canonical GEMM sizes
  int64_t Mp, Np, Kp; // padded: Mp % 256 == 0, Np % 256 == 0, Kp % 64 == 0
};

// Padded extents of the residue planes: the residue GEMM's CTA pairs cover
// 256 rows (two 128-row tiles) x 256 columns, its K slabs are 64 wide.  The
// K range of a pair (triangular Lft) or of a column tile (triangular Rgt) is
// set per block of kOzBlock rows of the triangular operand: [0, b + 256) when
// its nonzeros lie at k <= p, [b, K) when at k >= p (b = the block's first
// row); the slicing skips the residue tiles outside it.
constexpr int kOzBlock = 256;
inline int64_t oz_pad_rows(int64_t M) { return (M + 255) / 256 * 256; }
inline int64_t oz_pad_cols(int64_t N) { return (N + 255) / 256 * 256; }
// Product residue planes to allocate for n moduli: the reassembly reads them
// by threes.
inline int64_t oz_res_planes(int n) { return (n + 2) / 3 * 3; }

// Device pieces (ozaki_prep.cu).  `ctl` is null in the emulated tier; in the
// lossless route it holds the moduli count and bits, set by the scaling.

// Exponent arrays of one problem and the scaling launch's scratch, carved
// out of one block of oz_scale_bytes() bytes: e[p] = max over k of
// (ilogb|P[p,k]| + 1) for the rows of Lft and the columns of Rgt.
struct OzScaleBuf {
  int *e_row, *e_col;     // Mp, Np entries
  int *part_e, *part_n;   // per K split: partial maxima, pstride apart
  int64_t kps, pstride;   // k per split
  size_t bytes;
};
size_t oz_scale_bytes(int64_t Mp, int64_t Np, int64_t K);
OzScaleBuf oz_scale_buf(void *base, int64_t Mp, int64_t Np, int64_t K);
// Scales of both operands, one launch.  `cnt`: kScaleTiles counters that are
// zero between launches, used by one launch at a time.  With `ctl`, also the
// spans and the route's decision; `zero` (may be null) is then set to 0.
constexpr int kScaleTiles = 16384;
int oz_scales(const OzOperand &L, const OzOperand &R, const OzScaleBuf &b, int *cnt, OzCtl *ctl, int *zero,
              cudaStream_t st);
// Residues of moduli [l0, l1) of both operands as bf16 planes
// R[l - l0][p][k] (p < Mp or Np, k < Kp), one launch.
int oz_residues(const OzOperand &L, const OzOperand &R, const int *e_row, const int *e_col, const OzPlan &plan,
                const OzCtl *ctl, int l0, int l1, uint16_t *LR, uint16_t *RR, cudaStream_t st);
// oz_scales and oz_residues (all moduli) in one launch, for operands whose rows
// fit the SMs' shared memory; `taken` says whether it was launched.  `slots`:
// kFusedSlots words, zero at first, used by one launch at a time (with `ctl`;
// the last one is never written).  Where a block's wait for the others' words
// runs out, the decision is no, so that the FP64 kernel computes the call, and
// `status` says so; `expiry_polls` (0: off) makes one block's wait run out
// after that many polls.
constexpr int kFusedSlots = 1024;
int oz_prep_once(const OzOperand &L, const OzOperand &R, const OzScaleBuf &b, const OzPlan &plan, OzCtl *ctl, int *zero,
                 unsigned long long *slots, uint16_t *LR, uint16_t *RR, int *status, int num_sms, unsigned expiry_polls,
                 cudaStream_t st, bool *taken);
// CRT reassembly of C = alpha * product + beta * C (column-major, ldc) from
// residue planes res[l][j / 2][i][j % 2] (uint16, plane stride Mp*Np).  Where
// the route's decision says no, C is copied to `stage` (unless null) instead.
int oz_reassemble(const OzPlan &plan, const OzCtl *ctl, const uint16_t *res, const int *e_row, const int *e_col,
                  double alpha, double beta, double *C, int64_t ldc, double *stage, int64_t lds, cudaStream_t st);

// Grouped slicing and reassembly for a wave of problems (one launch per
// stage): scales (each block covers all of K, so no prior fill), residue
// planes of all moduli, and the CRT reassembly into C.
struct OzWaveItem {
  OzOperand L, R;
  OzScaleBuf sb;
  OzPlan plan;
  uint16_t *LR, *RR;
  const uint16_t *res;
  double alpha;
  double *C;
  int64_t ldc;
  OzCtl *ctl = nullptr;  // lossless route (the caller uploads kOzCtlInit once)
  bool scaled = false;   // the scales are there already
};
struct OzWaveTables {
  void *scale, *resid, *crt;
  int n_scale, n_resid, n_crt;
  int64_t b_scale, b_resid, b_crt;
};
size_t oz_wave_table_bytes(int nitems);
// Builds the job tables of `n` items into device memory `dev` (synchronous copies).
int oz_wave_tables(const OzWaveItem *items, int n, void *dev, OzWaveTables *out);
// The same tables as a host image (oz_wave_table_bytes(n) bytes) that the
// caller copies to `dev`; `out` already points into `dev`.
void oz_wave_image(const OzWaveItem *items, int n, void *dev, std::vector<char> &image, OzWaveTables *out);
int oz_wave_prep(const OzWaveTables &t, cudaStream_t st);
int oz_wave_reassemble(const OzWaveTables &t, cudaStream_t st);

// The tcgen05 residue GEMM (ozaki_gemm.cu): for moduli [l0, l1), with residue
// planes LR[l-l0][i][k] (Mp x Kp) and RR[l-l0][j][k] (Np x Kp), writes
// res[l][j / 2][i][j % 2] = a balanced residue of u_l sum_k LR*RR modulo m_l,
// plus kResidueBias.  K range per output tile follows the
// triangle (tri_left: rows of Lft; else columns of Rgt).
struct OzGroupProb;
struct OzGemmLaunch {
  const uint16_t *LR, *RR;
  uint16_t *res;
  int64_t Mp, Np, Kp, M, N, K;
  int l0, l1;
  int n_moduli = 0;  // moduli of the CRT set (sets u_l of the stored residues)
  bool tri_left, tri_lower;
  bool tri_none = false;         // neither operand triangular: every tile runs all of K
  int raster_group = 0;          // major tiles per raster group (0 = default: 3, 2 from 96 tiles on)
  const OzCtl *ctl = nullptr;    // lossless route: the moduli count, on the device
  int *status;
  int num_sms;
};
int launch_oz_gemm(const OzGemmLaunch &L, cudaStream_t st, const char **why);

// One residue GEMM of a grouped launch as the device reads it (128-byte
// aligned like CUtensorMap; TMA reads the two tensor maps from global memory).
struct alignas(128) OzGroupProb {
  CUtensorMap tmA, tmB;
  int64_t Mp, Np, M, N, K;
  int l0, l1;
  int tri_left, tri_lower, tri_none, grows;
  int tiles_m, tiles_n, tiles_per_mod, group, sorted;
  uint16_t *res;
  int64_t plane;
  int tile_begin, tile_count;
  int tile_offset;  // first of the problem's own tiles this launch covers
  int nmod;         // moduli of the problem's CRT set
  const OzCtl *ctl; // lossless route: tiles of moduli from ctl->n on are skipped (all of them unless ctl->go)
};
// Fills the descriptor of one residue GEMM (tile_begin left to the caller).
int oz_group_prob(const OzGemmLaunch &L, OzGroupProb *out, const char **why);
// Sets the residue GEMM's launch attributes (call before a stream capture).
int oz_gemm_prepare();
// One persistent launch over nprob residue GEMMs (device array sorted by tile_begin).
int launch_oz_gemm_group(const OzGroupProb *dprobs, int nprob, int total_tiles, int *status, int num_sms,
                         cudaStream_t st, const char **why);

}  // namespace uvt
