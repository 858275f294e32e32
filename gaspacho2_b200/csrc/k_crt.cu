// FP64 column-pair contractions on the INT8 tensor cores: the two dominant contractions of the
// FP64 path (the Gram over cells and the gradient pairs over genes, see k_dgemm.cu) as integer
// matrix products modulo fourteen small moduli, put together by the Chinese remainder theorem. The
// method is the published "Ozaki scheme II" (Ozaki, Uchino and Imamura, 2025: emulation of a
// floating-point matrix product by an integer modular technique).
//
// C[m, n] = sum_k A[m, k] B[n, k] in FP64. Row m of A is scaled by a power of two 2^s so that its
// 2-norm is at most R = sqrt(0.48 P), P the product of the moduli (2^110.5), and rounded to integers;
// rows of B the same way. By Cauchy-Schwarz the integer sum lies within +-0.48 P, so its residues
// modulo the p_l determine it exactly: the error of the whole sum is the rounding of the operands and of
// the final value to FP64. The operands' is relative to the rows' norms: an entry is off by less than
// 2^-s, |a| / R <= 2^-s < 2 |a| / R, and by nothing on average (crt_dither), so the sum by 0.58 R units of both
// rows at most (rms; 2^-54.9 |a| |b| on average). A chain of FP64 multiply-adds (the DMMA form) rounds at every step, by
// 0.15 sqrt(K) 2^-53 sum |a_k b_k| in all (rms). Measured against extended precision, relative to the diagonal
// of the Gram (14 shapes of 1,274 to 75,034 cells, rms): 5e-17 to 7e-17, DMMA 3e-16 to 5e-15. Where the norms'
// product stands far above the sum (weights over many orders of magnitude, on other cells than a column) it
// would be the other way round: k_crt_psi, k_crt_u and k_crt_t hold the rounding against the result, and the
// DMMA kernels run for the genes or cells where it is more than theirs (crt_share).
//
//   k_crt_norm_*   2-norms of the operand rows and their scales; a row that is not finite (or whose
//                  norm leaves the range where the scaling is exact) goes the same way: a gene or a cell by
//                  itself, all of them for a pair of columns.
//   k_crt_balance  powers of two per gene that bring the gradient's operands to a like size.
//   k_crt_conv_*   operand rows -> one INT8 plane per modulus (symmetric residues), K contiguous:
//                  the scaled integer in four signed 16-bit limbs, each residue as an FP32 dot
//                  product of the limbs with 2^(16 l) mod p (exact below 2^24), reduced by one
//                  rounded multiple of p. Bound: about 120 FP32 instructions per entry.
//   k_crt_gemm     per modulus, tcgen05.mma kind::i8 on CTA pairs (256 x 256 tiles, INT32
//                  accumulators in TMEM, TMA operands), residues out as bytes. Persistent.
//   k_crt_psi      residues -> integers -> FP64, into every gene's Psi_j.
//   k_crt_u        residues of a cell's pair row -> V in shared memory -> U_i = sum_b D_ib V[i, ab].
//   k_crt_t        residues -> Z^T diag(W/Omega) g of the genotype columns.
//
// The operands of all moduli take 14 bytes per entry in place of 8, so the cells are taken in
// ranges that fit the buffer the DMMA form uses for its pair products (at most 8 GiB).
#include <algorithm>
#include <cmath>
#include <vector>

#include "gpl_internal.cuh"
#include "pair_rows.cuh"
#include "tc_common.cuh"

namespace gpl {

using namespace tc;

// ---------------------------------------------------------------------------------------------
// Moduli: pairwise coprime, at most 256. A symmetric residue is formed with a quotient that is off by
// at most 0.502, so |r| <= 0.502 p fits INT8 for p <= 253; modulo 256 INT8 wraps to the right class.
// ---------------------------------------------------------------------------------------------
namespace {
constexpr int kMod = 14;
constexpr int kModuli[kMod] = {256, 253, 251, 249, 247, 245, 241, 239, 233, 229, 227, 223, 211, 199};
constexpr int kMaxK = 130048;  // |sum of products of residues| <= K 2^14 stays below 2^31 - 256
constexpr int kTile = 256;     // output tile (rows and columns) of a CTA pair
constexpr int kChunk = 128;    // K entries (bytes) per stage
constexpr int kStagesI8 = 6;   // 32 KB of operands per CTA and stage
constexpr int kOperand = 128 * kChunk;
constexpr int kThreadsI8 = 192;

typedef unsigned __int128 u128;

struct CrtConst {
  float ca[kMod][4], cb[kMod][4];  // 2^(16 l) y mod p and 2^(16 l) mod p, symmetric
  float p[kMod], ip[kMod];
  uint32_t pu[kMod], off[kMod], magic[kMod];  // INT32 -> byte: (x + off) mod p by a multiply-high
  uint32_t fr[5][kMod / 2];  // 1 / p_l to 80 bits in 16-bit digits (lowest first), two moduli per word
};

constexpr u128 product() {
  u128 v = 1;
  for (int l = 0; l < kMod; l++) v *= (u128)kModuli[l];
  return v;
}

constexpr CrtConst make_const() {
  CrtConst c{};
  const u128 P = product();
  for (int l = 0; l < kMod; l++) {
    const int p = kModuli[l];
    const u128 part = P / (u128)p;
    const int pm = (int)(part % (u128)p);
    int y = 1;
    while ((pm * y) % p != 1) y++;
    int w = 1;  // 2^(16 l4) mod p
    for (int q = 0; q < 4; q++) {
      int b = w, a = (w * y) % p;
      if (2 * b > p) b -= p;
      if (2 * a > p) a -= p;
      c.cb[l][q] = (float)b;
      c.ca[l][q] = (float)a;
      w = (int)(((long long)w * 65536) % p);
    }
    c.p[l] = (float)p;
    c.ip[l] = 1.0f / (float)p;
    c.pu[l] = (uint32_t)p;
    c.off[l] = (uint32_t)(((2147483648ull + p - 1) / p) * p);
    c.magic[l] = (uint32_t)((1ull << 39) / (unsigned long long)p);
    const u128 f = (((u128)1 << 80) + p / 2) / (u128)p;
    for (int k = 0; k < 5; k++) c.fr[k][l / 2] |= (uint32_t)((f >> (16 * k)) & 0xffff) << (16 * (l & 1));
  }
  return c;
}

// P = 2^110.5 as a double, and the value of one unit of the 64-bit fraction of P
constexpr double kProduct = (double)(uint64_t)(product() >> 64) * 18446744073709551616.0 + (double)(uint64_t)product();
constexpr double kUnit = kProduct / 18446744073709551616.0;
}  // namespace

__constant__ CrtConst crt = make_const();

// R: the largest 2-norm of a scaled row
static double crt_norm_limit() {
  return std::sqrt(0.48 * kProduct);
}

// The scale of a row from its squared norm: 2^s with norm 2^s <= R, and 2^-s. Rows below 1e-145 are
// taken as zeros; false for a norm that is not finite or beyond 1e100 (the row's residues are then
// those of no number in particular, and so is its product).
__device__ __forceinline__ bool crt_scale(double n2, double R, double* sc, double* inv) {
  if (!(n2 < 1e200)) {
    *sc = *inv = 0.0;
    return false;
  }
  if (n2 < 1e-290) {
    *sc = *inv = 0.0;
    return true;
  }
  const int s = ilogb(R / (sqrt(n2) * (1.0 + 1e-9)));
  *sc = ldexp(1.0, s);
  *inv = ldexp(1.0, -s);
  return true;
}

// Where a gene goes that the integer form cannot take: onto the Gram's list (CrtState::genes), once, or
// without a list into the flag of its 128 (CrtState::cols).
struct CrtGenes {
  int *state, *list;
  __device__ __forceinline__ void add(int j) const {
    if (!list) state[1 + (j >> 7)] = 1;
    else if (atomicExch(state + 2 + j, 1) == 0) list[atomicAdd(state + 1, 1)] = j;
  }
};

// ---- norms -------------------------------------------------------------------------------------
// rows with K contiguous: gene j over the cells [c0, c0 + len)
__global__ void __launch_bounds__(256) k_crt_norm_rows(const double* __restrict__ src, int64_t ld, int len, double R,
                                                       double* __restrict__ sc, double* __restrict__ inv,
                                                       CrtGenes genes) {
  __shared__ double sh[32];
  const double* r = src + (size_t)blockIdx.x * ld;
  double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
  int i = 2 * threadIdx.x;
  for (; i + 512 + 1 < len; i += 1024) {
    const double2 a = *reinterpret_cast<const double2*>(r + i);
    const double2 b = *reinterpret_cast<const double2*>(r + i + 512);
    s0 = fma(a.x, a.x, s0);
    s1 = fma(a.y, a.y, s1);
    s2 = fma(b.x, b.x, s2);
    s3 = fma(b.y, b.y, s3);
  }
  for (; i < len; i += 512) {
    s0 = fma(r[i], r[i], s0);
    if (i + 1 < len) s1 = fma(r[i + 1], r[i + 1], s1);
  }
  const double n2 = block_sum((s0 + s1) + (s2 + s3), sh);
  if (threadIdx.x == 0 && !crt_scale(n2, R, sc + blockIdx.x, inv + blockIdx.x)) genes.add(blockIdx.x);
}

// rows with K strided: src[k * ld + m] bal[k], row m over k; partial sums over K ranges, then the scales
__global__ void __launch_bounds__(256) k_crt_norm_cols(const double* __restrict__ src, int64_t ld, int M, int K,
                                                       int kper, const double* __restrict__ bal,
                                                       double* __restrict__ part) {
  const int m = blockIdx.x * 256 + threadIdx.x;
  if (m >= M) return;
  const int k0 = blockIdx.y * kper, k1 = min(K, k0 + kper);
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  int k = k0;
  for (; k + 8 <= k1; k += 8) {
    double v[8];
#pragma unroll
    for (int u = 0; u < 8; u++) v[u] = src[(size_t)(k + u) * ld + m];
#pragma unroll
    for (int u = 0; u < 8; u++) {
      v[u] *= bal[k + u];
      s[u & 3] = fma(v[u], v[u], s[u & 3]);
    }
  }
  for (; k < k1; k++) {
    const double v = src[(size_t)k * ld + m] * bal[k];
    s[0] = fma(v, v, s[0]);
  }
  part[(size_t)blockIdx.y * M + m] = (s[0] + s[1]) + (s[2] + s[3]);
}

// Pair products D_ia D_ib / Omega_i over the cells [c0, c1): 32 cells of every dense column in
// shared memory at a time, four pairs per thread, partial sums over blockIdx.y's cells.
constexpr int kNormPairs = 4;
__global__ void __launch_bounds__(256) k_crt_norm_pairs(int ldN, int n_d, int c0, int c1, int cper, int n_pairs,
                                                        const int2* __restrict__ pairs, const double* __restrict__ D,
                                                        const double* __restrict__ rOm, double* __restrict__ part) {
  extern __shared__ double ds[];  // [32][n_d + 1]: the last entry 1/Omega
  const int ld = n_d + 1;
  const int b0 = c0 + blockIdx.y * cper, b1 = min(c1, b0 + cper);
  int2 q[kNormPairs];
  double s[kNormPairs];
#pragma unroll
  for (int u = 0; u < kNormPairs; u++) {
    const int p = (blockIdx.x * kNormPairs + u) * 256 + threadIdx.x;
    q[u] = p < n_pairs ? pairs[p] : make_int2(0, 0);
    s[u] = 0.0;
  }
  for (int t0 = b0; t0 < b1; t0 += 32) {
    __syncthreads();
    for (int e = threadIdx.x; e < 32 * ld; e += 256) {
      const int a = e >> 5, r = e & 31, i = t0 + r;
      ds[r * ld + a] = i < b1 ? (a < n_d ? D[(size_t)a * ldN + i] : rOm[i]) : 0.0;
    }
    __syncthreads();
#pragma unroll 4
    for (int r = 0; r < 32; r++) {
      const double* row = ds + r * ld;
      const double ro = row[n_d];
#pragma unroll
      for (int u = 0; u < kNormPairs; u++) {
        const double v = row[q[u].x] * row[q[u].y] * ro;
        s[u] = fma(v, v, s[u]);
      }
    }
  }
#pragma unroll
  for (int u = 0; u < kNormPairs; u++) {
    const int p = (blockIdx.x * kNormPairs + u) * 256 + threadIdx.x;
    if (p < n_pairs) part[(size_t)blockIdx.y * n_pairs + p] = s[u];
  }
}

// flag[m >> shift] is raised for row m (shift 31: one flag for all rows)
__global__ void k_crt_scales(int M, int n_part, const double* __restrict__ part, double R, double* __restrict__ sc,
                             double* __restrict__ inv, int* __restrict__ flag, int shift) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= M) return;
  double s = 0.0;
  for (int k = 0; k < n_part; k++) s += part[(size_t)k * M + m];
  if (!crt_scale(s, R, sc + m, inv + m)) atomicExch(flag + (m >> shift), 1);
}

// The gradient's contraction runs over the genes, and its operands run against each other there: a gene's
// Psi_j^-1 falls as its weights grow. So each gene's row of W is multiplied by a power of two and its
// pairs by the inverse, which changes no product and brings both to a like size: half the difference of
// their mean exponents (over up to 256 cells, and over the diagonal of the dense block). Without it the
// product of the norms, which sets the rounding, stood up to 300 u above the sum of the products at gene
// means of log sd 1.2; with it at 0.4 to 3 u (u = 2^-53).
constexpr int kBalanceCells = 256;
__global__ void __launch_bounds__(256) k_crt_balance(int N, int64_t ldN, int n_d, int64_t ldp,
                                                     const double* __restrict__ W, const double* __restrict__ Sp,
                                                     double* __restrict__ bal_w, double* __restrict__ bal_s) {
  __shared__ double sh[32];
  const int j = blockIdx.x;
  const double *w = W + (size_t)j * ldN, *s = Sp + (size_t)j * ldp;
  double sum[2] = {0.0, 0.0}, num[2] = {0.0, 0.0};
  auto add = [&](int which, double v) {
    const int e = (__double2hiint(v) >> 20) & 0x7ff;
    if (e == 0 || e == 0x7ff) return;
    sum[which] += e - 1023;
    num[which] += 1.0;
  };
  const int n = min(N, kBalanceCells);
  for (int k = threadIdx.x; k < n; k += 256) add(0, w[(int)((int64_t)k * N / n)]);
  for (int a = threadIdx.x; a < n_d; a += 256) add(1, s[(int64_t)a * n_d - (int64_t)a * (a - 1) / 2]);
#pragma unroll
  for (int q = 0; q < 2; q++) {
    sum[q] = block_sum(sum[q], sh);
    num[q] = block_sum(num[q], sh);
  }
  if (threadIdx.x == 0) {
    const double d = num[0] > 0.0 && num[1] > 0.0 ? (sum[1] / num[1] - sum[0] / num[0]) / 2.0 : 0.0;
    const int e = (int)rint(fmin(fmax(d, -300.0), 300.0));
    bal_w[j] = ldexp(1.0, e);
    bal_s[j] = ldexp(1.0, -e);
  }
}

// ---- residues ------------------------------------------------------------------------------------
// Entries are rounded down after a number in [0, 1) has been added, one per contraction index k and operand,
// as if drawn at random (a multiplicative hash): an entry is off by 0.41 of a unit (rms; 0.29 rounded to
// nearest) and by nothing on average, and integers stay as they are. Rounded to nearest, a row of one value
// (1/Omega of cells that share it, equal weights) is off by the same fraction everywhere, and its sums by
// that: up to 103 u at 100,000 cells, where an entry has 46 bits and a chain of FP64 additions is off by 47 u.
template <bool kA>
__device__ __forceinline__ double crt_dither(uint32_t k) {
  uint32_t h = k * 0x9e3779b1u + (kA ? 0x7f4a7c15u : 0x1ce4e5b9u);
  h = (h ^ (h >> 15)) * 0x2c9277b5u;
  h = (h ^ (h >> 13)) * 0xac564b05u;
  return __hiloint2double((int)(0x3ff00000u | (h >> 12)), (int)(h << 20)) - 1.0;
}
// the four signed 16-bit limbs of floor(v sc + u), |v sc| < 2^60
__device__ __forceinline__ void crt_limbs(double v, double sc, double u, float (&l)[4]) {
  long long x = __double2ll_rd(__dadd_rd(__dmul_rn(v, sc), u));
  const int l0 = (int)(short)x;
  x = (x - l0) >> 16;
  const int l1 = (int)(short)x;
  x = (x - l1) >> 16;
  const int xs = (int)x;
  const int l2 = (int)(short)xs;
  l[0] = (float)l0;
  l[1] = (float)l1;
  l[2] = (float)l2;
  l[3] = (float)((xs - l2) >> 16);
}

constexpr float kRound = 12582912.0f;  // 1.5 * 2^23: adding it rounds to an integer in the low bits

// the symmetric residue of the limbs' integer times the constants' factor, in the low byte
template <bool kA>
__device__ __forceinline__ uint32_t crt_residue(const float (&l)[4], int m) {
  const float(&c)[4] = kA ? crt.ca[m] : crt.cb[m];
  const float v = fmaf(l[3], c[3], fmaf(l[2], c[2], fmaf(l[1], c[1], l[0] * c[0])));
  const float q = fmaf(v, crt.ip[m], kRound) - kRound;
  return __float_as_uint(fmaf(-crt.p[m], q, v) + kRound);
}

__device__ __forceinline__ uint32_t crt_pack(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  return __byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410);
}

// eight consecutive K entries v (scaled by sc) of row `row`: 8 bytes into every plane
template <bool kA>
__device__ __forceinline__ void crt_store8(const double (&v)[8], double sc, const double (&u)[8],
                                           int8_t* __restrict__ out, size_t plane) {
  float l[8][4];
#pragma unroll
  for (int e = 0; e < 8; e++) crt_limbs(v[e], sc, u[e], l[e]);
#pragma unroll
  for (int m = 0; m < kMod; m++) {
    uint32_t r[8];
#pragma unroll
    for (int e = 0; e < 8; e++) r[e] = crt_residue<kA>(l[e], m);
    *reinterpret_cast<uint2*>(out + (size_t)m * plane) =
        make_uint2(crt_pack(r[0], r[1], r[2], r[3]), crt_pack(r[4], r[5], r[6], r[7]));
  }
}

// rows with K contiguous (W's genes over a range of cells): planes [row][ldk], zeros in [len, kpad)
__global__ void __launch_bounds__(256) k_crt_conv_rows(const double* __restrict__ src, int64_t ld, int len, int kpad,
                                                       int64_t ldk, size_t plane, const double* __restrict__ sc,
                                                       int8_t* __restrict__ out, const int* __restrict__ flag) {
  if (*flag) return;
  const int j = blockIdx.x, i = (blockIdx.y * 256 + threadIdx.x) * 8;  // genes along x: more than 65,535
  if (i >= kpad) return;
  const double* r = src + (size_t)j * ld + i;
  double v[8];
  if (i + 8 <= len) {
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const double2 t = *reinterpret_cast<const double2*>(r + 2 * e);
      v[2 * e] = t.x;
      v[2 * e + 1] = t.y;
    }
  } else {
#pragma unroll
    for (int e = 0; e < 8; e++) v[e] = i + e < len ? r[e] : 0.0;
  }
  double u[8];
#pragma unroll
  for (int e = 0; e < 8; e++) u[e] = crt_dither<true>(i + e);
  crt_store8<true>(v, sc[j], u, out + (size_t)j * ldk + i, plane);
}

// the pair products of a range of cells: planes [pair][ldk]; kConvPairs pairs per block, which share
// D_a / Omega while a lasts
constexpr int kConvPairs = 8;
__global__ void __launch_bounds__(256) k_crt_conv_pairs(int ldN, int c0, int len, int kpad, int64_t ldk, size_t plane,
                                                        int n_pairs, const int2* __restrict__ pairs,
                                                        const double* __restrict__ D, const double* __restrict__ rOm,
                                                        const double* __restrict__ sc, int8_t* __restrict__ out,
                                                        const int* __restrict__ flag) {
  if (*flag) return;
  const int i = (blockIdx.x * 256 + threadIdx.x) * 8;
  if (i >= kpad) return;
  // the columns are padded to ldN >= the cells, in steps of 32: an 8-cell piece that starts inside
  // [0, len) can be read whole; products past the range are dropped
  const bool any = i < len;
  const int at = any ? c0 + i : c0;
  double u[8];
#pragma unroll
  for (int e = 0; e < 8; e++) u[e] = crt_dither<false>(i + e);
  for (int p = blockIdx.y * kConvPairs; p < min(n_pairs, (int)(blockIdx.y + 1) * kConvPairs); p++) {
    const int2 q = pairs[p];
    const double *da = D + (size_t)q.x * ldN + at, *db = D + (size_t)q.y * ldN + at;
    double v[8];
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const double2 a = *reinterpret_cast<const double2*>(da + 2 * e);
      const double2 b = *reinterpret_cast<const double2*>(db + 2 * e);
      const double2 o = *reinterpret_cast<const double2*>(rOm + at + 2 * e);
      v[2 * e] = i + 2 * e < len ? a.x * b.x * o.x : 0.0;
      v[2 * e + 1] = i + 2 * e + 1 < len ? a.y * b.y * o.y : 0.0;
    }
    crt_store8<false>(v, sc[p], u, out + (size_t)p * ldk + i, plane);
  }
}

// rows with K strided, src[k * ld + m] bal[k]: planes [m][ldk], zeros in [K, kpad). Tiles of 32 rows x 128
// K entries: lanes read along the rows, the packed residues turn through shared memory.
constexpr int kTurnWords = 33;  // 32 words of 4 residues per row, padded
template <bool kA>
__global__ void __launch_bounds__(256) k_crt_conv_cols(const double* __restrict__ src, int64_t ld, int M, int K,
                                                       int64_t ldk, size_t plane, const double* __restrict__ bal,
                                                       const double* __restrict__ sc, int8_t* __restrict__ out,
                                                       const int* __restrict__ flag) {
  extern __shared__ uint32_t turn[];  // [kMod][32][kTurnWords]
  __shared__ double u[128];
  if (*flag) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m = blockIdx.x * 32 + lane, k0 = blockIdx.y * 128;
  if (threadIdx.x < 128) u[threadIdx.x] = crt_dither<kA>(k0 + threadIdx.x);
  __syncthreads();
  const double s = m < M ? sc[m] : 0.0;
#pragma unroll 1
  for (int g = 0; g < 4; g++) {
    const int kw = warp * 4 + g;  // word of four K entries
    float l[4][4];
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const int k = k0 + kw * 4 + e;
      crt_limbs(m < M && k < K ? src[(size_t)k * ld + m] * bal[k] : 0.0, s, u[kw * 4 + e], l[e]);
    }
#pragma unroll
    for (int q = 0; q < kMod; q++)
      turn[(q * 32 + lane) * kTurnWords + kw] = crt_pack(crt_residue<kA>(l[0], q), crt_residue<kA>(l[1], q),
                                                         crt_residue<kA>(l[2], q), crt_residue<kA>(l[3], q));
  }
  __syncthreads();
  for (int e = warp; e < kMod * 32; e += 8) {  // a row of a plane per warp: 128 bytes
    const int q = e >> 5, r = e & 31, row = blockIdx.x * 32 + r;
    if (row < M)
      *reinterpret_cast<uint32_t*>(out + (size_t)q * plane + (size_t)row * ldk + k0 + 4 * lane) =
          turn[(q * 32 + r) * kTurnWords + lane];
  }
}

// ---- the product, one modulus at a time --------------------------------------------------------
struct I8Shared {
  uint64_t full[kStagesI8];
  uint64_t empty[kStagesI8];
  uint64_t accb[2];
  uint64_t drained[2];
  uint64_t fin;
  uint32_t tmem;
  int abort;
};

__device__ __forceinline__ void i8_fail(int* err, I8Shared* sh, int code) {
  atomicExch(&sh->abort, 1);
  atomicCAS(err, 0, code);
}

// kind::i8: signed 8-bit A and B (K-major), INT32 accumulator
__host__ __device__ constexpr uint32_t idesc_i8(int M, int N) {
  return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mma_i8_pair(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(da), "l"(db), "r"(idesc), "r"(accumulate));
}

struct I8Args {
  int tiles_m, tiles_n, group, chunks;
  int a_rows, b_rows;  // rows of one plane of A and of B
  size_t plane;        // bytes of one output plane
  int64_t ldo;
  uint8_t* out;
  const int* flag;
  int* err;
};

// tile t of the walk: modulus by modulus; within one, `group` row tiles down each column tile, so
// that the pairs running at a time share both operands through L2
__device__ __forceinline__ void i8_tile(const I8Args& a, int t, int* mod, int* tm, int* tn) {
  const int per = a.tiles_m * a.tiles_n;
  *mod = t / per;
  t -= *mod * per;
  const int strip = a.group * a.tiles_n, s = t / strip, first = s * a.group;
  const int rows = min(a.tiles_m - first, a.group), r = t - s * strip;
  *tm = first + r % rows;
  *tn = r / rows;
}

// Persistent CTA pairs (cta_group::2): a pair owns a 256 x 256 tile, each CTA 128 rows of A, half of
// B's rows and 128 rows of the accumulator; 64 KB of operands per 128 K entries for the pair, where
// a single CTA's 128 x 256 tile would take half as much again from L2 per product. Warp 0 loads
// (TMA, six stages of 128 K entries), warp 1 of the even CTA issues the MMAs, warps 2-5 reduce the
// finished tile to bytes while the next one accumulates in the other half of TMEM. Barriers as in
// k_tc_gram2 (k_tc.cu); every wait is bounded.
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreadsI8, 1)
    k_crt_gemm(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const I8Args a) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* base = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* As = base;
  unsigned char* Bs = As + kStagesI8 * kOperand;
  I8Shared* sh = (I8Shared*)(Bs + kStagesI8 * kOperand);
  if (*a.flag) return;  // set before this launch: every CTA returns

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
  const int tiles = kMod * a.tiles_m * a.tiles_n;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStagesI8; s++) {
      mbar_init(&sh->full[s], 1);
      mbar_init(&sh->empty[s], 1);
    }
    for (int b = 0; b < 2; b++) {
      mbar_init(&sh->accb[b], 1);
      mbar_init(&sh->drained[b], 8);  // one arrival per drain warp of both CTAs
    }
    mbar_init(&sh->fin, 1);
    sh->abort = *(const volatile int*)a.err != 0;
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc_pair(&sh->tmem, 512);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem = sh->tmem;

  if (warp == 0) {
    if (lane == 0) {
      int it = 0;
      bool ok = true;
      for (int t = pair; t < tiles && ok; t += n_pairs) {
        int mod, tm, tn;
        i8_tile(a, t, &mod, &tm, &tn);
        const int ya = mod * a.a_rows + tm * kTile + 128 * (int)rank;
        const int yb = mod * a.b_rows + tn * kTile + 128 * (int)rank;
        for (int c = 0; c < a.chunks; c++, it++) {
          const int s = it % kStagesI8;
          if (it >= kStagesI8 && !mbar_wait(&sh->empty[s], ((it / kStagesI8) - 1) & 1, a.err)) {
            i8_fail(a.err, sh, 41);
            ok = false;
            break;
          }
          if (*(const volatile int*)&sh->abort) {
            ok = false;
            break;
          }
          const uint32_t fb = mapa_shared(smem_u32(&sh->full[s]), 0);
          if (rank == 0) mbar_arrive_expect_tx(&sh->full[s], 4u * kOperand);
          tma_load_2d_pair(As + s * kOperand, &map_a, fb, c * kChunk, ya);
          tma_load_2d_pair(Bs + s * kOperand, &map_b, fb, c * kChunk, yb);
        }
      }
      // the even CTA sees both CTAs' last loads land before the final cluster barrier
      if (rank == 0)
        for (int k = max(0, it - kStagesI8); k < it; k++)
          if (!mbar_wait(&sh->full[k % kStagesI8], (k / kStagesI8) & 1, nullptr)) atomicCAS(a.err, 0, 42);
    }
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {
      constexpr uint32_t idesc = idesc_i8(kTile, kTile);
      int it = 0, n = 0;
      bool ok = true;
      for (int t = pair; t < tiles && ok; t += n_pairs, n++) {
        const int buf = n & 1;
        if (n >= 2 && !mbar_wait(&sh->drained[buf], ((n >> 1) - 1) & 1, a.err)) {
          i8_fail(a.err, sh, 46);
          break;
        }
        const uint32_t acc = tmem + buf * kTile;
        for (int c = 0; c < a.chunks; c++, it++) {
          const int s = it % kStagesI8;
          if (!mbar_wait(&sh->full[s], (it / kStagesI8) & 1, a.err)) {
            i8_fail(a.err, sh, 43);
            ok = false;
            break;
          }
          if (*(const volatile int*)&sh->abort) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t as = smem_u32(As + s * kOperand), bs = smem_u32(Bs + s * kOperand);
#pragma unroll
          for (int k = 0; k < kChunk / 32; k++)
            mma_i8_pair(acc, umma_desc_sw128(as + k * 32), umma_desc_sw128(bs + k * 32), idesc, (c | k) ? 1u : 0u);
          mma_commit_pair_mc(&sh->empty[s], 3);
        }
        if (ok) mma_commit_pair_mc(&sh->accb[buf], 3);
      }
      mma_commit_pair(&sh->fin);
      if (!mbar_wait(&sh->fin, 0, nullptr)) atomicCAS(a.err, 0, 47);
    }
  } else {
    const int q = warp & 3;
    const int row = q * 32 + lane;
    const uint32_t lane_addr = tmem + ((uint32_t)(q * 32) << 16);
    const uint32_t dr[2] = {mapa_shared(smem_u32(&sh->drained[0]), 0), mapa_shared(smem_u32(&sh->drained[1]), 0)};
    int n = 0;
    for (int t = pair; t < tiles; t += n_pairs, n++) {
      const int buf = n & 1;
      const bool w = mbar_wait(&sh->accb[buf], (n >> 1) & 1, a.err);
      if (!__all_sync(0xffffffffu, w)) {
        if (!w) i8_fail(a.err, sh, 45);
        break;
      }
      tc_fence_after();
      int mod, tm, tn;
      i8_tile(a, t, &mod, &tm, &tn);
      const uint32_t p = crt.pu[mod], off = crt.off[mod], magic = crt.magic[mod];
      uint8_t* o = a.out + (size_t)mod * a.plane + (size_t)(tm * kTile + 128 * (int)rank + row) * a.ldo + tn * kTile;
#pragma unroll 1
      for (int cb = 0; cb < kTile; cb += 32) {
        float f[32];
        tmem_ld32(lane_addr + buf * kTile + cb, f);
        if (cb + 32 == kTile) {  // the last read of this buffer
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(dr[buf]);
        }
        uint32_t w4[8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
          uint32_t r[4];
#pragma unroll
          for (int e = 0; e < 4; e++) {
            const uint32_t x = __float_as_uint(f[4 * k + e]) + off;
            r[e] = x - (__umulhi(x, magic) >> 7) * p;  // in [0, 256)
          }
          w4[k] = crt_pack(r[0], r[1], r[2], r[3]);
        }
        *reinterpret_cast<uint4*>(o + cb) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
        *reinterpret_cast<uint4*>(o + cb + 16) = make_uint4(w4[4], w4[5], w4[6], w4[7]);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // both CTAs are done with TMEM and the even CTA saw every load land
  tc_fence_after();
  if (warp == 0) tmem_dealloc_pair(tmem, 512);
}

// ---- back to FP64 ----------------------------------------------------------------------------------
// Four neighbouring entries from their residue bytes c_l (one word per plane), in units of
// P / 2^64: with the CRT factors in the operands the integer is x = P frac(sum_l c_l / p_l), frac in
// [-1/2, 1/2), so the sum is taken modulo 1 in a 64-bit fraction (plus 16 guard bits), whose
// rounding, 2^-64 P, lies below that of the operands.
__device__ __forceinline__ void crt_values(const uint8_t* __restrict__ in, size_t plane, double (&v)[4]) {
  uint32_t w[kMod];
#pragma unroll
  for (int l = 0; l < kMod; l++) w[l] = __ldcs(reinterpret_cast<const uint32_t*>(in + (size_t)l * plane));
  // two entries at a time: digit sums q[k] = sum_l c_l (digit k of 1 / p_l) < 2^28, two moduli per
  // instruction (64 a clock and SM, as a multiply-add; the 64-bit multiply-adds they replace, 20)
#pragma unroll
  for (int e = 0; e < 4; e += 2) {
    uint32_t q0[5] = {1u << 15, 0, 0, 0, 0}, q1[5] = {1u << 15, 0, 0, 0, 0};
#pragma unroll
    for (int h = 0; h < kMod / 2; h++) {
      const uint32_t c = __byte_perm(w[2 * h], w[2 * h + 1], e ? 0x7362 : 0x5140);  // bytes of both planes
#pragma unroll
      for (int k = 0; k < 5; k++) {
        q0[k] = __dp2a_lo(crt.fr[k][h], c, q0[k]);
        q1[k] = __dp2a_hi(crt.fr[k][h], c, q1[k]);
      }
    }
    auto value = [](const uint32_t (&q)[5]) {
      const uint64_t x = (uint64_t)((q[0] >> 16) + q[1]) + ((uint64_t)q[2] << 16) + ((uint64_t)q[3] << 32) +
                         ((uint64_t)q[4] << 48);
      return (double)(int64_t)x;
    };
    v[e] = value(q0);
    v[e + 1] = value(q1);
  }
}

// Psi_j's dense block (both triangles, plus DeltaInv) from the residues of gene rows x pair columns;
// over several ranges of cells the partial sums collect in acc (first / last: the range's place).
// A gene's row of W cannot be balanced for all pairs at once: where its mass lies on other cells than a
// column's, the sum is far below the product of the norms. So a gene goes on the list of the DMMA form
// when the rounding of a diagonal entry, `unit` inv_j inv_p (0.58 R units; its ranges added up, in err), is
// more than `share` of that entry. The diagonal is enough, as in k_crt_u: |p_ab|^2 <= |p_aa| |p_bb| by
// Cauchy-Schwarz, so the rounding of entry (a, b) stays within that share of sqrt(Psi_aa Psi_bb), the
// scale by which a factorization sees it.
__global__ void __launch_bounds__(256) k_crt_psi(int P, int n_pairs, int64_t ldo, size_t plane,
                                                 const uint8_t* __restrict__ in, const double* __restrict__ inv_j,
                                                 const double* __restrict__ inv_p, const int2* __restrict__ pairs,
                                                 const int* __restrict__ dcol, const double* __restrict__ Dinv,
                                                 double* __restrict__ acc, int64_t lda, int first, int last,
                                                 double* __restrict__ Psi, int n_d, double unit, double share,
                                                 double* __restrict__ err, CrtGenes genes) {
  if (*(const volatile int*)genes.state) return;
  const int j = blockIdx.x, p0 = (blockIdx.y * 256 + threadIdx.x) * 4;
  if (p0 >= n_pairs) return;
  double v[4];
  crt_values(in + (size_t)j * ldo + p0, plane, v);
  const double sj = inv_j[j] * kUnit;
  double* Pj = Psi + (size_t)j * P * P;
#pragma unroll
  for (int e = 0; e < 4; e++) {
    const int p = p0 + e;
    if (p >= n_pairs) break;
    double x = v[e] * inv_p[p] * sj;
    if (!first) x += acc[(size_t)j * lda + p];
    const int2 q = pairs[p];
    double off = 0.0;
    if (q.x == q.y) {
      off = unit * inv_j[j] * inv_p[p];
      if (!first) off += err[(size_t)j * n_d + q.x];
      if (!last) err[(size_t)j * n_d + q.x] = off;
    }
    if (!last) {
      acc[(size_t)j * lda + p] = x;
    } else {
      const size_t mk = dcol[q.x], ml = dcol[q.y];
      x += Dinv[mk + ml * P];
      if (q.x == q.y && !(off <= share * x)) genes.add(j);
      Pj[mk + ml * P] = x;
      Pj[ml + mk * P] = x;
    }
  }
}

// U_i = sum_b D_ib V[i, pair(a, b)], V[i, p] = (1/Omega_i) sum_j W_ij S_j[p], W warps per cell: the
// cell's row of V from its residues into shared memory (pair_rows.cuh). The operands' entries are off by 0.41
// of a unit (rms), so a sum by at most 0.58 R units, R bounding both rows' norms. Where that is more than its
// share (crt_share) of a diagonal V[i, (a, a)], the value below `least` units, the cell's 128 cells go to the
// DMMA form. The diagonal is enough: W_ij and the
// S_j[a, a] are positive, |S_j[a, b]| <= sqrt(S_j[a, a] S_j[b, b]), and so by Cauchy-Schwarz the rounding of
// V[i, (a, b)] stays within the same share of sqrt(V[i, (a, a)] V[i, (b, b)]).
// Bound by the entries' arithmetic (crt_values) while 24 to 32 warps share an SM; without the limit on
// registers the compiler keeps several entries' loads and all the digits in flight at half the warps
// (50,000 cells x 132 columns x 1,000 genes: 6.0 against 2.9 ms).
template <int S, int W>
__global__ void __launch_bounds__(256, S > 9 ? 2 : S > 5 ? 4 : 3) k_crt_u(int ldN, int n_d, int len, int c0, int64_t ldo, size_t plane,
                                               const uint8_t* __restrict__ in, const double* __restrict__ inv_i,
                                               const double* __restrict__ inv_p, const double* __restrict__ rOm,
                                               const double* __restrict__ D, double least, double* __restrict__ U,
                                               int* __restrict__ cells) {
  extern __shared__ __align__(16) double vs[];
  if (cells[0]) return;
  const int g = W == 8 ? 0 : threadIdx.x >> 5, r = blockIdx.x * (8 / W) + g, i = c0 + r;
  if (r >= len) return;  // W = 1: a whole warp, no barrier of the block follows
  double* vc = vs + g * u_space<W, true>(n_d);
  const double s = inv_i[r] * rOm[i] * kUnit;
  const uint8_t* row_in = in + (size_t)r * ldo;
  const double* dv = pair_rows_to_u<S, W, true>(i, ldN, n_d, vc, D, U, [&](int from, int p1, int tid, int nt) {
    for (int p = from + 4 * tid; p < p1; p += 4 * nt) {
      double v[4];
      crt_values(row_in + p, plane, v);
      const double2 x = *reinterpret_cast<const double2*>(inv_p + p), y = *reinterpret_cast<const double2*>(inv_p + p + 2);
      *reinterpret_cast<double2*>(vc + p - from) = make_double2(v[0] * x.x * s, v[1] * x.y * s);
      *reinterpret_cast<double2*>(vc + p - from + 2) = make_double2(v[2] * y.x * s, v[3] * y.y * s);
    }
  });
  bool out = false;
  for (int a = W == 8 ? threadIdx.x : threadIdx.x & 31; a < n_d; a += 32 * W)
    out |= !(dv[a] >= least * inv_p[a * n_d - a * (a - 1) / 2] * s);
  if (out) cells[1 + (i >> 7)] = 1;
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
namespace {
constexpr int kSmemI8 = 1024 + kStagesI8 * 2 * kOperand + (int)sizeof(I8Shared);
constexpr int kSmemTurn = kMod * 32 * kTurnWords * (int)sizeof(uint32_t);
constexpr int kNormSmem = (int)sizeof(double) * 32 * (kUMaxDense + 1);
constexpr int kGroupI8 = 8;

int up(int64_t v, int m) { return (int)((v + m - 1) / m * m); }
}  // namespace

// Where the integer form is taken: by both forms' times (us), as estimated by costs fitted to measurements.
// The Gram, over 600 to 20,000 cells, 40 to 2,500 genes and 55 to 8,515 pairs (within 36%; the faster form
// was missed by more than 5% at three of 86 sizes): the DMMA form's tiles (pair_gram_cost) and its pair products;
// this one's 256 x 256 tiles of each modulus on 74 CTA pairs, the conversions and the way back. E.g. 2,000 cells
// x 300 x 595: 154 integer, 111 DMMA; 5,000 x 1,000 x 595: 268 / 393; 20,000 x 1,000 x 8,515: 3,736 / 12,668.
static bool crt_gram_faster(const Ctx* c, double N, double J, double pairs) {
  const double dmma = 54 + pair_gram_cost(c, c->pr.n_pairs) * N / 16 / 1900 + N * (3.8e-6 * pairs + 1.7e-6 * J) +
                      19e-6 * J * pairs;
  const double tiles = kMod * std::ceil(J / kTile) * std::ceil(pairs / kTile);
  const double integer = 126 + 0.40 * std::ceil(tiles / (c->sm_count / 2)) * std::ceil(N / kChunk) +
                         N * (7.9e-6 * pairs + 10.4e-6 * J) + 24e-6 * J * pairs;
  return integer < dmma;
}
// The gradient pairs, over 1,000 to 30,000 cells, 20 to 1,000 genes and 21 to 4,851 pairs. DMMA: 0.165 per
// gene and wave of tiles, and the pair rows. Integer: the conversions of both operands, the way back to FP64,
// padded tiles and chunks, and the products. E.g. 1,000 x 1,000 x 105: 169 / 65; 3,000 x 300 x 595: 74 / 107;
// 30,000 x 300 x 105: 167 / 391; 30,000 x 300 x 4,851: 3,707 / 2,495 (DMMA / integer).
static bool crt_grad_faster(const Ctx* c, double N, double J, double pairs, double Jk, double Pp) {
  const double waves = std::ceil(std::ceil(N / 128) * std::ceil(pairs / 128) / c->sm_count);
  const double dmma = 10 + 0.165 * J * waves + 5e-6 * N * pairs;
  const double integer = 50 + N * (15e-6 * Pp + 10e-6 * Jk) + N * Jk * Pp * 2 * kMod / 2.9e9;
  return integer < dmma;
}
void crt_plan(Ctx* c, size_t cap) {
  PairState& s = c->pr;
  CrtState& t = s.crt;
  t = CrtState();
  const int64_t N = c->N, J = c->J;
  t.Jp = up(J, kTile);
  t.Pp = up(s.n_pairs, kTile);
  t.Jk = up(J, kChunk);
  if (J > kMaxK || c->n_d > kUMaxDense) return;
  int64_t most = std::min<int64_t>(up(N, kTile), kMaxK / kTile * kTile);
  if (c->pair_range_cells > 0) {  // ranges below a tile: the DMMA form
    if (c->pair_range_cells < kTile) return;
    most = std::min<int64_t>(most, c->pair_range_cells / kTile * kTile);
  }
  const int64_t acc = sizeof(double) * J * t.Pp;
  auto gram = [&](int64_t n) { return kMod * ((int64_t)(t.Jp + t.Pp) * n + (int64_t)t.Jp * t.Pp) + (n < N ? acc : 0); };
  auto grad = [&](int64_t n) {
    return kMod * ((int64_t)t.Pp * t.Jk + n * (t.Jk + t.Pp));
  };
  auto cells = [&](auto&& bytes) -> int64_t {
    int64_t n = most;
    if ((size_t)bytes(n) > cap) {
      const int64_t per = bytes(2 * kTile) - bytes(kTile);
      const int64_t base = bytes(kTile) - per + acc;
      n = ((int64_t)cap - base) / std::max<int64_t>(1, per / kTile) / kTile * kTile;
    }
    if (n < std::min<int64_t>(most, 4 * kTile)) return 0;
    const int64_t ranges = (N + n - 1) / n;  // ranges of one size
    return std::min<int64_t>(n, up((N + ranges - 1) / ranges, kTile));
  };
  t.gram_cells = crt_gram_faster(c, N, J, s.n_pairs) ? (int)cells(gram) : 0;
  t.grad_cells = crt_grad_faster(c, N, J, s.n_pairs, t.Jk, t.Pp) ? (int)cells(grad) : 0;
  t.bytes = (size_t)std::max(t.gram_cells ? gram(t.gram_cells) : 0, t.grad_cells ? grad(t.grad_cells) : 0);
  t.on = t.gram_cells > 0 || t.grad_cells > 0;
}

int crt_prepare(Ctx* c) {
  PairState& s = c->pr;
  CrtState& t = s.crt;
  if (!t.on) return GPL_OK;
  const size_t rows = (size_t)2 * (t.Jp + t.Pp + t.grad_cells), tiles = div_up(c->N, 128);
  const size_t ints = 5 + tiles + 2 * (size_t)c->J + div_up(c->J, 128);
  const size_t errs = t.gram_cells && t.gram_cells < c->N ? (size_t)c->J * c->n_d : 0;
  if (cudaMalloc((void**)&t.scales, sizeof(double) * (rows + 2 * t.Jp + errs)) != cudaSuccess ||
      cudaMalloc((void**)&t.err, ints * sizeof(int)) != cudaSuccess) {
    cudaGetLastError();
    c->err = "device allocation failed: scales of the integer pair products";
    return GPL_ERR_ALLOC;
  }
  t.balance = t.scales + rows;  // of W, then of the pairs
  t.cells = t.err + 1;
  t.genes = t.cells + 1 + tiles;
  t.list = t.genes + 2 + c->J;
  t.cols = t.list + c->J;
  t.g_err = t.balance + 2 * t.Jp;
  GPL_TRY(c, cudaMemset(t.err, 0, ints * sizeof(int)));
  int8_t* pool = reinterpret_cast<int8_t*>(s.V);
  // Gram: gene planes, pair planes, residues out, partial sums over the ranges
  t.g_a = pool;
  t.g_b = t.g_a + (size_t)kMod * t.Jp * t.gram_cells;
  t.g_out = reinterpret_cast<uint8_t*>(t.g_b + (size_t)kMod * t.Pp * t.gram_cells);
  t.g_acc = reinterpret_cast<double*>(t.g_out + (size_t)kMod * t.Jp * t.Pp);
  // gradient: pair planes over the genes, cell planes, residues out
  t.v_b = pool;
  t.v_a = t.v_b + (size_t)kMod * t.Pp * t.Jk;
  t.v_out = reinterpret_cast<uint8_t*>(t.v_a + (size_t)kMod * t.grad_cells * t.Jk);
  if ((t.gram_cells && (!tc_map_u8(&t.map_ga, t.g_a, t.gram_cells, (uint64_t)kMod * t.Jp) ||
                        !tc_map_u8(&t.map_gb, t.g_b, t.gram_cells, (uint64_t)kMod * t.Pp))) ||
      (t.grad_cells && (!tc_map_u8(&t.map_va, t.v_a, t.Jk, (uint64_t)kMod * t.grad_cells) ||
                        !tc_map_u8(&t.map_vb, t.v_b, t.Jk, (uint64_t)kMod * t.Pp)))) {
    c->err = "cuTensorMapEncodeTiled failed";
    return GPL_ERR_CUDA;
  }
  GPL_TRY(c, cudaFuncSetAttribute(k_crt_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemI8));
  GPL_TRY(c, cudaFuncSetAttribute(k_crt_conv_cols<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemTurn));
  GPL_TRY(c, cudaFuncSetAttribute(k_crt_conv_cols<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemTurn));
  GPL_TRY(c, cudaFuncSetAttribute(k_crt_norm_pairs, cudaFuncAttributeMaxDynamicSharedMemorySize, kNormSmem));
  return GPL_OK;
}

void crt_release(Ctx* c) {
  CrtState& t = c->pr.crt;
  if (t.scales) cudaFree(t.scales);
  if (t.err) cudaFree(t.err);
  t = CrtState();
}

static int crt_gemm(Ctx* c, const CUtensorMap& ma, const CUtensorMap& mb, int rows, int cols, int a_rows, int b_rows,
                    int k, uint8_t* out, size_t plane, int64_t ldo, const int* flag) {
  I8Args a{};
  a.tiles_m = div_up(rows, kTile);
  a.tiles_n = div_up(cols, kTile);
  a.group = kGroupI8;
  a.chunks = div_up(k, kChunk);
  a.a_rows = a_rows;
  a.b_rows = b_rows;
  a.plane = plane;
  a.ldo = ldo;
  a.out = out;
  a.flag = flag;
  a.err = c->pr.crt.err;
  const int tiles = kMod * a.tiles_m * a.tiles_n;
  const int grid = 2 * std::min(tiles, c->sm_count / 2);
  k_crt_gemm<<<grid, kThreadsI8, kSmemI8, c->stream>>>(ma, mb, a);
  GPL_LAUNCHED(c, "k_crt_gemm");
  return GPL_OK;
}

// What the rounding of an integer product may be of the diagonal it is measured by (k_crt_psi, k_crt_u), over K
// terms: what a chain of K FP64 multiply-adds is off by, 0.15 sqrt(K) u (rms; 12 u measured at K = 6,001, 19 u
// at 19,997), and 4 u at least. The rounding is taken at its bound, which lies up to twice above its rms.
static double crt_share(double K) {
  return 0x1p-53 * std::max(4.0, 0.15 * std::sqrt(K));
}

// scales of rows with K strided (src[k * ld + m] bal[k]); `part` holds at least 16 sums per row
static int crt_col_scales(Ctx* c, const double* src, int64_t ld, int M, int K, const double* bal, double* part,
                          double* sc, double* inv, int* flag, int shift) {
  const int nb = div_up(M, 256);
  const int ks = std::max(1, std::min({16, 1184 / std::max(1, nb), div_up(K, 64)}));
  const int kper = div_up(K, ks);
  k_crt_norm_cols<<<dim3(nb, ks), 256, 0, c->stream>>>(src, ld, M, K, kper, bal, part);
  GPL_LAUNCHED(c, "k_crt_norm_cols");
  k_crt_scales<<<nb, 256, 0, c->stream>>>(M, ks, part, crt_norm_limit(), sc, inv, flag, shift);
  GPL_LAUNCHED(c, "k_crt_scales");
  return GPL_OK;
}

// Every Psi_j's dense block from W, 1/Omega (s.rOm) and the dense columns.
int launch_crt_gram(Ctx* c) {
  PairState& s = c->pr;
  CrtState& t = s.crt;
  const double R = crt_norm_limit();
  double *sc_j = t.scales, *inv_j = sc_j + t.Jp, *sc_p = inv_j + t.Jp, *inv_p = sc_p + t.Pp;
  double* part = reinterpret_cast<double*>(t.g_out);
  const CrtGenes genes{t.genes, t.list};
  GPL_TRY(c, cudaMemsetAsync(t.genes, 0, (2 + c->J) * sizeof(int), c->stream));
  for (int c0 = 0; c0 < c->N; c0 += t.gram_cells) {
    const int len = std::min(t.gram_cells, c->N - c0), kpad = up(len, kChunk);
    const size_t plane_a = (size_t)t.Jp * t.gram_cells, plane_b = (size_t)t.Pp * t.gram_cells;
    const size_t plane_o = (size_t)t.Jp * t.Pp;
    k_crt_norm_rows<<<c->J, 256, 0, c->stream>>>(c->W + c0, c->ldN, len, R, sc_j, inv_j, genes);
    GPL_LAUNCHED(c, "k_crt_norm_rows");
    const int gx = div_up(s.n_pairs, 256 * kNormPairs);
    // as many cell parts as fill the SMs, within the partial sums' space (14 bytes x 256 rows per pair)
    const int gy = std::max(1, std::min({div_up(len, 64), 592 / gx, 256}));
    const int cper = up(div_up(len, gy), 32);
    const int ny = div_up(len, cper);
    k_crt_norm_pairs<<<dim3(gx, ny), 256, sizeof(double) * 32 * (c->n_d + 1), c->stream>>>(
        c->ldN, c->n_d, c0, c0 + len, cper, s.n_pairs, s.pairs, c->Dm, s.rOm, part);
    GPL_LAUNCHED(c, "k_crt_norm_pairs");
    k_crt_scales<<<div_up(s.n_pairs, 256), 256, 0, c->stream>>>(s.n_pairs, ny, part, R, sc_p, inv_p, t.genes, 31);
    GPL_LAUNCHED(c, "k_crt_scales");
    k_crt_conv_rows<<<dim3(c->J, div_up(kpad, 2048)), 256, 0, c->stream>>>(c->W + c0, c->ldN, len, kpad, t.gram_cells,
                                                                          plane_a, sc_j, t.g_a, t.genes);
    GPL_LAUNCHED(c, "k_crt_conv_rows");
    k_crt_conv_pairs<<<dim3(div_up(kpad, 2048), div_up(s.n_pairs, kConvPairs)), 256, 0, c->stream>>>(
        c->ldN, c0, len, kpad, t.gram_cells, plane_b, s.n_pairs, s.pairs, c->Dm, s.rOm, sc_p, t.g_b, t.genes);
    GPL_LAUNCHED(c, "k_crt_conv_pairs");
    const int rc = crt_gemm(c, t.map_ga, t.map_gb, c->J, s.n_pairs, t.Jp, t.Pp, len, t.g_out, plane_o, t.Pp, t.genes);
    if (rc) return rc;
    k_crt_psi<<<dim3(c->J, div_up(s.n_pairs, 1024)), 256, 0, c->stream>>>(
        c->P, s.n_pairs, t.Pp, plane_o, t.g_out, inv_j, inv_p, s.pairs, c->dcol_d, c->DeltaInv, t.g_acc, t.Pp,
        c0 == 0, c0 + len >= c->N, c->Psi, c->n_d, 0.58 * R, crt_share(c->N), t.g_err, genes);
    GPL_LAUNCHED(c, "k_crt_psi");
  }
  return GPL_OK;
}

// U from W, 1/Omega and the gathered pairs of every Psi_j^{-1} (s.Sp).
int launch_crt_uq(Ctx* c) {
  PairState& s = c->pr;
  CrtState& t = s.crt;
  double *sc_p = t.scales + 2 * t.Jp, *inv_p = sc_p + t.Pp, *sc_i = inv_p + t.Pp, *inv_i = sc_i + t.grad_cells;
  double* part = reinterpret_cast<double*>(t.v_out);
  const size_t plane_b = (size_t)t.Pp * t.Jk, plane_a = (size_t)t.grad_cells * t.Jk;
  const size_t plane_o = (size_t)t.grad_cells * t.Pp;
  const double *bal_w = t.balance, *bal_s = bal_w + t.Jp;
  GPL_TRY(c, cudaMemsetAsync(t.cells, 0, (1 + div_up(c->N, 128)) * sizeof(int), c->stream));
  k_crt_balance<<<c->J, 256, 0, c->stream>>>(c->N, c->ldN, c->n_d, s.pairs_pad, c->W, s.Sp, t.balance,
                                             t.balance + t.Jp);
  GPL_LAUNCHED(c, "k_crt_balance");
  int rc;
  if ((rc = crt_col_scales(c, s.Sp, s.pairs_pad, s.n_pairs, c->J, bal_s, part, sc_p, inv_p, t.cells, 31))) return rc;
  const double least = 0.58 * crt_norm_limit() / crt_share(c->J) / kUnit;
  k_crt_conv_cols<false><<<dim3(div_up(s.n_pairs, 32), t.Jk / 128), 256, kSmemTurn, c->stream>>>(
      s.Sp, s.pairs_pad, s.n_pairs, c->J, t.Jk, plane_b, bal_s, sc_p, t.v_b, t.cells);
  GPL_LAUNCHED(c, "k_crt_conv_cols");
  for (int c0 = 0; c0 < c->N; c0 += t.grad_cells) {
    const int len = std::min(t.grad_cells, c->N - c0);
    {
      ProfScope ps(c, "uq");
      // c0 is a multiple of 256: the cells' own flags, of 128 each
      if ((rc = crt_col_scales(c, c->W + c0, c->ldN, len, c->J, bal_w, part, sc_i, inv_i, t.cells + 1 + c0 / 128, 7)))
        return rc;
      k_crt_conv_cols<true><<<dim3(div_up(len, 32), t.Jk / 128), 256, kSmemTurn, c->stream>>>(
          c->W + c0, c->ldN, len, c->J, t.Jk, plane_a, bal_w, sc_i, t.v_a, t.cells);
      GPL_LAUNCHED(c, "k_crt_conv_cols");
      if ((rc = crt_gemm(c, t.map_va, t.map_vb, len, s.n_pairs, t.grad_cells, t.Pp, t.Jk, t.v_out, plane_o, t.Pp,
                         t.cells)))
        return rc;
    }
    ProfScope ps(c, "v_to_u");
    pair_rows_form(c->n_d, len, 96, [&](auto S, auto W) {
      constexpr int per = 8 / W;
      const int smem = (int)sizeof(double) * u_space<W, true>(c->n_d) * per;
      if (smem > 48 * 1024)  // 85 or more columns, a warp per cell
        cudaFuncSetAttribute(k_crt_u<S, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
      k_crt_u<S, W><<<div_up(len, per), 256, smem, c->stream>>>(c->ldN, c->n_d, len, c0, t.Pp, plane_o, t.v_out, inv_i,
                                                               inv_p, s.rOm, c->Dm, least, c->U, t.cells);
    });
    GPL_LAUNCHED(c, "k_crt_u");
  }
  return GPL_OK;
}

// T[l][j][dcol a] = sum_i D_ia g_il W_ij / Omega_i: the Gram's operands and kernels with the products of the
// dense columns and the L per-cell columns in place of the dense pairs, as many columns at a time as
// the pairs' space holds. An entry's rounding (as in k_crt_psi; each range of cells has its part of it) is held
// against sqrt(Psi_aa g^T diag(W/Omega) g), which bounds the sum of its terms' sizes; a gene with one
// beyond its share sends its 128 genes to the DMMA form.
__global__ void k_crt_column_pairs(int n_d, int rows, int2* __restrict__ pairs) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r < rows) pairs[r] = make_int2(r % n_d, n_d + r / n_d);
}
__global__ void __launch_bounds__(256) k_crt_t(int J, int P, int n_d, int rows, int64_t ldo, size_t plane,
                                               const uint8_t* __restrict__ in, const double* __restrict__ inv_j,
                                               const double* __restrict__ inv_p, const int* __restrict__ dcol,
                                               int first, double unit, const double* __restrict__ root,
                                               const double* __restrict__ gg, double* __restrict__ T, int* cols) {
  if (*(const volatile int*)cols) return;
  const int j = blockIdx.x, r0 = (blockIdx.y * 256 + threadIdx.x) * 4;
  if (r0 >= rows) return;
  double v[4];
  crt_values(in + (size_t)j * ldo + r0, plane, v);
  const double sj = inv_j[j] * kUnit;
#pragma unroll
  for (int e = 0; e < 4; e++) {
    const int r = r0 + e;
    if (r >= rows) break;
    const int l = r / n_d, a = r % n_d;
    double* t = T + ((size_t)l * J + j) * P + dcol[a];
    const double x = v[e] * inv_p[r] * sj;
    *t = first ? x : *t + x;
    if (!(unit * inv_j[j] * inv_p[r] <= root[(size_t)j * n_d + a] * sqrt(gg[j + (size_t)l * J]))) cols[1 + (j >> 7)] = 1;
  }
}
// root[j][a] = sqrt(Psi_j[dcol a, dcol a]) from the rows of its factor
__global__ void __launch_bounds__(160) k_crt_roots(int P, int n_d, const int* __restrict__ dcol,
                                                   const double* __restrict__ Psi, double* __restrict__ root) {
  const int a = threadIdx.x, j = blockIdx.x;
  if (a >= n_d) return;
  const int r = dcol[a];
  const double* L = Psi + (size_t)j * P * P + r;
  double s = 0.0;
#pragma unroll 4
  for (int k = 0; k <= r; k++) s = fma(L[(size_t)k * P], L[(size_t)k * P], s);
  root[(size_t)j * n_d + a] = sqrt(s);
}

// The two forms' times (us), by the rates measured at 30,000 x 1,000 with 132 dense columns: 330 per
// column for the DMMA form (24 TFLOP/s, at least 15), and for this one the conversions, the products
// (at 2.7e9 per us) and some nine launches. 20 columns there: 6.5 ms and 1.1 ms.
static int crt_column_group(const Ctx* c, int L) { return std::min(L, c->pr.n_pairs / c->n_d); }
bool crt_columns_faster(const Ctx* c, int L) {
  const PairState& s = c->pr;
  if (!s.ready || !s.crt.on || !s.crt.gram_cells || c->n_d > 144) return false;
  const double N = c->N, J = c->J, per = crt_column_group(c, L), rows = per * c->n_d;
  const double dmma = L * std::max(15.0, 2.0 * N * J * c->n_d / 24e6);
  const double one = 60 + N * (2.2e-6 * J + 2.3e-6 * rows) + 2.0 * kMod * N * s.crt.Jp * up(rows, kTile) / 2.7e9;
  return std::ceil(L / per) * one < dmma;
}
size_t crt_columns_work(const Ctx* c, int L) {
  const int per = crt_column_group(c, L);
  return (size_t)(c->n_d + per) * c->ldN + (size_t)per * c->n_d + (size_t)c->J * c->n_d + 2;
}

int launch_crt_columns(Ctx* c, int L, const double* G, const double* gg, double* T, double* work, int* left) {
  PairState& s = c->pr;
  CrtState& t = s.crt;
  const int per = crt_column_group(c, L);
  const double* rOm = nullptr;
  int rc = recip_omega(c, &rOm);
  if (rc) return rc;
  ProfScope ps(c, "zt_u");
  double* D = work + (reinterpret_cast<uintptr_t>(work) / sizeof(double) & 1);  // 16-byte aligned columns
  int2* pairs = reinterpret_cast<int2*>(D + (size_t)(c->n_d + per) * c->ldN);
  double* root = D + (size_t)(c->n_d + per) * c->ldN + (size_t)per * c->n_d;
  const double R = crt_norm_limit();
  double *sc_j = t.scales, *inv_j = sc_j + t.Jp, *sc_p = inv_j + t.Jp, *inv_p = sc_p + t.Pp;
  double* part = reinterpret_cast<double*>(t.g_out);
  const size_t plane_a = (size_t)t.Jp * t.gram_cells, plane_b = (size_t)t.Pp * t.gram_cells;
  const size_t plane_o = (size_t)t.Jp * t.Pp, col = sizeof(double) * c->ldN;
  const int smem_n = (int)sizeof(double) * 32 * (c->n_d + per + 1);
  const int tiles = div_up(c->J, 128);
  GPL_TRY(c, cudaMemsetAsync(t.cols, 0, (1 + tiles) * sizeof(int), c->stream));
  k_crt_roots<<<c->J, 160, 0, c->stream>>>(c->P, c->n_d, c->dcol_d, c->Psi, root);  // at most 144 dense columns
  GPL_LAUNCHED(c, "k_crt_roots");
  GPL_TRY(c, cudaMemcpyAsync(D, c->Dm, col * c->n_d, cudaMemcpyDeviceToDevice, c->stream));
  GPL_TRY(c, cudaMemsetAsync(D + (size_t)c->n_d * c->ldN, 0, col * per, c->stream));
  k_crt_column_pairs<<<div_up(per * c->n_d, 256), 256, 0, c->stream>>>(c->n_d, per * c->n_d, pairs);
  GPL_LAUNCHED(c, "k_crt_column_pairs");
  for (int l0 = 0; l0 < L; l0 += per) {
    const int nl = std::min(per, L - l0), rows = nl * c->n_d, cols = c->n_d + nl;
    GPL_TRY(c, cudaMemcpy2DAsync(D + (size_t)c->n_d * c->ldN, col, G + (size_t)l0 * c->N, sizeof(double) * c->N,
                                 sizeof(double) * c->N, nl, cudaMemcpyDeviceToDevice, c->stream));
    for (int c0 = 0; c0 < c->N; c0 += t.gram_cells) {
      const int len = std::min(t.gram_cells, c->N - c0), kpad = up(len, kChunk);
      k_crt_norm_rows<<<c->J, 256, 0, c->stream>>>(c->W + c0, c->ldN, len, R, sc_j, inv_j, CrtGenes{t.cols, nullptr});
      GPL_LAUNCHED(c, "k_crt_norm_rows");
      const int gx = div_up(rows, 256 * kNormPairs);
      const int gy = std::max(1, std::min({div_up(len, 64), 592 / gx, 256}));
      const int cper = up(div_up(len, gy), 32);
      const int ny = div_up(len, cper);
      k_crt_norm_pairs<<<dim3(gx, ny), 256, smem_n, c->stream>>>(c->ldN, cols, c0, c0 + len, cper, rows, pairs, D, rOm,
                                                                part);
      GPL_LAUNCHED(c, "k_crt_norm_pairs");
      k_crt_scales<<<div_up(rows, 256), 256, 0, c->stream>>>(rows, ny, part, R, sc_p, inv_p, t.cols, 31);
      GPL_LAUNCHED(c, "k_crt_scales");
      k_crt_conv_rows<<<dim3(c->J, div_up(kpad, 2048)), 256, 0, c->stream>>>(c->W + c0, c->ldN, len, kpad,
                                                                            t.gram_cells, plane_a, sc_j, t.g_a, t.cols);
      GPL_LAUNCHED(c, "k_crt_conv_rows");
      k_crt_conv_pairs<<<dim3(div_up(kpad, 2048), div_up(rows, kConvPairs)), 256, 0, c->stream>>>(
          c->ldN, c0, len, kpad, t.gram_cells, plane_b, rows, pairs, D, rOm, sc_p, t.g_b, t.cols);
      GPL_LAUNCHED(c, "k_crt_conv_pairs");
      if ((rc = crt_gemm(c, t.map_ga, t.map_gb, c->J, rows, t.Jp, t.Pp, len, t.g_out, plane_o, t.Pp, t.cols))) return rc;
      k_crt_t<<<dim3(c->J, div_up(rows, 1024)), 256, 0, c->stream>>>(c->J, c->P, c->n_d, rows, t.Pp, plane_o, t.g_out,
                                                                    inv_j, inv_p, c->dcol_d, c0 == 0,
                                                                    0.58 * R / crt_share(c->N) * c->N / len, root,
                                                                    gg + (size_t)l0 * c->J,
                                                                    T + (size_t)l0 * c->J * c->P, t.cols);
      GPL_LAUNCHED(c, "k_crt_t");
    }
  }
  std::vector<int> out(1 + tiles);
  GPL_TRY(c, cudaMemcpyAsync(out.data(), t.cols, sizeof(int) * out.size(), cudaMemcpyDeviceToHost, c->stream));
  if ((rc = crt_error_flag(c))) return rc;  // waits for the stream
  *left = out[0] ? 2 : std::find(out.begin(), out.end(), 1) != out.end() ? 1 : 0;
  return GPL_OK;
}

// GPL_ERR_TIMEOUT if a wait of the integer product gave up.
int crt_error_flag(Ctx* c) {
  if (!c->pr.crt.on || !c->pr.crt.err) return GPL_OK;
  int flag = 0;
  GPL_TRY(c, cudaMemcpyAsync(&flag, c->pr.crt.err, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
  GPL_TRY(c, cudaStreamSynchronize(c->stream));
  if (flag) {
    c->err = "tensor-core kernel gave up waiting (code " + std::to_string(flag) + ")";
    return GPL_ERR_TIMEOUT;
  }
  return GPL_OK;
}

}  // namespace gpl
