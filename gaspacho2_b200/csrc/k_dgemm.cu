// FP64 tensor-core (DMMA, mma.sync m16n8k4 .f64) forms of the two dominant contractions of
// the plain FP64 path. Both are written over the unique column pairs (a <= b) of the dense
// model columns, which turns the per-gene P x P products into two plain GEMMs and uses the
// symmetry of Psi_j and Psi_j^{-1} to halve the work.
//
//   k_pair_products  A[i, p] = D_ia D_ib / Omega_i for a range of cells, row-major with the
//                 pairs contiguous (the layout of V): the Gram's K-major A operand, written once
//                 per range (N * pairs doubles in all; a few ms of HBM writes per Gram).
//   k_pair_gram   G[p, j] = sum_i A[i, p] W_ij over a range of cells (M = pairs, N = genes,
//                 K = cells), both operands by cp.async (three stages, one barrier per slice),
//                 written straight into Psi_j (both triangles, plus DeltaInv) at model columns
//                 (dcol a, dcol b) when one range covers all cells: the dense block of getPsi
//                 (ggplvm.cu:621-680); otherwise added up range by range in a pairs x genes
//                 buffer that k_pair_scatter moves into Psi. Work: N*J*n_d*(n_d+1) flops.
//                 Behind the integer form (k_crt.cu) these three run for the genes that it left.
//   k_pair_v      V[i, p] = (1/Omega_i) sum_j W_ij S_j[a, b] for a cell range, S_j = Psi_j^{-1}
//                 gathered per pair (k_gather_spair). M = cells, N = pairs, K = genes; both
//                 operands by cp.async. Work: N*J*n_d*(n_d+1) flops.
//   k_v_to_u      U[i, a] = sum_b D_ib V[i, pair(a, b)]: the gradient contraction
//                 sum_j O_ij S_j[DD] d_i of getGradLogOmega (ggplvm.cu:301-376) from V.
//
// CTA tile 128 x 128 x 16 (K; the Gram also 64 x 64 and 64 x 16), 8 warps as 2 (M) x 4 (N), warp tile 64 x 32
// (4 x 4 DMMA tiles of 16 x 8), three-stage cp.async pipelines with one barrier per slice. m16n8k4 fragments (lane = 4*g + t):
// A 16x4 row-major a0 = A[g][t], a1 = A[g+8][t]; B 4x8 b0 = B[t][g]; C 16x8
// c0,c1 = C[g][2t, 2t+1], c2,c3 = C[g+8][2t, 2t+1]. Shared rows are padded so that the
// 16 lanes of each half-warp hit 16 distinct 8-byte bank pairs.
#include <algorithm>
#include <climits>
#include <cstdlib>

#include "dmma_common.cuh"
#include "gpl_internal.cuh"
#include "pair_rows.cuh"

namespace gpl {

namespace {
constexpr int BM = 128, BN = 128, BK = 16;
constexpr int SA = BM + 4;   // As[k][m]
constexpr int SBT = BK + 4;  // Bs[n][k] (weights, k contiguous)
constexpr int SBN = BN + 4;  // Bs[k][n] (S pairs, n contiguous)
constexpr int kThreads = 256;
}  // namespace

// Grouped tile order: a 1-D grid of tm x tn output tiles in which consecutive blocks walk
// group_m tile rows down one tile column before moving to the next column, so that the ~148
// resident blocks cover a group_m x ~(148 / group_m) patch and share both operands' tiles
// through L2 (row-major order would re-read one operand from DRAM for nearly every block).
// group_m is the autotuner's choice (default 12); it changes only which block computes which
// tile, never a tile's sums.
constexpr int kGroupM = 12;
__device__ __forceinline__ int2 grouped_tile(int id, int tm, int tn, int group_m) {
  const int per = group_m * tn;
  const int grp = id / per, first = grp * group_m;
  const int gm = min(tm - first, group_m);
  const int r = id - grp * per;
  return make_int2(first + r % gm, r / gm);
}

// One 16-deep K slice of the 64 x 32 warp tile, both operands stored [k][..].
__device__ __forceinline__ void warp_slice(const double* __restrict__ As, const double* __restrict__ Bs, int wm,
                                           int wn, int g, int t, double (&acc)[4][4][4]) {
#pragma unroll
  for (int kk = 0; kk < BK / 4; kk++) {
    double a[4][2], b[4];
    const double* ar = As + (kk * 4 + t) * SA + wm * 64 + g;
#pragma unroll
    for (int mt = 0; mt < 4; mt++) {
      a[mt][0] = ar[mt * 16];
      a[mt][1] = ar[mt * 16 + 8];
    }
#pragma unroll
    for (int nt = 0; nt < 4; nt++) {
      const int n = wn * 32 + nt * 8 + g;
      b[nt] = Bs[(kk * 4 + t) * SBN + n];
    }
#pragma unroll
    for (int mt = 0; mt < 4; mt++)
#pragma unroll
      for (int nt = 0; nt < 4; nt++) dmma_16x8x4(acc[mt][nt], a[mt][0], a[mt][1], b[nt]);
  }
}

// ---------------------------------------------------------------------------------------------
// Gram over the dense column pairs
// ---------------------------------------------------------------------------------------------
// A[(i - c0) * pairs_pad + p] for cells [c0, c1): 8 cells per block, their dense-column
// values and 1/Omega staged in shared memory, stores along the pairs (coalesced). Padding
// pairs and cells past N (1/Omega = 0 there) give 0.
constexpr int kProdCells = 8;

__global__ void __launch_bounds__(256) k_pair_products(int ldN, int n_d, int c0, int c1, int n_pairs, int pairs_pad,
                                                       const int2* __restrict__ pairs, const double* __restrict__ D,
                                                       const double* __restrict__ rOm, double* __restrict__ A,
                                                       const int* __restrict__ state) {
  extern __shared__ double dsh[];  // [n_d][kProdCells] then rOm[kProdCells]
  if (state && !state[0] && !state[1]) return;  // no gene on the list (GramGenes)
  for (int i0 = c0 + blockIdx.x * kProdCells; i0 < c1; i0 += gridDim.x * kProdCells) {
    __syncthreads();
    const int nc = min(kProdCells, c1 - i0);
    for (int e = threadIdx.x; e < n_d * kProdCells; e += blockDim.x) {
      const int a = e / kProdCells, r = e - a * kProdCells;
      dsh[e] = r < nc ? D[(size_t)a * ldN + i0 + r] : 0.0;
    }
    if (threadIdx.x < kProdCells) dsh[n_d * kProdCells + threadIdx.x] = threadIdx.x < nc ? rOm[i0 + threadIdx.x] : 0.0;
    __syncthreads();
    const double* ro = dsh + n_d * kProdCells;
    for (int p = threadIdx.x; p < pairs_pad; p += blockDim.x) {
      double v[kProdCells];
      if (p < n_pairs) {
        const int2 q = pairs[p];
        const double* da = dsh + q.x * kProdCells;
        const double* db = dsh + q.y * kProdCells;
#pragma unroll
        for (int r = 0; r < kProdCells; r++) v[r] = da[r] * db[r] * ro[r];
      } else {
#pragma unroll
        for (int r = 0; r < kProdCells; r++) v[r] = 0.0;
      }
      for (int r = 0; r < nc; r++) A[(size_t)(i0 - c0 + r) * pairs_pad + p] = v[r];
    }
  }
}

// epilogue modes of k_pair_gram
constexpr int kGramPsi = 0;  // one range: Psi_j[mk, ml] = Psi_j[ml, mk] = G + DeltaInv
constexpr int kGramSet = 1;  // first of several ranges: Gacc[p * J + j] = G
constexpr int kGramAdd = 2;  // later ranges: Gacc[p * J + j] += G

// Output tiles of TM pairs x TN genes, WM x WN warps. A CTA's time is its tile's multiply-adds for every cell,
// so few pairs or genes, or a last wave that is nearly empty, want small tiles (launch_pair_gram). An entry is one
// chain of DMMAs over the cells, whatever the tile, or (kRuns, the small tiles outside an OrderScope) the sum of
// chains of 128 cells, whose rounding is what is left of the chain's: 4e-16 to 6e-16 of the diagonal (rms) at 1,274
// to 2,000 cells, 6e-17 in runs, in the same time.
template <int TM, int TN>
struct GramTile {
  static constexpr int WM = TM / TN >= 4 ? 4 : 2, WN = 8 / WM;
  static constexpr int MT = TM / WM / 16, NT = TN / WN / 8;
  static constexpr int SAm = TM + 4;  // As[k][m], 4 mod 16
  static constexpr int smem = (int)sizeof(double) * 3 * (BK * SAm + TN * SBT);
};

// The genes that a launch takes: all of them, or those on the list that the integer form left (CrtState):
// state[0] all, state[1] how many. Launches for few and for many of them stand one behind the other
// (lo <= count < hi), as the count is not known to the host.
struct GramGenes {
  const int *state, *list;
  int lo, hi;
  __device__ __forceinline__ int count(int J) const { return !state || state[0] ? J : state[1]; }
  __device__ __forceinline__ int gene(int k) const { return !state || state[0] ? k : list[k]; }
};

template <int TM, int TN, bool kRuns>
__global__ void __launch_bounds__(kThreads, TM == 128 ? 1 : kRuns && TN == 64 ? 2 : 3)
    k_pair_gram(int N, int ldN, int J, int P, int c0, int c1, int pairs_pad, int n_pairs, int mode,
                const double* __restrict__ A, const int2* __restrict__ pairs, const int* __restrict__ dcol,
                const double* __restrict__ W, const double* __restrict__ Dinv, double* __restrict__ Psi,
                double* __restrict__ Gacc, int group_m, GramGenes genes) {
  using G = GramTile<TM, TN>;
  constexpr int SAm = G::SAm, MT = G::MT, NT = G::NT;
  extern __shared__ __align__(16) double smem_d[];
  const int n_j = genes.count(J);
  if (n_j < genes.lo || n_j >= genes.hi) return;
  double* As = smem_d;               // [3][BK][SAm]  pair products (pairs contiguous)
  double* Bs = As + 3 * BK * SAm;    // [3][TN][SBT]  weights (cells contiguous)
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3, wm = warp / G::WN, wn = warp % G::WN;
  const int tm = (n_pairs + TM - 1) / TM, tn = (n_j + TN - 1) / TN;
  const int nsl = (c1 - c0 + BK - 1) / BK;
  for (int id = blockIdx.x; id < tm * tn; id += gridDim.x) {
    const int2 tile = grouped_tile(id, tm, tn, group_m);
    const int p0 = tile.x * TM, j0 = tile.y * TN;
    // the weights' rows that this thread copies
    constexpr int kRowsB = (TN * BK / 2 + kThreads - 1) / kThreads;
    const double* rows_b[kRowsB];
#pragma unroll
    for (int r = 0; r < kRowsB; r++)
      rows_b[r] = W + (size_t)genes.gene(min(j0 + ((tid + r * kThreads) >> 3), n_j - 1)) * ldN;
    __syncthreads();  // the last tile's slices are read

    // slice s: cells [c0 + 16 s, c0 + 16 s + 16) of both operands (16-byte copies; rows of A
    // past the range and weights past N arrive as zeros)
    auto load = [&](int s, int st) {
      const int kb = s * BK;
#pragma unroll
      for (int r = 0; r < (TM * BK / 2) / kThreads; r++) {
        const int ch = tid + r * kThreads;
        const int k = ch / (TM / 2), part = ch % (TM / 2);
        const int row = kb + k;
        const int nb = (c0 + row < c1) ? 16 : 0;
        const double* src = A + (size_t)min(row, c1 - c0 - 1) * pairs_pad + p0 + part * 2;
        cp_async16(As + st * BK * SAm + k * SAm + part * 2, src, nb);
      }
#pragma unroll
      for (int r = 0; r < kRowsB; r++) {
        const int ch = tid + r * kThreads;
        if (TN * BK / 2 < kThreads && ch >= TN * BK / 2) break;
        const int n = ch >> 3, part = ch & 7;
        const int j = j0 + n, i = c0 + kb + part * 2;
        const int nb = (j < n_j) ? 8 * max(0, min(2, min(N, c1) - i)) : 0;
        const double* src = rows_b[r] + min(i, ldN - 2);
        cp_async16(Bs + st * TN * SBT + n * SBT + part * 2, src, nb);
      }
    };

    double acc[MT][NT][4], sum[MT][NT][4];
#pragma unroll
    for (int x = 0; x < MT; x++)
#pragma unroll
      for (int y = 0; y < NT; y++)
#pragma unroll
        for (int z = 0; z < 4; z++) acc[x][y][z] = sum[x][y][z] = 0.0;

    // three stages, one barrier per slice (as k_pair_v)
    load(0, 0);
    cp_async_commit();
    if (nsl > 1) load(1, 1);
    cp_async_commit();
    for (int s = 0; s < nsl; s++) {
      cp_async_wait<1>();  // slice s landed
      __syncthreads();
      if (s + 2 < nsl) load(s + 2, (s + 2) % 3);
      cp_async_commit();
      const double* as = As + (s % 3) * BK * SAm;
      const double* bs = Bs + (s % 3) * TN * SBT;
#pragma unroll
      for (int kk = 0; kk < BK / 4; kk++) {
        double a[MT][2], b[NT];
        const double* ar = as + (kk * 4 + t) * SAm + wm * MT * 16 + g;
#pragma unroll
        for (int mt = 0; mt < MT; mt++) {
          a[mt][0] = ar[mt * 16];
          a[mt][1] = ar[mt * 16 + 8];
        }
#pragma unroll
        for (int nt = 0; nt < NT; nt++) b[nt] = bs[(wn * NT * 8 + nt * 8 + g) * SBT + kk * 4 + t];
#pragma unroll
        for (int mt = 0; mt < MT; mt++)
#pragma unroll
          for (int nt = 0; nt < NT; nt++) dmma_16x8x4(acc[mt][nt], a[mt][0], a[mt][1], b[nt]);
      }
      if (kRuns && ((s & 7) == 7 || s + 1 == nsl)) {
#pragma unroll
        for (int x = 0; x < MT; x++)
#pragma unroll
          for (int y = 0; y < NT; y++)
#pragma unroll
            for (int z = 0; z < 4; z++) {
              sum[x][y][z] += acc[x][y][z];
              acc[x][y][z] = 0.0;
            }
      }
    }
    cp_async_wait<0>();

#pragma unroll
    for (int mt = 0; mt < MT; mt++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int p = p0 + (wm * MT + mt) * 16 + g + h * 8;
        if (p >= n_pairs) continue;
        size_t mk = 0, ml = 0;
        double dv = 0.0;
        if (mode == kGramPsi) {
          const int2 q = pairs[p];
          mk = dcol[q.x];
          ml = dcol[q.y];
          dv = Dinv[mk + ml * P];
        }
#pragma unroll
        for (int nt = 0; nt < NT; nt++)
#pragma unroll
          for (int e = 0; e < 2; e++) {
            if (j0 + (wn * NT + nt) * 8 + 2 * t + e >= n_j) continue;
            const int j = genes.gene(j0 + (wn * NT + nt) * 8 + 2 * t + e);
            const double v = kRuns ? sum[mt][nt][h * 2 + e] : acc[mt][nt][h * 2 + e];
            if (mode == kGramPsi) {
              double* Pj = Psi + (size_t)j * P * P;
              Pj[mk + ml * P] = v + dv;
              Pj[ml + mk * P] = v + dv;
            } else if (mode == kGramSet) {
              Gacc[(size_t)p * J + j] = v;
            } else {
              Gacc[(size_t)p * J + j] += v;
            }
          }
      }
  }
}

// Psi_j[mk, ml] = Psi_j[ml, mk] = Gacc[p * J + j] + DeltaInv[mk, ml] after several ranges
__global__ void k_pair_scatter(int J, int P, int n_pairs, const int2* __restrict__ pairs,
                               const int* __restrict__ dcol, const double* __restrict__ Gacc,
                               const double* __restrict__ Dinv, double* __restrict__ Psi, GramGenes genes) {
  const int n_j = genes.count(J), p = blockIdx.x;
  if (n_j == 0) return;
  const int2 q = pairs[p];
  const size_t mk = dcol[q.x], ml = dcol[q.y];
  const double dv = Dinv[mk + ml * P];
  for (int k = threadIdx.x; k < n_j; k += blockDim.x) {
    const int j = genes.gene(k);
    const double v = Gacc[(size_t)p * J + j] + dv;
    double* Pj = Psi + (size_t)j * P * P;
    Pj[mk + ml * P] = v;
    Pj[ml + mk * P] = v;
  }
}

__global__ void k_recip_omega(int N, int cpad, const double* __restrict__ Omega, double* __restrict__ rOm) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < cpad) rOm[i] = i < N ? 1.0 / Omega[i] : 0.0;
}

// ---------------------------------------------------------------------------------------------
// Gradient contraction over the pairs
// ---------------------------------------------------------------------------------------------
// Spair[j][p] = S_j[dcol a_p, dcol b_p] (0 for the padding pairs)
__global__ void k_gather_spair(int J, int P, int n_pairs, int pairs_pad, const int2* __restrict__ pairs,
                               const int* __restrict__ dcol, const double* __restrict__ S,
                               double* __restrict__ Sp) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= pairs_pad) return;
  int2 q = make_int2(0, 0);
  const bool live = p < n_pairs;
  if (live) q = pairs[p];
  const size_t off = live ? (size_t)dcol[q.x] + (size_t)dcol[q.y] * P : 0;
  for (int j = blockIdx.y; j < J; j += gridDim.y)
    Sp[(size_t)j * pairs_pad + p] = live ? S[(size_t)j * P * P + off] : 0.0;
}

__global__ void __launch_bounds__(kThreads, 1)
    k_pair_v(int N, int ldN, int J, int c0, int c1, int pairs_pad, const double* __restrict__ W,
             const double* __restrict__ Sp, const double* __restrict__ rOm, double* __restrict__ V, int group_m,
             const int* __restrict__ cells) {
  extern __shared__ __align__(16) double smem_d[];
  double* As = smem_d;                // [3][BK][SA]  W rows (cells contiguous)
  double* Bs = smem_d + 3 * BK * SA;  // [3][BK][SBN] S pairs (pairs contiguous)
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3, wm = warp >> 2, wn = warp & 3;
  const int nsl = (J + BK - 1) / BK, tm = (c1 - c0 + BM - 1) / BM, tn = pairs_pad / BN;
  for (int id = blockIdx.x; id < tm * tn; id += gridDim.x) {
    const int2 tile = grouped_tile(id, tm, tn, group_m);
    const int i0 = c0 + tile.x * BM, n0 = tile.y * BN;
    if (cells && !cells[0] && !cells[1 + i0 / BM]) continue;  // c0 is a multiple of BM
    __syncthreads();  // the last tile's slices are read

    auto load = [&](int s, int buf) {
      const int jb = s * BK;
#pragma unroll
      for (int r = 0; r < (BM * BK / 2) / kThreads; r++) {
        const int ch = tid + r * kThreads;
        const int k = ch >> 6, part = ch & 63;
        const int j = jb + k, i = i0 + part * 2;
        const int nb = (j < J) ? 8 * max(0, min(2, min(N, c1) - i)) : 0;
        const double* src = W + (size_t)min(j, J - 1) * ldN + min(max(i, 0), ldN - 2);
        cp_async16(As + buf * BK * SA + k * SA + part * 2, src, nb);
      }
#pragma unroll
      for (int r = 0; r < (BN * BK / 2) / kThreads; r++) {
        const int ch = tid + r * kThreads;
        const int k = ch >> 6, part = ch & 63;
        const int j = jb + k;
        const int nb = (j < J) ? 16 : 0;
        const double* src = Sp + (size_t)min(j, J - 1) * pairs_pad + n0 + part * 2;
        cp_async16(Bs + buf * BK * SBN + k * SBN + part * 2, src, nb);
      }
    };

    double acc[4][4][4];
#pragma unroll
    for (int x = 0; x < 4; x++)
#pragma unroll
      for (int y = 0; y < 4; y++)
#pragma unroll
        for (int z = 0; z < 4; z++) acc[x][y][z] = 0.0;

    // three stages, one barrier per slice: after the barrier of iteration s every warp is done
    // with slice s - 1, whose stage (s + 2) % 3 is refilled while slice s is multiplied
    load(0, 0);
    cp_async_commit();
    if (nsl > 1) load(1, 1);
    cp_async_commit();
    for (int s = 0; s < nsl; s++) {
      cp_async_wait<1>();  // slice s landed
      __syncthreads();
      if (s + 2 < nsl) load(s + 2, (s + 2) % 3);
      cp_async_commit();
      warp_slice(As + (s % 3) * BK * SA, Bs + (s % 3) * BK * SBN, wm, wn, g, t, acc);
    }
    cp_async_wait<0>();

#pragma unroll
    for (int mt = 0; mt < 4; mt++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int i = i0 + wm * 64 + mt * 16 + g + h * 8;
        if (i >= N || i >= c1) continue;
        const double r = rOm[i];
        double* vrow = V + (size_t)(i - c0) * pairs_pad + n0 + wn * 32 + 2 * t;
#pragma unroll
        for (int nt = 0; nt < 4; nt++) {
          double2 v = make_double2(acc[mt][nt][h * 2] * r, acc[mt][nt][h * 2 + 1] * r);
          *reinterpret_cast<double2*>(vrow + nt * 8) = v;
        }
      }
  }
}

// U[i, a] = sum_b D_ib V[i, pair(min(a,b), max(a,b))], W warps per cell (pair_rows.cuh), the cell's V row
// by asynchronous copies.
template <int S, int W>
__global__ void __launch_bounds__(256, S > 9 ? 2 : 4) k_v_to_u(int ldN, int n_d, int pairs_pad, int c0, int c1,
                                                   const double* __restrict__ D, const double* __restrict__ V,
                                                   double* __restrict__ U, const int* __restrict__ cells) {
  extern __shared__ __align__(16) double vs[];
  const int g = W == 8 ? 0 : threadIdx.x >> 5, r = blockIdx.x * (8 / W) + g;
  if (c0 + r >= c1) return;  // W = 1: a whole warp, no barrier of the block follows
  if (cells && !cells[0] && !cells[1 + (c0 + r) / BM]) return;
  double* vc = vs + g * u_space<W, false>(n_d);
  const double* vr = V + (size_t)r * pairs_pad;
  pair_rows_to_u<S, W, false>(c0 + r, ldN, n_d, vc, D, U, [&](int from, int p1, int tid, int nt) {
    for (int p = from + 2 * tid; p < p1; p += 2 * nt) cp_async16(vc + p - from, vr + p, 16);
    cp_async_commit();
    cp_async_wait<0>();
  });
}

// The same for more dense columns than that takes (512): the row is read from global memory (L1 / L2)
// instead of staged, the dense row of the cell is staged.
__global__ void __launch_bounds__(256) k_v_to_u_wide(int N, int ldN, int n_d, int pairs_pad, int c0, int c1,
                                                     const double* __restrict__ D, const double* __restrict__ V,
                                                     double* __restrict__ U) {
  extern __shared__ __align__(16) double ds[];  // D row of the cell
  for (int i = c0 + blockIdx.x; i < c1 && i < N; i += gridDim.x) {
    const double* vr = V + (size_t)(i - c0) * pairs_pad;
    for (int e = threadIdx.x; e < n_d; e += blockDim.x) ds[e] = D[(size_t)e * ldN + i];
    __syncthreads();
    for (int a = threadIdx.x; a < n_d; a += blockDim.x) {
      double s = 0.0;
      for (int b = 0; b < a; b++) s = fma(ds[b], __ldg(vr + b * n_d - b * (b - 1) / 2 + (a - b)), s);
      const double* row = vr + a * n_d - a * (a - 1) / 2 - a;
      for (int b = a; b < n_d; b++) s = fma(ds[b], __ldg(row + b), s);
      U[i + (size_t)a * ldN] = s;
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
int pair_prepare(Ctx* c) {
  PairState& s = c->pr;
  if (s.ready) return GPL_OK;
  const int n_d = c->n_d;
  std::vector<int2> pairs;
  for (int a = 0; a < n_d; a++)
    for (int b = a; b < n_d; b++) pairs.push_back(make_int2(a, b));
  s.n_pairs = (int)pairs.size();
  s.pairs_pad = (s.n_pairs + BN - 1) / BN * BN;
  s.cpad = (c->N + BM - 1) / BM * BM;
  // V (the gradient's V rows, or the Gram's pair products) holds a range of cells at a time:
  // all cells when that fits in 8 GiB (one range: the Gram writes Psi directly), else ranges
  // of at most 8 GiB. The option pair_range_cells sets a smaller range (tests of the multi-range path).
  const size_t row = (size_t)s.pairs_pad * sizeof(double);
  size_t cap = std::max<size_t>(BM, ((size_t)8 << 30) / row / BM * BM);
  if (c->pair_range_cells >= BM) cap = std::min<size_t>(cap, (size_t)c->pair_range_cells / BM * BM);
  s.v_cells = (int)std::min<size_t>((size_t)s.cpad, cap);
  s.smem_v = (int)sizeof(double) * 3 * (BK * SA + BK * SBN);
  // the integer form (k_crt.cu) keeps its operands in the same buffer, of 1 GiB at least: with 14 bytes
  // per operand entry it takes the cells in a few ranges where the DMMA form takes one, which costs it
  // less than a larger buffer costs a new context (about 10 ms per GiB)
  const size_t dmma_bytes = sizeof(double) * (size_t)s.v_cells * s.pairs_pad;
  crt_plan(c, std::max(dmma_bytes, (size_t)1 << 30));
  const size_t v_bytes = std::max(dmma_bytes, s.crt.bytes);
  if (cudaMalloc((void**)&s.pairs, sizeof(int2) * pairs.size()) != cudaSuccess ||
      cudaMalloc((void**)&s.rOm, sizeof(double) * s.cpad) != cudaSuccess ||
      cudaMalloc((void**)&s.Sp, sizeof(double) * (size_t)c->J * s.pairs_pad) != cudaSuccess ||
      cudaMalloc((void**)&s.V, v_bytes) != cudaSuccess) {
    cudaGetLastError();
    pair_release(c);
    c->err = "device allocation failed: pair GEMM buffers";
    return GPL_ERR_ALLOC;
  }
  GPL_TRY(c, cudaMemcpy(s.pairs, pairs.data(), sizeof(int2) * pairs.size(), cudaMemcpyHostToDevice));
  if (s.v_cells < c->N &&
      cudaMalloc((void**)&s.Gacc, sizeof(double) * (size_t)s.n_pairs * c->J) != cudaSuccess) {
    cudaGetLastError();
    pair_release(c);
    c->err = "device allocation failed: pair Gram accumulator";
    return GPL_ERR_ALLOC;
  }
  GPL_TRY(c, cudaFuncSetAttribute(k_pair_gram<128, 128, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  GramTile<128, 128>::smem));
  GPL_TRY(c, cudaFuncSetAttribute(k_pair_gram<64, 64, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  GramTile<64, 64>::smem));
  GPL_TRY(c, cudaFuncSetAttribute(k_pair_gram<64, 64, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  GramTile<64, 64>::smem));
  GPL_TRY(c, cudaFuncSetAttribute(k_pair_v, cudaFuncAttributeMaxDynamicSharedMemorySize, s.smem_v));
  const int rc = crt_prepare(c);
  if (rc) {
    pair_release(c);
    return rc;
  }
  s.ready = true;
  return GPL_OK;
}

void pair_release(Ctx* c) {
  graph_reset(c);
  PairState& s = c->pr;
  crt_release(c);
  void* bufs[] = {s.pairs, s.rOm, s.Sp, s.V, s.Gacc};
  for (void* p : bufs)
    if (p) cudaFree(p);
  s = PairState();
}

int recip_omega(Ctx* c, const double** rOm) {
  int rc = pair_prepare(c);
  if (rc) return rc;
  PairState& s = c->pr;
  *rOm = s.rOm;
  if (c->rOm_done) return GPL_OK;
  k_recip_omega<<<div_up(s.cpad, 256), 256, 0, c->stream>>>(c->N, s.cpad, c->Omega, s.rOm);
  GPL_LAUNCHED(c, "k_recip_omega");
  c->rOm_done = c->in_phase;
  return GPL_OK;
}

// The Gram's tile for n_pairs x J outputs, by its time per 16 cells: the tile's multiply-adds (64 per clock
// and SM) times the tiles an SM takes, at least 400 clocks of copies and barriers; the smaller tiles with a
// tenth for their operands' traffic.
static double gram_tile_cost(const Ctx* c, int n_pairs, int tm, int tn) {
  const double tiles = (double)div_up(n_pairs, tm) * div_up(c->J, tn);
  return std::ceil(tiles / c->sm_count) * std::max(tm * tn * 16 / 64, 400) * (tm < 128 ? 1.1 : 1.0);
}
static int gram_tile(const Ctx* c, int n_pairs, double* cost) {
  const double big = gram_tile_cost(c, n_pairs, 128, 128), mid = gram_tile_cost(c, n_pairs, 64, 64),
               small = gram_tile_cost(c, n_pairs, 64, 16);
  if (cost) *cost = std::min({big, mid, small});
  return big <= mid && big <= small ? 0 : mid <= small ? 1 : 2;
}
double pair_gram_cost(const Ctx* c, int n_pairs) {
  double cost;
  gram_tile(c, n_pairs, &cost);
  return cost;
}

int launch_pair_gram(Ctx* c) {
  const double* rOm = nullptr;
  int rc = recip_omega(c, &rOm);
  if (rc) return rc;
  PairState& s = c->pr;
  ProfScope ps(c, "gram");
  // the integer form, where it is planned; the kernels below then run for the genes that it left
  const bool crt = s.crt.gram_cells && !c->one_order;
  if (crt && (rc = launch_crt_gram(c))) return rc;
  const int* state = crt ? s.crt.genes : nullptr;
  const bool one = s.v_cells >= c->N;
  for (int c0 = 0; c0 < c->N; c0 += s.v_cells) {
    const int c1 = std::min(c->N, c0 + s.v_cells);
    const int smem_p = (int)sizeof(double) * (c->n_d + 1) * kProdCells;
    const int gp = div_up(c1 - c0, kProdCells);
    k_pair_products<<<crt ? std::min(gp, 8 * c->sm_count) : gp, 256, smem_p, c->stream>>>(
        c->ldN, c->n_d, c0, c1, s.n_pairs, s.pairs_pad, s.pairs, c->Dm, s.rOm, s.V, state);
    GPL_LAUNCHED(c, "k_pair_products");
    const int mode = one ? kGramPsi : (c0 == 0 ? kGramSet : kGramAdd);
    Tunable* tu = nullptr;
    const int gm = crt ? kGroupM : tune_pick(c, "pair_gram", {8, 12, 16}, kGroupM, &tu);
    TuneScope ts(c, one ? tu : nullptr);
    auto run = [&](auto tm, auto tn, int most, const GramGenes& genes) {
      constexpr int TM = decltype(tm)::value, TN = decltype(tn)::value;
      auto* fn = TM == 128 || c->one_order ? k_pair_gram<TM, TN, false> : k_pair_gram<TM, TN, TM != 128>;
      fn<<<std::min(most, div_up(s.n_pairs, TM) * div_up(c->J, TN)), kThreads, GramTile<TM, TN>::smem,
                            c->stream>>>(c->N, c->ldN, c->J, c->P, c0, c1, s.pairs_pad, s.n_pairs, mode, s.V, s.pairs,
                                         c->dcol_d, c->W, c->DeltaInv, c->Psi, s.Gacc, gm, genes);
    };
    using std::integral_constant;
    constexpr integral_constant<int, 128> n128;
    constexpr integral_constant<int, 64> n64;
    constexpr integral_constant<int, 16> n16;
    const int all = INT_MAX, resident = 3 * c->sm_count;
    if (crt) {  // up to 48 genes in tiles of 16
      run(n64, n16, resident, GramGenes{state, s.crt.list, 1, 49});
      GPL_LAUNCHED(c, "k_pair_gram");
      run(n64, n64, resident, GramGenes{state, s.crt.list, 49, all});
    } else {
      const GramGenes genes{nullptr, nullptr, 0, all};
      const int form = gram_tile(c, s.n_pairs, nullptr);
      if (form == 0) run(n128, n128, all, genes);
      else if (form == 1) run(n64, n64, all, genes);
      else run(n64, n16, all, genes);
    }
    GPL_LAUNCHED(c, "k_pair_gram");
  }
  if (!one) {
    k_pair_scatter<<<s.n_pairs, 256, 0, c->stream>>>(c->J, c->P, s.n_pairs, s.pairs, c->dcol_d, s.Gacc,
                                                    c->DeltaInv, c->Psi, GramGenes{state, s.crt.list, 0, INT_MAX});
    GPL_LAUNCHED(c, "k_pair_scatter");
  }
  return GPL_OK;
}

int launch_pair_uq(Ctx* c) {
  const double* rOm = nullptr;
  int rc = recip_omega(c, &rOm);
  if (rc) return rc;
  PairState& s = c->pr;
  {
    ProfScope ps(c, "spair");
    dim3 g(div_up(s.pairs_pad, 256), std::min(c->J, 65535));
    k_gather_spair<<<g, 256, 0, c->stream>>>(c->J, c->P, s.n_pairs, s.pairs_pad, s.pairs, c->dcol_d, c->PsiInv,
                                             s.Sp);
    GPL_LAUNCHED(c, "k_gather_spair");
  }
  // the integer form, where it is planned; the kernels below then run for the tiles of cells that it sent here
  const int* cells = s.crt.grad_cells ? s.crt.cells : nullptr;
  if (cells && (rc = launch_crt_uq(c))) return rc;
  for (int c0 = 0; c0 < c->N; c0 += s.v_cells) {
    const int c1 = std::min(c->N, c0 + s.v_cells);
    {
      ProfScope ps(c, "uq");
      // behind the integer form most tiles have nothing to do: a block per SM walks them (thousands of blocks
      // that return at once took 0.19 ms at 100,000 cells x 8,778 pairs)
      const int tiles = div_up(c1 - c0, BM) * (s.pairs_pad / BN), g = cells ? std::min(tiles, c->sm_count) : tiles;
      Tunable* tu = nullptr;
      const int gm = cells ? kGroupM : tune_pick(c, "pair_v", {8, 12, 16}, kGroupM, &tu);
      TuneScope ts(c, c1 - c0 == c->N ? tu : nullptr);
      k_pair_v<<<g, kThreads, s.smem_v, c->stream>>>(c->N, c->ldN, c->J, c0, c1, s.pairs_pad, c->W, s.Sp, s.rOm,
                                                     s.V, gm, cells);
      GPL_LAUNCHED(c, "k_pair_v");
    }
    if ((rc = launch_v_to_u_rows(c, c0, c1, c->Dm, s.V, cells))) return rc;
  }
  return GPL_OK;
}

int launch_v_to_u_cells(Ctx* c, int c0, int c1, const double* D) {
  return launch_v_to_u_rows(c, c0, c1, D, c->pr.V, nullptr);
}

int launch_v_to_u_rows(Ctx* c, int c0, int c1, const double* D, const double* V, const int* cells) {
  PairState& s = c->pr;
  ProfScope ps(c, "v_to_u");
  if (c->n_d > kUMaxDense) {
    const int grid = std::min(c1 - c0, 8 * c->sm_count);
    k_v_to_u_wide<<<grid, 256, sizeof(double) * c->n_d, c->stream>>>(c->N, c->ldN, c->n_d, s.pairs_pad, c0, c1, D,
                                                                    V, c->U);  // never gated: crt_plan
    GPL_LAUNCHED(c, "k_v_to_u_wide");
    return GPL_OK;
  }
  const int len = std::min(c1, c->N) - c0;
  pair_rows_form(c->n_d, len, 160, [&](auto S, auto W) {
    constexpr int per = 8 / W;
    const int smem = (int)sizeof(double) * u_space<W, false>(c->n_d) * per;
    if (smem > 48 * 1024)  // 97 or more columns, a warp per cell
      cudaFuncSetAttribute(k_v_to_u<S, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    k_v_to_u<S, W><<<div_up(len, per), 256, smem, c->stream>>>(c->ldN, c->n_d, s.pairs_pad, c0, c0 + len, D, V, c->U,
                                                              cells);
  });
  GPL_LAUNCHED(c, "k_v_to_u");
  return GPL_OK;
}

// ---------------------------------------------------------------------------------------------
// Linear predictor over the dense columns (option eta_tc)
// ---------------------------------------------------------------------------------------------
// out[j * ldN + i] = D_i . B_j[dcol] + Lv[group(i), j] for 128-cell x 128-gene tiles, where
// Lv[g, j] is the sum of gene j's coefficients of the levels of cell group g (k_level_sums, per
// launch; genes contiguous in rows of ldJ, even, so that a lane reads its two genes' sums as one
// 16-byte load and the eight cells of a quad row touch at most eight lines): K = the dense columns in 16-deep slices (DMMA steps past n_d skipped), A = D by
// 16-byte cp.async (cells contiguous), B = the genes' dense coefficients gathered through dcol by
// 8-byte cp.async (k contiguous in shared memory). Persistent: one CTA per SM walks the tiles
// cell-tile-major with a stride of the grid, so the CTAs resident at any time share a few cell
// tiles of D and all of B through L2; the next tile's first two slices are in flight while the
// current tile's epilogue stores (evict-first) run. The weights that follow (W, Nu) are an
// element-wise pass of their own: inside this kernel's epilogue, at one CTA per SM, the
// dependent FP64 operations of exp() left the tensor pipe idle for most of the launch.
struct EtaArgs {
  int N, ldN, P, J, ldJ, n_d, n_grp;
  const double *D, *B, *lvt;
  const int *dcol, *gid;
  double* out;
};

// Lv[g * ldJ + j] = sum over the grouped variables v (in order) of B[cv_nh[v] + level + j * P]
__global__ void k_level_sums(int J, int ldJ, int n_grp, int n_cv, int P, const int* __restrict__ cv_nh,
                             const int* __restrict__ glev, const double* __restrict__ B, double* __restrict__ Lv) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (int64_t)J * n_grp) return;
  const int g = (int)(e / J), j = (int)(e - (int64_t)g * J);
  double s = 0.0;
  for (int v = 0; v < n_cv; v++) s += B[cv_nh[v] + glev[(size_t)g * n_cv + v] + (size_t)j * P];
  Lv[(size_t)g * ldJ + j] = s;
}

// One 16-deep K slice of a warp tile of MT x 16 cells x 32 genes (A rows of stride sa), with only
// the first nkk of its four k4 steps live when kLive.
template <int MT, bool kLive>
__device__ __forceinline__ void warp_slice_eta(const double* __restrict__ As, const double* __restrict__ Bs, int sa,
                                               int wm, int wn, int g, int t, int nkk, double (&acc)[MT][4][4]) {
#pragma unroll
  for (int kk = 0; kk < BK / 4; kk++) {
    if (kLive && kk >= nkk) break;
    double av[MT][2], b[4];
    const double* ar = As + (kk * 4 + t) * sa + wm * (MT * 16) + g;
#pragma unroll
    for (int mt = 0; mt < MT; mt++) {
      av[mt][0] = ar[mt * 16];
      av[mt][1] = ar[mt * 16 + 8];
    }
#pragma unroll
    for (int nt = 0; nt < 4; nt++) b[nt] = Bs[(wn * 32 + nt * 8 + g) * SBT + kk * 4 + t];
#pragma unroll
    for (int mt = 0; mt < MT; mt++)
#pragma unroll
      for (int nt = 0; nt < 4; nt++) dmma_16x8x4(acc[mt][nt], av[mt][0], av[mt][1], b[nt]);
  }
}

// Tiles of MT x 32 cells x 128 genes: MT = 4 (128 cells, one CTA per SM) or MT = 2 (64 cells, two
// CTAs per SM, so that one CTA's epilogue overlaps the other's MMAs). Every output is the same
// sum in the same order in both, so the autotuner may pick either.
template <int MT>
size_t eta_smem_bytes(int n_d) {
  const int KP = (n_d + BK - 1) / BK * BK;
  return sizeof(double) * (3 * BK * (MT * 32 + 4) + 3 * BN * SBT) + sizeof(int) * (size_t)KP;
}

template <int MT>
__global__ void __launch_bounds__(kThreads, MT == 2 ? 2 : 1) k_eta_dmma(const EtaArgs a) {
  constexpr int BMt = MT * 32, SAt = BMt + 4;
  extern __shared__ __align__(16) double smem_d[];
  double* As = smem_d;             // [3][BK][SAt] D rows (cells contiguous)
  double* Bs = As + 3 * BK * SAt;  // [3][BN][SBT] dense coefficients (k contiguous)
  const int KP = (a.n_d + BK - 1) / BK * BK;
  int* dcs = reinterpret_cast<int*>(Bs + 3 * BN * SBT);  // [KP] dcol, 0 past n_d
  const double* __restrict__ D = a.D;
  const double* __restrict__ B = a.B;
  const double* __restrict__ lvt = a.lvt;
  const int* __restrict__ gid = a.gid;
  double* __restrict__ out = a.out;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3, wm = warp >> 2, wn = warp & 3;
  const int tm = (a.N + BMt - 1) / BMt, tn = (a.J + BN - 1) / BN;
  const int tiles = tm * tn, nsl = KP / BK;
  for (int k = tid; k < KP; k += kThreads) dcs[k] = k < a.n_d ? a.dcol[k] : 0;
  __syncthreads();

  // slice s of the tile at (m0, j0) into stage st
  auto load = [&](int m0, int j0, int s, int st) {
    const int kb = s * BK;
#pragma unroll
    for (int r = 0; r < (BMt * BK / 2) / kThreads; r++) {
      const int ch = tid + r * kThreads;
      const int k = ch / (BMt / 2), part = ch % (BMt / 2);
      const int col = kb + k, i = m0 + part * 2;
      const int nb = (col < a.n_d && i < a.ldN) ? 16 : 0;  // ldN is even: a chunk is in or out whole
      const double* src = D + (size_t)min(col, a.n_d - 1) * a.ldN + min(i, a.ldN - 2);
      cp_async16(As + st * BK * SAt + k * SAt + part * 2, src, nb);
    }
#pragma unroll
    for (int r = 0; r < (BN * BK) / kThreads; r++) {
      const int ch = tid + r * kThreads;
      const int n = ch >> 4, k = ch & 15;
      const int col = kb + k, j = j0 + n;
      const int nb = (col < a.n_d && j < a.J) ? 8 : 0;
      const double* src = B + dcs[col] + (size_t)min(j, a.J - 1) * a.P;
      cp_async8(Bs + st * BN * SBT + n * SBT + k, src, nb);
    }
  };

  int base = 0;  // slices issued before this tile (stage of slice s = (base + s) % 3)
  int w = blockIdx.x;
  if (w < tiles) {
    const int m0 = (w / tn) * BMt, j0 = (w % tn) * BN;
    load(m0, j0, 0, 0);
    cp_async_commit();
    if (nsl > 1) load(m0, j0, 1, 1);
    cp_async_commit();
  }
  for (; w < tiles; w += gridDim.x) {
    const int m0 = (w / tn) * BMt, j0 = (w % tn) * BN;
    double acc[MT][4][4];
#pragma unroll
    for (int x = 0; x < MT; x++)
#pragma unroll
      for (int y = 0; y < 4; y++)
#pragma unroll
        for (int z = 0; z < 4; z++) acc[x][y][z] = 0.0;
    for (int s = 0; s < nsl; s++) {
      cp_async_wait<1>();  // slice s landed
      __syncthreads();
      if (s + 2 < nsl) load(m0, j0, s + 2, (base + s + 2) % 3);
      cp_async_commit();
      const int st = (base + s) % 3;
      if (s + 1 < nsl) {
        warp_slice_eta<MT, false>(As + st * BK * SAt, Bs + st * BN * SBT, SAt, wm, wn, g, t, 4, acc);
      } else {  // the last slice: only the k4 steps that reach a dense column
        const int nkk = min(BK / 4, (a.n_d - s * BK + 3) / 4);
        warp_slice_eta<MT, true>(As + st * BK * SAt, Bs + st * BN * SBT, SAt, wm, wn, g, t, nkk, acc);
      }
    }
    // the next tile's first two slices go to the two stages that no warp reads any more
    base += nsl;
    const int wn2 = w + gridDim.x;
    if (wn2 < tiles) {
      const int m1 = (wn2 / tn) * BMt, j1 = (wn2 % tn) * BN;
      load(m1, j1, 0, base % 3);
      cp_async_commit();
      if (nsl > 1) load(m1, j1, 1, (base + 1) % 3);
      cp_async_commit();
    }
    // the cells' level sums, then the stores
    if (a.n_grp > 0) {
#pragma unroll
      for (int mt = 0; mt < MT; mt++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int i = min(m0 + wm * (MT * 16) + mt * 16 + g + h * 8, a.N - 1);
          const double* lg = lvt + (size_t)gid[i] * a.ldJ;
#pragma unroll
          for (int nt = 0; nt < 4; nt++) {
            // genes j, j + 1 (j even); past J only columns that are never stored
            const int j = min(j0 + wn * 32 + nt * 8 + 2 * t, a.ldJ - 2);
            const double2 v = *reinterpret_cast<const double2*>(lg + j);
            acc[mt][nt][h * 2] += v.x;
            acc[mt][nt][h * 2 + 1] += v.y;
          }
        }
    }
#pragma unroll
    for (int mt = 0; mt < MT; mt++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int i = m0 + wm * (MT * 16) + mt * 16 + g + h * 8;
        if (i >= a.N) continue;
#pragma unroll
        for (int nt = 0; nt < 4; nt++)
#pragma unroll
          for (int e = 0; e < 2; e++) {
            const int j = j0 + wn * 32 + nt * 8 + 2 * t + e;
            if (j < a.J) __stcs(out + (size_t)j * a.ldN + i, acc[mt][nt][h * 2 + e]);
          }
      }
  }
  cp_async_wait<0>();
}

int launch_eta_dmma(Ctx* c, const double* B, double* out) {
  if (eta_smem_bytes<4>(c->n_d) > 227 * 1024) {
    c->err = "too many dense columns for the linear-predictor kernel";
    return GPL_ERR_LIMIT;
  }
  if (c->n_grp > 0) {
    const int64_t n = (int64_t)c->J * c->n_grp;
    k_level_sums<<<(unsigned)div_up(n, 256), 256, 0, c->stream>>>(c->J, lvt_ld(c->J), c->n_grp, c->n_cv, c->P,
                                                                 c->cv_nh_d, c->glev_d, B, c->lvt);
    GPL_LAUNCHED(c, "k_level_sums");
  }
  EtaArgs a{};
  a.N = c->N;
  a.ldN = c->ldN;
  a.P = c->P;
  a.J = c->J;
  a.ldJ = lvt_ld(c->J);
  a.n_d = c->n_d;
  a.n_grp = c->n_grp;
  a.D = c->Dm;
  a.B = B;
  a.lvt = c->lvt;
  a.dcol = c->dcol_d;
  a.gid = c->gid_d;
  a.out = out;
  // tile height: 128 cells (one CTA per SM) or 64 (two), the autotuner's choice (same sums)
  Tunable* tu = nullptr;
  const int cells = tune_pick(c, "eta_tile", {128, 64}, 128, &tu);
  TuneScope ts(c, tu);
  if (cells == 64) {
    const size_t smem = eta_smem_bytes<2>(c->n_d);
    GPL_TRY(c, cudaFuncSetAttribute(k_eta_dmma<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int tiles = div_up(c->N, 64) * div_up(c->J, BN);
    k_eta_dmma<2><<<std::min(tiles, 2 * c->sm_count), kThreads, smem, c->stream>>>(a);
  } else {
    const size_t smem = eta_smem_bytes<4>(c->n_d);
    GPL_TRY(c, cudaFuncSetAttribute(k_eta_dmma<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int tiles = div_up(c->N, 128) * div_up(c->J, BN);
    k_eta_dmma<4><<<std::min(tiles, c->sm_count), kThreads, smem, c->stream>>>(a);
  }
  GPL_LAUNCHED(c, "k_eta_dmma");
  return GPL_OK;
}

}  // namespace gpl
