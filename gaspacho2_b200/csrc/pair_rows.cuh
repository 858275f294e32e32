// U_a = sum_b d_b V[pair(a, b)] for one cell, V over the unique column pairs a <= b (row-major upper
// triangle: pair(a, b) = a n_d - a (a - 1) / 2 + b - a), by a block of 256 threads (W = 8 warps) or by
// one warp (W = 1): whole rows a of the triangle pass through shared memory, and every entry is used
// once for both of its columns (a warp per row, two rows at a time: the row's sum over the lanes, the
// other column's sums in the lanes' registers). Used for V from memory (k_v_to_u) and for V from
// residues (k_crt_u).
//
// A warp per cell where there are cells enough: with a block per cell its barriers and its rows'
// reductions, each waiting for the last, cost more than the entries. Measured (ms, block / warp), V from
// memory: 30,000 cells x 34 columns 0.215 / 0.103, x 94 0.506 / 0.299; 50,000 x 132 1.30 / 0.85 (2.63
// with a thread per column); 1,000 x 66 0.019 / 0.021. V from residues, where the entries' own
// arithmetic counts: 30,000 x 34 0.323 / 0.191, x 94 1.04 / 0.94, 50,000 x 132 3.16 / 3.38.
#pragma once

#include <type_traits>

#include "gpl_internal.cuh"

namespace gpl {

constexpr int kUMaxDense = 512;   // columns: 8 warps' column sums fit where V was
constexpr int kUWarpCells = 2368;  // 16 warps per SM

// entries of V in shared memory at a time
template <int W>
constexpr int u_entries() {
  return W == 8 ? 4096 : 512;
}
// doubles of a cell's shared memory: V, the D row, the row sums and, where they are asked for, the diagonals
template <int W, bool kDiag>
__host__ __device__ constexpr int u_space(int n_d) {
  return u_entries<W>() + 4 + (kDiag ? 3 : 2) * ((n_d + 1) & ~1);
}

// f(slots, warps): the form for n_d columns and `cells` cells, as two integral constants; a warp per
// cell up to warp_dense columns (at most 160)
template <class F>
void pair_rows_form(int n_d, int cells, int warp_dense, F f) {
  using std::integral_constant;
  const bool warp = cells >= kUWarpCells && n_d <= warp_dense;
  if (warp && n_d <= 96) f(integral_constant<int, 3>(), integral_constant<int, 1>());
  else if (warp) f(integral_constant<int, 5>(), integral_constant<int, 1>());
  else if (n_d <= 160) f(integral_constant<int, 5>(), integral_constant<int, 8>());
  else if (n_d <= 288) f(integral_constant<int, 9>(), integral_constant<int, 8>());
  else f(integral_constant<int, 16>(), integral_constant<int, 8>());
}

// S: 32-column slots, n_d <= 32 S. vs: the cell's u_space doubles. fill(from, p1, t, n): the threads t of n
// write V[from ..] to vs[0 ..], up to p1 (from: a multiple of four). kDiag: returns where the diagonals
// V[pair(a, a)] lie in shared memory, complete for the threads of the cell.
template <int S, int W, bool kDiag, class Fill>
__device__ __forceinline__ const double* pair_rows_to_u(int i, int ldN, int n_d, double* vs,
                                                        const double* __restrict__ D, double* __restrict__ U,
                                                        Fill fill) {
  constexpr int kThr = 32 * W, kOwn = (32 * S + kThr - 1) / kThr;
  double *ds = vs + u_entries<W>() + 4, *rs = ds + ((n_d + 1) & ~1), *dv = rs + ((n_d + 1) & ~1);
  const int lane = threadIdx.x & 31, warp = W == 8 ? threadIdx.x >> 5 : 0, tid = W == 8 ? threadIdx.x : lane;
  auto sync = [&]() {
    if (W == 8) __syncthreads();
    else __syncwarp();
  };
  double own[kOwn];
#pragma unroll
  for (int k = 0; k < kOwn; k++) own[k] = tid + kThr * k < n_d ? D[(size_t)(tid + kThr * k) * ldN + i] : 0.0;
  double col[S], db[S];
#pragma unroll
  for (int t = 0; t < S; t++) col[t] = db[t] = 0.0;
  for (int a0 = 0, p0 = 0; a0 < n_d;) {
    // rows [a0, a1): pairs [p0, p1), from the multiple of four at or below p0
    int a1 = a0, p1 = p0;
    const int from = p0 & ~3;
    while (a1 < n_d && p1 + (n_d - a1) - from <= u_entries<W>()) p1 += n_d - a1++;
    fill(from, p1, tid, kThr);
    if (a0 == 0) {
#pragma unroll
      for (int k = 0; k < kOwn; k++)
        if (tid + kThr * k < n_d) ds[tid + kThr * k] = own[k];
    }
    sync();
    if (a0 == 0) {
#pragma unroll
      for (int t = 0; t < S; t++)
        if (32 * t + lane < n_d) db[t] = ds[32 * t + lane];
    }
    for (int a = a0 + warp; a < a1; a += 2 * W) {
      // V[pair(a, b)] at row[b], b >= a
      const int e = a + W;
      const bool two = e < a1;
      const double* row = vs + (a * n_d - a * (a - 1) / 2 - a - from);
      const double* row2 = vs + (e * n_d - e * (e - 1) / 2 - e - from);
      const double da = ds[a], de = two ? ds[e] : 0.0;
      double sum = 0.0, sum2 = 0.0;
#pragma unroll
      for (int t = 0; t < S; t++) {
        const int b = 32 * t + lane;
        if (32 * t < n_d && 32 * t + 31 >= a) {
          if (b >= a && b < n_d) {
            const double v = row[b];
            sum = fma(db[t], v, sum);
            if (b > a) col[t] = fma(da, v, col[t]);
          }
          if (two && b >= e && b < n_d) {
            const double v = row2[b];
            sum2 = fma(db[t], v, sum2);
            if (b > e) col[t] = fma(de, v, col[t]);
          }
        }
      }
      sum = warp_sum(sum);
      sum2 = warp_sum(sum2);
      if (lane == 0) {
        rs[a] = sum;
        if (kDiag) dv[a] = row[a];
        if (two) {
          rs[e] = sum2;
          if (kDiag) dv[e] = row2[e];
        }
      }
    }
    a0 = a1;
    p0 = p1;
    sync();
  }
  if (W == 1) {
#pragma unroll
    for (int t = 0; t < S; t++)
      if (32 * t + lane < n_d) U[i + (size_t)(32 * t + lane) * ldN] = rs[32 * t + lane] + col[t];
    return dv;
  }
  double* cs = vs;  // [8][n_d] the warps' column sums
#pragma unroll
  for (int t = 0; t < S; t++)
    if (32 * t + lane < n_d) cs[warp * n_d + 32 * t + lane] = col[t];
  __syncthreads();
  for (int a = threadIdx.x; a < n_d; a += 256) {
    double u = rs[a];
#pragma unroll
    for (int w = 0; w < 8; w++) u += cs[w * n_d + a];
    U[i + (size_t)a * ldN] = u;
  }
  return dv;
}

}  // namespace gpl
