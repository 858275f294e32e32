// Batched inverse of the per-gene Psi_j from their Cholesky factors (solvePsi,
// ggplvm.cu:46-53, which runs cholsl chol.cu:45-56 on every column of the identity):
// Psi_j^{-1} = V^T V with V = L^{-1}, in 32-column panels with FP64 tensor-core (DMMA)
// block products.
//
//   k_tri_diag     one warp per (32 x 32 diagonal block, gene): V_ii = L_ii^{-1} by substitution.
//   k_trtri_panel  one CTA per (panel jb, gene): the columns [32 jb, 32 jb + 32) of V by
//                  forward substitution over 32-row blocks, Y_i = V_ii (-L[i, jb..i) Y[jb..i)).
//                  Work: P^3/6 multiply-adds per gene.
//   k_lauum_panel  one CTA per (panel b, gene): S[a, b] = sum_{k >= a} V[k, a]^T V[k, b]
//                  for the blocks a >= b, written to both triangles. Work: P^3/6 per gene.
// In the panel kernels the panel stays in shared memory and all the 32 x 32 blocks it meets are ONE
// stream through three buffers (asynchronous copies two blocks ahead, one barrier per block): they are
// bound by the latency of a block's step (the MMAs are 0.7 ms of the 2.3 below at 35 TFLOP/s). With each
// row block's copies started when the last was done, and its diagonal block solved by 32 steps of
// shuffles, 3,000 inverses of P = 232 took 4.4 ms, now 2.3; 2,000 of 69: 0.35, now 0.19; 501 of 564
// (one CTA per SM): 8.3, now 4.1.
// Both fit two CTAs per SM up to P = 256 (the panel's rows plus the buffers).
//
// L is the lower triangle (with diagonal) of the factored Psi_j (column-major, ld P); V is
// written column-major (ld P) below and on the diagonal of each panel, the strict upper part of
// the diagonal blocks holding exact zeros. A factor zero-filled by a failed Cholesky gives
// infinities and NaNs, as in the reference.
#include <algorithm>
#include <cmath>

#include "dmma_common.cuh"
#include "gpl_internal.cuh"
#include "in_order.cuh"

namespace gpl {

namespace {
constexpr int IB = 32;  // block size
constexpr int IS = 36;  // shared row stride (doubles): conflict-free fragment loads
constexpr int NB = 3;   // buffers of the inverse's block stream
constexpr int CW = 8;   // finished columns per chunk of the Cholesky's panel update
// Largest P each kernel is launched for. k_potrf_panel's update covers 256 rows of a panel
// (8 warps x 2 row tiles of 16), so its panels below the first may hold at most 256 rows:
// P <= 288. The inverse panels hold any P their shared memory admits (P <= 640 within 220 KiB).
constexpr int kPotrfMaxP = 288;
// With half the threads (128 rows below the first panel), up to four CTAs per SM hide more of a
// panel's latency.
constexpr int kPotrfHalfP = 160;
constexpr int kInverseMaxP = 640;
}  // namespace

// Lane c solves L_ii v = e_c with v in registers; L's columns are read as broadcasts.
__global__ void __launch_bounds__(128) k_tri_diag(const double* __restrict__ Psi, int P, int64_t stride, int blocks,
                                                  double* __restrict__ V) {
  __shared__ __align__(16) double Ls[4][IB][IB + 2];  // [q][m]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nb = (P + IB - 1) / IB;
  const int w = blockIdx.x * 4 + warp;
  if (w >= blocks) return;
  const int gene = w / nb, r0 = (w - gene * nb) * IB, n = min(IB, P - r0);
  const double* L = Psi + (size_t)gene * stride + r0 + (size_t)r0 * P;
  double* Vm = V + (size_t)gene * stride + r0 + (size_t)r0 * P;
#pragma unroll
  for (int q = 0; q < IB; q++)
    Ls[warp][q][lane] = (q < n && lane < n && lane >= q) ? L[lane + (size_t)q * P] : (lane == q ? 1.0 : 0.0);
  __syncwarp();
  const double rd = 1.0 / Ls[warp][lane][lane];
  double v[IB];
#pragma unroll
  for (int m = 0; m < IB; m++) v[m] = m == lane ? 1.0 : 0.0;
#pragma unroll
  for (int q = 0; q < IB; q++) {
    v[q] *= __shfl_sync(0xffffffffu, rd, q);
#pragma unroll
    for (int m = q + 1; m < IB; m++) v[m] = fma(-Ls[warp][q][m], v[q], v[m]);
  }
  __syncwarp();
#pragma unroll
  for (int m = 0; m < IB; m++) Ls[warp][lane][m] = v[m];  // column `lane`
  __syncwarp();
  if (lane < n)
    for (int q = 0; q < n; q++) Vm[lane + (size_t)q * P] = Ls[warp][q][lane];
}

// The block A[r.., c..] (column-major, ld P, zeros past P) into dst[q][IS], column q of the block.
// The thread's copies are one group.
__device__ __forceinline__ void stage_block(double* dst, const double* __restrict__ A, int r, int c, int P, bool pairs) {
  if (pairs) {  // even P: every column starts 16-byte aligned
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const int e = threadIdx.x + 256 * k, q = e >> 4, m = 2 * (e & 15);
      const bool ok = r + m < P && c + q < P;
      cp_async16(dst + q * IS + m, A + (ok ? (size_t)(r + m) + (size_t)(c + q) * P : 0), ok ? 16 : 0);
    }
  } else {
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int e = threadIdx.x + 256 * k, q = e >> 5, m = e & 31;
      const bool ok = r + m < P && c + q < P;
      cp_async8(dst + q * IS + m, A + (ok ? (size_t)(r + m) + (size_t)(c + q) * P : 0), ok ? 8 : 0);
    }
  }
}

__global__ void __launch_bounds__(256, 2)
    k_trtri_panel(const double* __restrict__ Psi, int P, int64_t stride, double* V) {
  extern __shared__ __align__(16) double sm[];
  const int nb = (P + IB - 1) / IB, SY = nb * IB + 4;
  const int jb = blockIdx.x, r0 = jb * IB;
  const double* L = Psi + (size_t)blockIdx.y * stride;
  double* Vm = V + (size_t)blockIdx.y * stride;
  double* Yt = sm;                      // [32][SY] column n, row k (global row r0 + k)
  double* Rt = Yt + (size_t)IB * SY;    // [32][IS] a row block's right-hand sides, column n
  double* St = Rt + IB * IS;            // [NB][32][IS] the stream, column k of each block
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int m0 = (warp >> 2) * 16, n0 = (warp & 3) * 8;
  const bool pairs = (P & 1) == 0;
  // the stream: for each row block i > jb the blocks L[i, jb .. i - 1], then V[i, i]
  int li = jb + 1, lc = jb, lbuf = 0;  // the next block to load
  auto load = [&]() {
    if (li < nb) {
      double* dst = St + lbuf * IB * IS;
      if (lc < li) stage_block(dst, L, li * IB, lc * IB, P, pairs);
      else stage_block(dst, Vm, li * IB, li * IB, P, pairs);
      if (++lc > li) {
        li++;
        lc = jb;
      }
      lbuf = lbuf + 1 == NB ? 0 : lbuf + 1;
    }
    cp_async_commit();
  };
  for (int e = tid; e < IB * IB; e += 256) {
    const int n = e >> 5, k = e & 31;
    const bool ok = r0 + k < P && r0 + n < P;
    cp_async8(Yt + n * SY + k, Vm + (ok ? (size_t)(r0 + k) + (size_t)(r0 + n) * P : 0), ok ? 8 : 0);
  }
  for (int k = 0; k < NB - 1; k++) load();
  int buf = 0;
  for (int i = jb + 1; i < nb; i++) {
    // two accumulators over alternating K steps break the DMMA chain
    double acc[2][4] = {};
    for (int ch = jb; ch <= i; ch++) {
      cp_async_wait<NB - 2>();
      __syncthreads();  // the block is there; the buffer loaded next, Rt and Yt are as the last step left them
      load();
      const bool diag = ch == i;
      const double* as = St + buf * IB * IS;
      const double* bt = diag ? Rt : Yt + (ch - jb) * IB;
      const int sb = diag ? IS : SY;
      if (diag) {
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
          for (int z = 0; z < 4; z++) acc[h][z] = 0.0;
      }
#pragma unroll
      for (int kb = 0; kb < IB; kb += 8)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const double* ar = as + (kb + 4 * h + t) * IS + m0 + g;
          dmma_16x8x4(acc[h], ar[0], ar[8], bt[(n0 + g) * sb + kb + 4 * h + t]);
        }
      if (ch + 1 >= i) {  // the right-hand sides are complete, or the solution is
        double* o = diag ? Yt + (i - jb) * IB : Rt;
        const int so = diag ? SY : IS;
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
          for (int e = 0; e < 2; e++) {
            const double v = acc[0][2 * h + e] + acc[1][2 * h + e];
            o[(n0 + 2 * t + e) * so + m0 + g + 8 * h] = diag ? v : -v;
          }
      }
      buf = buf + 1 == NB ? 0 : buf + 1;
    }
  }
  __syncthreads();
  // the panel below its diagonal block (k_tri_diag wrote that)
  const int ncol = min(IB, P - r0);
  for (int n = warp; n < ncol; n += 8)
    for (int r = IB + lane; r < P - r0; r += 32) Vm[(size_t)(r0 + r) + (size_t)(r0 + n) * P] = Yt[n * SY + r];
}

__global__ void __launch_bounds__(256, 2)
    k_lauum_panel(const double* __restrict__ V, int P, int64_t stride, double* __restrict__ S) {
  extern __shared__ __align__(16) double sm[];
  const int nb = (P + IB - 1) / IB, SY = nb * IB + 4;
  const int b = blockIdx.x, c0 = b * IB;
  const double* Vm = V + (size_t)blockIdx.y * stride;
  double* Sm = S + (size_t)blockIdx.y * stride;
  double* Vb = sm;                       // [32][SY] column n of the panel, row k (global row c0 + k)
  double* St = Vb + (size_t)IB * SY;     // [NB][32][IS] the stream, column m of each block
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int m0 = (warp >> 2) * 16, n0 = (warp & 3) * 8;
  const bool pairs = (P & 1) == 0;
  // the stream: for each block column a >= b the blocks V[a .. nb - 1, a]
  int la = b, lk = b, lbuf = 0;
  auto load = [&]() {
    if (la < nb) {
      stage_block(St + lbuf * IB * IS, Vm, lk * IB, la * IB, P, pairs);
      if (++lk == nb) lk = ++la;
      lbuf = lbuf + 1 == NB ? 0 : lbuf + 1;
    }
    cp_async_commit();
  };
  const int krows = (nb - b) * IB;
  for (int n = warp; n < IB; n += 8) {
    const bool okn = c0 + n < P;
    if (pairs) {
      for (int k = 2 * lane; k < krows; k += 64) {
        const bool ok = okn && c0 + k < P;
        cp_async16(Vb + n * SY + k, Vm + (ok ? (size_t)(c0 + k) + (size_t)(c0 + n) * P : 0), ok ? 16 : 0);
      }
    } else {
      for (int k = lane; k < krows; k += 32) {
        const bool ok = okn && c0 + k < P;
        cp_async8(Vb + n * SY + k, Vm + (ok ? (size_t)(c0 + k) + (size_t)(c0 + n) * P : 0), ok ? 8 : 0);
      }
    }
  }
  for (int k = 0; k < NB - 1; k++) load();
  int buf = 0;
  for (int a = b; a < nb; a++) {
    double acc[2][4] = {};
    for (int kc = a; kc < nb; kc++) {
      cp_async_wait<NB - 2>();
      __syncthreads();
      load();
      const double* at = St + buf * IB * IS + (m0 + g) * IS + t;
      const double* bt = Vb + (n0 + g) * SY + (kc - b) * IB + t;
#pragma unroll
      for (int kb = 0; kb < IB; kb += 8)
#pragma unroll
        for (int h = 0; h < 2; h++)
          dmma_16x8x4(acc[h], at[kb + 4 * h], at[8 * IS + kb + 4 * h], bt[kb + 4 * h]);
      buf = buf + 1 == NB ? 0 : buf + 1;
    }
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int row = a * IB + m0 + g + 8 * h, col = c0 + n0 + 2 * t + e;
        if (row < P && col < P) {
          const double v = acc[0][2 * h + e] + acc[1][2 * h + e];
          Sm[(size_t)row + (size_t)col * P] = v;
          Sm[(size_t)col + (size_t)row * P] = v;
        }
      }
  }
}

// A 32 x 32 diagonal block in columns at Ap (column stride SP), the first ncol of its rows and columns
// in use, factored in place by one warp, right-looking with row `lane` in registers; Rd gets the
// diagonal's reciprocals. Entry (r, q) takes its products l_rk l_qk in increasing k and is scaled by
// 1/l_qq last, as choldc's sums. The chain from pivot to pivot (lane cc + 1 needs only its own entries)
// is kept apart from the update of the other columns, which fills its gaps; a finished column is
// read back from shared memory. The root and its reciprocal are the library's, rounded correctly over the
// whole range of a pivot. (A hand-made root without their rare branches took half the cycles of a block,
// but a pivot that cancels to a subnormal number has no estimate there.) Returns true for a pivot <= 0; a
// NaN pivot passes, as in choldc.
template <bool kFull>
__device__ __noinline__ bool factor_block(double* Ap, int SP, int ncol, double* Rd) {
  const int lane = threadIdx.x & 31;
  double a[IB];
#pragma unroll
  for (int q = 0; q < IB; q++) a[q] = lane < ncol ? Ap[q * SP + lane] : 0.0;
  bool bad = false;
  double piv = __shfl_sync(0xffffffffu, a[0], 0);
#pragma unroll
  for (int cc = 0; cc < IB; cc++) {
    if (kFull || cc < ncol) {
      const double l = sqrt(piv), rd = 1.0 / l;
      bad |= piv <= 0.0;
      if (lane == 0) Rd[cc] = rd;
      const double x = a[cc] * rd;
      a[cc] = lane == cc ? l : x;
      double* col = Ap + cc * SP;  // its final place; rows past ncol are not stored, rows above cc not read
      col[lane] = a[cc];
      if (cc + 1 < IB) piv = __shfl_sync(0xffffffffu, fma(-x, x, a[cc + 1]), cc + 1);
      __syncwarp();
#pragma unroll
      for (int q = cc + 1; q < IB; q++) a[q] = fma(-a[cc], col[q], a[q]);
    }
  }
  return bad;
}
__device__ __forceinline__ bool factor_diagonal(double* Ap, int SP, int ncol, double* Rd) {
  return ncol == IB ? factor_block<true>(Ap, SP, ncol, Rd) : factor_block<false>(Ap, SP, ncol, Rd);
}

// Batched Cholesky (cholPsi, ggplvm.cu:683-692), one CTA per gene, 32-column panels left to
// right (left-looking): the panel is loaded into shared memory, takes the product of the
// finished columns (DMMA, the finished part streamed through shared memory, two CTAs per SM), then
// its 32 x 32 diagonal block is factored by one warp (lane = row; each entry's sum in increasing
// column order as in choldc) and the rows below solve against it (thread per row). A non-positive pivot zero-fills the matrix, as choldc does. Reads the lower triangle,
// writes the factor over it; the strict upper triangle is left as it was.
// The factorization of one matrix A (P x P, ld P) by the CTA (256 threads); `sm` is the dynamic
// shared memory (potrf_panel_smem bytes for `ns` buffers), `fail` a shared flag. Used by k_potrf_panel
// (one matrix per CTA) and by the persistent IRLS tail (k_irls_tail, matrices from a queue).
//
// Bound by latency (the MMAs take 36,000 cycles of a partition at P = 232). Of 577,000 cycles per matrix
// there, two CTAs per SM, 400,000 went on the copies and the finished columns' chunks (an element's
// place from a division, each chunk waited for, the panel in rows with 4-way bank conflicts) and
// 146,000 on the diagonal blocks. Here the panel lies in columns, everything arrives by asynchronous
// copies (16 bytes where P is even), a chunk is as many columns as the space holds at the panel's
// height with one or two more in flight, and the next panel's first chunks arrive during the
// diagonal block. 3,000 matrices of P = 232: 3.1 -> 1.93 ms; 2,000 of 69: 0.28 -> 0.19 ms; 1,000 of
// 285: 2.4 -> 1.01 ms. Each entry's operations and their order are the same.
template <int T>
__device__ __forceinline__ void potrf_panel_one(double* A, int P, int ns, int sms, double* sm, int& fail) {
  const int rows_pad = max(IB, (P + 15) / 16 * 16);
  const int SP = rows_pad + 2, space = ns * CW * (rows_pad + 4);
  double* Ap = sm;                          // [32][SP]: the panel, column cc, row r
  double* La = Ap + (size_t)IB * SP;        // `space` doubles: chunks of finished columns
  double* Rd = La + space;                  // [32] reciprocals of the diagonal
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const bool pairs = (P & 1) == 0 && (reinterpret_cast<uintptr_t>(A) & 15) == 0;
  const int dw = (blockIdx.x / sms) & 3;  // a CTA's neighbours on its SM were launched about a block per SM apart
  if (tid == 0) fail = 0;
  // the panel that copies are issued for: its first row, the chunks' stride, columns and buffers that
  // the space holds at its height, and the next chunk to load
  int p0, rpad, SA, cw, nbuf, lch, lbuf;
  auto panel = [&](int c0) {
    p0 = c0;
    rpad = (P - c0 + 15) / 16 * 16;
    SA = max(IB, rpad) + 4;
    cw = IB;
    while (cw > CW && 2 * cw * SA > space) cw >>= 1;
    nbuf = 3 * cw * SA <= space ? 3 : 2;
    lch = lbuf = 0;
  };
  // rows p0 .. of column col, zeros to rpad (all zeros if !ok)
  auto column = [&](double* dst, int col, bool ok) {
    const double* src = A + p0 + (size_t)(ok ? col : 0) * P;
    const int rows = P - p0;
    if (pairs) {
      for (int r = 2 * lane; r < rpad; r += 64) cp_async16(dst + r, src + (r < rows ? r : 0), ok && r < rows ? 16 : 0);
    } else {
      for (int r = lane; r < rpad; r += 32) cp_async8(dst + r, src + (r < rows ? r : 0), ok && r < rows ? 8 : 0);
    }
  };
  auto stage = [&]() {
    if (lch < p0 / cw) {
      for (int q = warp; q < cw; q += T / 32) column(La + (size_t)(lbuf * cw + q) * SA, lch * cw + q, true);
      lch++;
      lbuf = lbuf + 1 == nbuf ? 0 : lbuf + 1;
    }
    cp_async_commit();
  };
  panel(0);
  for (int c0 = 0; c0 < P; c0 += IB) {
    const int rows = P - c0, ncol = min(IB, rows), nch = c0 / cw;
    for (int k = lch; k < nbuf - 1; k++) stage();
    // the panel itself, in the group of the chunk that the first step issues: it is needed last
    for (int cc = warp; cc < IB; cc += T / 32) column(Ap + (size_t)cc * SP, c0 + cc, cc < ncol);
    // Ap -= L[c0.., 0..c0) L[c0..c0+32, 0..c0)^T, cw finished columns per chunk
    double acc[2][4][4];
#pragma unroll
    for (int x = 0; x < 2; x++)
#pragma unroll
      for (int y = 0; y < 4; y++)
#pragma unroll
        for (int z = 0; z < 4; z++) acc[x][y][z] = 0.0;
    for (int ch = 0, buf = 0; ch < nch; ch++) {
      if (nbuf == 3) cp_async_wait<1>();
      else cp_async_wait<0>();
      __syncthreads();
      stage();
      const double* la = La + (size_t)buf * cw * SA;
#pragma unroll 2
      for (int k4 = 0; k4 < cw / 4; k4++) {
        const double* lr = la + (k4 * 4 + t) * SA;
        double b[4];
#pragma unroll
        for (int y = 0; y < 4; y++) b[y] = lr[y * 8 + g];  // B[k][n] = L[c0 + n][q]
#pragma unroll
        for (int x = 0; x < 2; x++) {
          const int mt = warp + T / 32 * x;
          if (mt * 16 < rpad) {
            const double a0 = lr[mt * 16 + g], a1 = lr[mt * 16 + g + 8];
#pragma unroll
            for (int y = 0; y < 4; y++) dmma_16x8x4(acc[x][y], a0, a1, b[y]);
          }
        }
      }
      buf = buf + 1 == nbuf ? 0 : buf + 1;
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    if (nch > 0) {
#pragma unroll
      for (int x = 0; x < 2; x++) {
        const int mt = warp + T / 32 * x;
        if (mt * 16 >= rpad) continue;
#pragma unroll
        for (int y = 0; y < 4; y++)
#pragma unroll
          for (int h = 0; h < 2; h++)
#pragma unroll
            for (int e = 0; e < 2; e++) Ap[(y * 8 + 2 * t + e) * SP + mt * 16 + g + 8 * h] -= acc[x][y][2 * h + e];
      }
      __syncthreads();
    }
    // the next panel's first chunks, as far as their columns are finished, arrive during the rest
    if (c0 + IB < P) {
      panel(c0 + IB);
      while (lch < nbuf - 1 && (lch + 1) * cw <= c0) stage();
    }
    // the diagonal block, then the rows below it, thread per row, in the same order. Co-resident CTAs
    // take different warps for it: warp w of every CTA runs on the SM's partition w mod 4
    if (warp == dw) {
      if (factor_diagonal(Ap, SP, ncol, Rd) && lane == 0) fail = 1;
    }
    __syncthreads();
    for (int r = IB + tid; r < rows; r += T) {
      double a[IB];
#pragma unroll
      for (int q = 0; q < IB; q++) a[q] = Ap[q * SP + r];
#pragma unroll
      for (int cc = 0; cc < IB; cc++) {  // rows below: the panel has all 32 columns
        const double x = a[cc] * Rd[cc];
        a[cc] = x;
#pragma unroll
        for (int q = cc + 1; q < IB; q++) a[q] -= x * Ap[cc * SP + q];
      }
#pragma unroll
      for (int q = 0; q < IB; q++) Ap[q * SP + r] = a[q];
    }
    __syncthreads();
    for (int cc = warp; cc < ncol; cc += T / 32)
      for (int r = lane; r < rows; r += 32)
        if (r >= cc) A[(size_t)(c0 + r) + (size_t)(c0 + cc) * P] = Ap[cc * SP + r];
    __threadfence_block();
    __syncthreads();
  }
  if (fail)
    for (int e = tid; e < P * P; e += T) A[e] = 0.0;
}

template <int T>
__global__ void __launch_bounds__(T, 512 / T) k_potrf_panel(double* __restrict__ Psi, int P, int64_t stride, int ns,
                                                             int sms) {
  extern __shared__ __align__(16) double sm[];
  __shared__ int fail;
  potrf_panel_one<T>(Psi + (size_t)blockIdx.x * stride, P, ns, sms, sm, fail);
}

int potrf_panel_smem(int P, int ns) {
  const int rows_pad = std::max(IB, (P + 15) / 16 * 16);
  return (int)sizeof(double) * (IB * (rows_pad + 2) + ns * CW * (rows_pad + 4) + IB);
}

// Chunk buffers: three while two CTAs still share an SM (with `extra` bytes each), else two.
int potrf_buffers(int P, int extra) { return 2 * (potrf_panel_smem(P, 3) + extra + 1536) <= 228 * 1024 ? 3 : 2; }

// The same factorization for any n: the rows of a 32-column panel in blocks of 128 (a row tile of 16
// per warp), each block taking the product of the finished columns (its own rows against the
// panel's 32 diagonal rows, 16 columns per chunk through two buffers), the first one then factoring
// the diagonal block, all solving against it. 85 KB of shared memory whatever n is, two CTAs per
// SM. At n = 564 (501 matrices) a column-at-a-time kernel that read the finished columns from
// global memory for every entry took 57.6 ms, this one 2.8 ms.
namespace {
constexpr int RB = 128, RC = 16;           // rows per block, finished columns per chunk
constexpr int RSA = RB + 4, RSB = IB + 4;  // strides 4 mod 16
constexpr int DS = IB + 2;                 // the diagonal block's column stride
constexpr int kRowsSmem = (int)sizeof(double) * (RB * IS + 2 * RC * (RSA + RSB) + IB * DS + IB);
}  // namespace

__global__ void __launch_bounds__(256, 2) k_potrf_rows(double* __restrict__ Psi, int P, int64_t stride) {
  extern __shared__ __align__(16) double sm[];
  __shared__ int fail;
  double* Ap = sm;                    // [RB][IS] the block of the panel
  double* La = Ap + RB * IS;          // [2][RC][RSA] finished columns, the block's rows
  double* Lb = La + 2 * RC * RSA;     // [2][RC][RSB] finished columns, the diagonal rows
  double* Dg = Lb + 2 * RC * RSB;     // [32][DS] the panel's factored diagonal block, in columns
  double* Rd = Dg + IB * DS;          // [32] reciprocals of its diagonal
  double* A = Psi + (size_t)blockIdx.x * stride;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const bool even = (P & 1) == 0;  // rows start at even offsets: 16-byte copies
  if (tid == 0) fail = 0;
  for (int c0 = 0; c0 < P; c0 += IB) {
    const int ncol = min(IB, P - c0);
    for (int r0 = c0; r0 < P; r0 += RB) {
      const int rows = min(RB, P - r0);
      // finished columns [RC ch, RC ch + RC) of the block's rows and of the diagonal rows
      auto stage = [&](int ch, int buf) {
        double* da = La + buf * RC * RSA;
        double* db = Lb + buf * RC * RSB;
        const double* src = A + (size_t)(ch * RC) * P;
        if (even) {
          for (int e = tid; e < RC * (RB + IB) / 2; e += 256) {
            const int q = e / ((RB + IB) / 2), r = 2 * (e - q * ((RB + IB) / 2));
            const bool a = r < RB;
            const int row = a ? r0 + r : c0 + r - RB;
            const int nb = row < P ? 16 : 0;
            cp_async16(a ? da + q * RSA + r : db + q * RSB + r - RB, src + (size_t)q * P + min(row, P - 2), nb);
          }
        } else {
          for (int e = tid; e < RC * (RB + IB); e += 256) {
            const int q = e / (RB + IB), r = e - q * (RB + IB);
            const bool a = r < RB;
            const int row = a ? r0 + r : c0 + r - RB;
            const int nb = row < P ? 8 : 0;
            cp_async8(a ? da + q * RSA + r : db + q * RSB + r - RB, src + (size_t)q * P + min(row, P - 1), nb);
          }
        }
        cp_async_commit();
      };
      const int nch = c0 / RC;
      if (nch > 0) stage(0, 0);
      for (int e = tid; e < RB * IB; e += 256) {  // rows fastest: coalesced columns
        const int cc = e / RB, r = e - cc * RB;
        Ap[r * IS + cc] = (r < rows && cc < ncol) ? A[(size_t)(r0 + r) + (size_t)(c0 + cc) * P] : 0.0;
      }
      double acc[4][4];
#pragma unroll
      for (int y = 0; y < 4; y++)
#pragma unroll
        for (int z = 0; z < 4; z++) acc[y][z] = 0.0;
      for (int ch = 0; ch < nch; ch++) {
        if (ch + 1 < nch) {
          stage(ch + 1, (ch + 1) & 1);
          cp_async_wait<1>();
        } else {
          cp_async_wait<0>();
        }
        __syncthreads();
        const double* la = La + (ch & 1) * RC * RSA;
        const double* lb = Lb + (ch & 1) * RC * RSB;
        if (warp * 16 < rows) {
#pragma unroll
          for (int k4 = 0; k4 < RC / 4; k4++) {
            const double* ar = la + (k4 * 4 + t) * RSA + warp * 16 + g;
            const double* br = lb + (k4 * 4 + t) * RSB + g;
            const double a0 = ar[0], a1 = ar[8];
#pragma unroll
            for (int y = 0; y < 4; y++) dmma_16x8x4(acc[y], a0, a1, br[y * 8]);
          }
        }
        __syncthreads();  // the buffer is refilled two chunks on
      }
      if (nch == 0) __syncthreads();  // Ap complete
      else if (warp * 16 < rows) {
#pragma unroll
        for (int y = 0; y < 4; y++)
#pragma unroll
          for (int h = 0; h < 2; h++)
#pragma unroll
            for (int e = 0; e < 2; e++) Ap[(warp * 16 + g + 8 * h) * IS + y * 8 + 2 * t + e] -= acc[y][2 * h + e];
      }
      __syncthreads();
      if (r0 == c0) {
        // the diagonal block, one warp, as in potrf_panel_one
        if (warp == 0) {
          for (int q = 0; q < IB; q++) Dg[q * DS + lane] = lane < ncol ? Ap[lane * IS + q] : 0.0;
          __syncwarp();
          if (factor_diagonal(Dg, DS, ncol, Rd) && lane == 0) fail = 1;
          __syncwarp();
          if (lane < ncol)
            for (int q = 0; q < IB; q++) Ap[lane * IS + q] = Dg[q * DS + lane];
        }
        __syncthreads();
      }
      const int first = r0 == c0 ? IB : 0;
      for (int r = first + tid; r < rows; r += 256) {
        double a[IB];
#pragma unroll
        for (int q = 0; q < IB; q++) a[q] = Ap[r * IS + q];
#pragma unroll
        for (int cc = 0; cc < IB; cc++) {
          if (cc < ncol) {
            const double x = a[cc] * Rd[cc];
            a[cc] = x;
#pragma unroll
            for (int q = cc + 1; q < IB; q++) a[q] -= x * Dg[cc * DS + q];
          }
        }
#pragma unroll
        for (int q = 0; q < IB; q++) Ap[r * IS + q] = a[q];
      }
      __syncthreads();
      for (int e = tid; e < rows * IB; e += 256) {
        const int cc = e / rows, r = e - cc * rows;
        if (cc < ncol && (r0 > c0 || r >= cc)) A[(size_t)(r0 + r) + (size_t)(c0 + cc) * P] = Ap[r * IS + cc];
      }
      __threadfence_block();
      __syncthreads();
    }
  }
  if (fail)
    for (int e = tid; e < P * P; e += 256) A[e] = 0.0;
}

// GPL_ERR_ARG within an OrderScope beyond the panel kernel's range: the row-block kernel takes its sums in
// another order than the entry-by-entry form.
int launch_potrf_panels(Ctx* c, double* A, int n, int batch, int64_t stride) {
  const int ns = potrf_buffers(n, 0), smem = potrf_panel_smem(n, ns);
  if (n > kPotrfMaxP || smem > 220 * 1024) {
    if (c->one_order) return GPL_ERR_ARG;
    GPL_TRY(c, cudaFuncSetAttribute(k_potrf_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, kRowsSmem));
    GPL_TRY(c, cudaFuncSetAttribute(k_potrf_rows, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    k_potrf_rows<<<batch, 256, kRowsSmem, c->stream>>>(A, n, stride);
    GPL_LAUNCHED(c, "k_potrf_rows");
    return GPL_OK;
  }
  auto* kernel = n <= kPotrfHalfP ? k_potrf_panel<128> : k_potrf_panel<256>;
  GPL_TRY(c, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  GPL_TRY(c, cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
  kernel<<<batch, n <= kPotrfHalfP ? 128 : 256, smem, c->stream>>>(A, n, stride, ns, c->sm_count);
  GPL_LAUNCHED(c, "k_potrf_panel");
  return GPL_OK;
}

// trtri: the panel, the right-hand sides and the stream's buffers (lauum needs the panel and the
// buffers). 103 KB at P = 236: two CTAs per SM.
int inverse_panel_smem(int P) {
  const int nb = (P + IB - 1) / IB;
  return (int)sizeof(double) * (IB * (nb * IB + 4) + IB * IS + NB * IB * IS);
}

// Returns GPL_ERR_ARG when P is beyond the panel kernels' checked range.
int launch_inverse_panels(Ctx* c) {
  const int P = c->P;
  const int smem = inverse_panel_smem(P);
  if (P > kInverseMaxP || smem > 220 * 1024) return GPL_ERR_ARG;
  GPL_TRY(c, cudaFuncSetAttribute(k_trtri_panel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  GPL_TRY(c, cudaFuncSetAttribute(k_lauum_panel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  GPL_TRY(c, cudaFuncSetAttribute(k_trtri_panel, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
  GPL_TRY(c, cudaFuncSetAttribute(k_lauum_panel, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
  const int64_t st = (int64_t)P * P;
  const int nb = (P + IB - 1) / IB;
  k_tri_diag<<<(unsigned)(((int64_t)c->J * nb + 3) / 4), 128, 0, c->stream>>>(c->Psi, P, st, c->J * nb, c->scratch);
  GPL_LAUNCHED(c, "k_tri_diag");
  if (nb > 1) {
    k_trtri_panel<<<dim3(nb - 1, c->J), 256, smem, c->stream>>>(c->Psi, P, st, c->scratch);
    GPL_LAUNCHED(c, "k_trtri_panel");
  }
  const dim3 g(nb, c->J);
  k_lauum_panel<<<g, 256, smem, c->stream>>>(c->scratch, P, st, c->PsiInv);
  GPL_LAUNCHED(c, "k_lauum_panel");
  return GPL_OK;
}

}  // namespace gpl

namespace gpl {

// The per-gene tail of one IRLS sweep as ONE persistent launch (getBetaPhi's cholPsi, cholsl and
// coefficient update, then getLkhdPois: ggplvm.cu:683-692, 418-464, 703-724). Each CTA takes
// genes from a queue (an atomic head over `order`, the genes by decreasing matched count) and for each:
//   1. factors Psi_j in place (potrf_panel_one, as k_potrf_panel);
//   2. solves L L^T x = b_j with one warp, in k_solve's operation order, and stores x (sol);
//   3. beta_j <- (1 - r) beta_j + r x and phi_j from nu^T diag(W/Omega) nu - |L^T beta_j|^2 with
//      the reference's clamps, in k_beta_phi's order;
//   4. the Poisson log-likelihood of the gene's matched counts, in k_lkhd_pois's order.
// Every sum is taken in the same per-thread order and reduced by the same block tree as in the
// separate kernels, so the results are the same bits; which CTA takes which gene changes nothing.
// The W and nu columns are read once for steps 3 and 4 together.
__global__ void __launch_bounds__(256, 2)
    k_irls_tail(int J, int N, int ldN, int P, int pvars, double r, double wt, double* __restrict__ Psi,
                const double* __restrict__ bvec, double* __restrict__ sol, double* __restrict__ Beta,
                double* __restrict__ phi, const double* __restrict__ W, const double* __restrict__ Nu,
                const double* __restrict__ Omega, const double* __restrict__ delta,
                const double* __restrict__ titsias, const int32_t* __restrict__ cell,
                const int64_t* __restrict__ gptr, const int32_t* __restrict__ gvalid,
                const double* __restrict__ cnt, double* __restrict__ lkhds, const int* __restrict__ order,
                int* __restrict__ head, int ns, int sms) {
  extern __shared__ __align__(16) double sm[];
  __shared__ int fail, next;
  __shared__ double sh[32];
  const int rows_pad = max(IB, (P + 15) / 16 * 16);
  double* y = sm + (size_t)IB * (rows_pad + 2) + ns * (size_t)CW * (rows_pad + 4) + IB;  // past the panel's space
  double* sb = y + P;
  double* dg = sb + P;  // the factor's diagonal
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = blockDim.x >> 5;
  const int sw = (blockIdx.x / sms) & 3;  // the solving warp: not on the same SM partition as the neighbour's
  const int64_t PP = (int64_t)P * P;
  for (;;) {
    __syncthreads();  // the previous gene's shared values are no longer read
    if (tid == 0) next = atomicAdd(head, 1);
    __syncthreads();
    const int q = next;
    if (q >= J) break;
    const int j = order[q];
    double* L = Psi + (size_t)j * PP;
    potrf_panel_one<256>(L, P, ns, sms, sm, fail);
    __syncthreads();
    // 2. (L L^T) x = b_j, one warp, in k_solve's operation order (lane l updates the rows
    // k + 1 + l + 32 m of column k, and sums the rows i + 1 + l + 32 m of row i's column). The columns
    // pass through a ring in the panel's space, kRing - 1 of them in flight: with only the next one in
    // flight each of the 2 P steps waited for it (770,000 cycles at P = 232, against 330,000 for the
    // factorization)
    if (wid == sw) {
      constexpr int NR = (kPotrfMaxP + 31) / 32, kRing = 16;  // rows per lane, columns in the ring
      const int RS = rows_pad + 2;
      const bool pairs = (P & 1) == 0 && (reinterpret_cast<uintptr_t>(L) & 15) == 0;
      // rows below the diagonal of column k (from an even row when copied in pairs)
      auto fetch = [&](int k) {
        if (k >= 0 && k < P) {
          const double* src = L + (size_t)k * P;
          double* dst = sm + (k % kRing) * RS;
          if (pairs) {
            for (int r = ((k + 1) & ~1) + 2 * lane; r < P; r += 64) cp_async16(dst + r, src + r, 16);
          } else {
            for (int r = k + 1 + lane; r < P; r += 32) cp_async8(dst + r, src + r, 8);
          }
        }
        cp_async_commit();
      };
      const double* rhs = bvec + (size_t)j * P;
      for (int k = 0; k < kRing - 1; k++) fetch(k);
      double yr[NR], dr[NR];  // rows lane + 32 m
#pragma unroll
      for (int m = 0; m < NR; m++) {
        const int i = lane + 32 * m;
        yr[m] = i < P ? rhs[i] : 0.0;
        dr[m] = i < P ? L[i + (size_t)i * P] : 1.0;
        if (i < P) dg[i] = dr[m];
      }
#pragma unroll
      for (int kb = 0; kb < NR; kb++) {
        if (kb * 32 >= P) break;
        const int kn = min(32, P - kb * 32);
        for (int kk = 0; kk < kn; kk++) {
          const int k = kb * 32 + kk;
          const double xk = __shfl_sync(0xffffffffu, yr[kb] / dr[kb], kk);
          cp_async_wait<kRing - 2>();
          __syncwarp();  // column k is there, column k - 1 is no longer read
          fetch(k + kRing - 1);
          const double* col = sm + (k % kRing) * RS + lane;
          if (lane > kk && lane + 32 * kb < P) yr[kb] -= col[32 * kb] * xk;
          if (lane == kk) yr[kb] = xk;
#pragma unroll
          for (int m = kb + 1; m < NR; m++)
            if (lane + 32 * m < P) yr[m] -= col[32 * m] * xk;
        }
      }
#pragma unroll
      for (int m = 0; m < NR; m++)
        if (lane + 32 * m < P) y[lane + 32 * m] = yr[m];
      __syncwarp();
      for (int k = 0; k < kRing - 1; k++) fetch(P - 1 - k);
      for (int i = P - 1; i >= 0; i--) {
        cp_async_wait<kRing - 2>();
        __syncwarp();
        fetch(i - (kRing - 1));
        const double* col = sm + (i % kRing) * RS + i + 1 + lane;
        const double* ys = y + i + 1 + lane;
        const double yi = y[i], di = dg[i];
        double part = 0.0, cv[NR], yv[NR];
#pragma unroll
        for (int m = 0; m < NR; m++) {
          const bool in = i + 1 + lane + 32 * m < P;
          cv[m] = in ? col[32 * m] : 0.0;
          yv[m] = in ? ys[32 * m] : 0.0;
        }
#pragma unroll
        for (int m = 0; m < NR; m++)
          if (i + 1 + lane + 32 * m < P) part += cv[m] * yv[m];
        part = warp_sum(part);
        const double xi = (yi - part) / di;
        __syncwarp();
        if (lane == 0) y[i] = xi;
      }
      __syncwarp();
      double* x = sol + (size_t)j * P;
      for (int i = lane; i < P; i += 32) x[i] = y[i];
    }
    // 3. and 4.: one pass over the gene's cells for both per-cell sums
    const double* Wj = W + (size_t)j * ldN;
    const double* nj = Nu + (size_t)j * ldN;
    double qpart = 0.0, lpart = 0.0;
    in_order<8>(
        tid, N, 256, [&](int i) { return make_double3(nj[i], Wj[i], Omega[i]); },
        [&](const double3& v) {
          qpart += v.x * v.x * v.y / v.z;
          lpart -= v.y;
        });
    const int64_t b0 = gptr[j], b1 = gptr[j] + gvalid[j];
    const double dgp = delta[pvars - 1];
    in_order<4>(
        b0 + tid, b1, 256, [&](int64_t l) { return CountAt{cell[l], cnt[l]}; },
        [&](const CountAt& x) { return make_double2(Wj[x.cell], titsias[x.cell]); },
        [&](const CountAt& x, const double2& v) { lpart += (log(v.x) - dgp * v.y * wt) * x.y; });
    const double quad = block_sum(qpart, sh);  // syncs: the solution y is complete
    double* bj = Beta + (size_t)j * P;
    for (int k = tid; k < P; k += blockDim.x) {
      const double nb = bj[k] * (1 - r) + y[k] * r;
      bj[k] = nb;
      sb[k] = nb;
    }
    __syncthreads();
    double sq = 0.0;
    for (int k = wid; k < P; k += nw) {
      double t = 0.0;
      for (int i = k + lane; i < P; i += 32) t += L[i + (size_t)k * P] * sb[i];
      t = warp_sum(t);
      sq += t * t;
    }
    if (lane != 0) sq = 0.0;
    const double s2 = block_sum(sq, sh);
    const double lk = block_sum(lpart, sh);
    if (tid == 0) {
      double ph = (quad - s2) / (double)N;
      if (isnan(ph)) ph = 1.0;
      if (ph < 0.0) ph = 1.0;
      if (ph < 0.01) ph = 0.01;
      if (ph > 1000.0) ph = 1000.0;
      phi[j] = ph;
      lkhds[j] = lk;
    }
  }
}

// GPL_ERR_ARG when the fused tail does not apply: P beyond the panel Cholesky's range, or more genes
// than CTAs that can be resident. Up to there the one launch saves the gaps and the tails of four
// (separate / fused, P = 36: 290 genes 101 / 95 us; P = 72: 337 / 222; P = 232: 1.13 / 0.79 ms); beyond,
// a CTA's genes run one after another, each bound by its own chain, where the separate kernels give
// every step its own grid (600 genes: 138 / 238 us at P = 36, 402 / 515 at 72; 2,001 genes at 232:
// 2.45 / 3.85 ms).
int launch_irls_tail(Ctx* c, int jtr, int ctas_per_sm) {
  const int P = c->P;
  const int vecs = 3 * (int)sizeof(double) * P, ns = potrf_buffers(P, vecs), smem = potrf_panel_smem(P, ns) + vecs;
  if (P > kPotrfMaxP || smem > 220 * 1024 || !c->gene_order_d || c->J > 2 * c->sm_count) return GPL_ERR_ARG;
  GPL_TRY(c, cudaFuncSetAttribute(k_irls_tail, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  GPL_TRY(c, cudaFuncSetAttribute(k_irls_tail, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
  double r = (double)(jtr + 1) / 100.0;  // the damping of getBetaPhi (ggplvm.cu:426)
  if (jtr > 100) r = 1.0;
  Tunable* tu = nullptr;
  ctas_per_sm = tune_pick(c, "irls_tail", {1, 2}, ctas_per_sm, &tu);
  const int grid = std::max(1, std::min(c->J, std::max(1, ctas_per_sm) * c->sm_count));
  GPL_TRY(c, cudaMemsetAsync(c->queue_head_d, 0, sizeof(int), c->stream));
  ProfScope ps(c, "irls_tail");
  TuneScope ts(c, tu);
  k_irls_tail<<<grid, 256, smem, c->stream>>>(c->J, c->N, c->ldN, P, c->p, r, c->vcomp ? 1.0 : kWt, c->Psi, c->bvec,
                                              c->sol, c->Beta, c->phi, c->W, c->Nu, c->Omega, c->delta,
                                              c->titsias, c->cell, c->gptr, c->gvalid, c->cnt, c->lkhds,
                                              c->gene_order_d, c->queue_head_d, ns, c->sm_count);
  GPL_LAUNCHED(c, "k_irls_tail");
  return GPL_OK;
}

}  // namespace gpl
