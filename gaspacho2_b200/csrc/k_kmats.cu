// Kernel matrices of the sparse GP (replaces kernel_funcs.cu:61-162 and util_cuda.cu:249-269).
//
//   k_knm        Knm[i, m] = exp(-(sin^2((x_i0 - t_m0)/2)/rho_0 + sum_q>=1 (x_iq - t_mq)^2/(2 rho_q)))
//                written into the model matrix's GP block (column-major, cell fastest); with
//                lv >= 0 only latent dimension lv enters (the DE driver's per-dimension models).
//                Bound: N*M*Q transcendental work, ~2% of one objective evaluation.
//   k_kmm        Kmm (upper, unit diagonal, zero lower) and its copy Kinv.
//   k_kmm_solve  per cell: x = Kmm^{-1} k_n against the factor in Kinv's lower triangle (cholslg),
//                titsias_n = (1 - k_n . x)/2; also Kmm^{-1} itself. A cell per thread, 32-row blocks
//                of the solution in registers.
//   k_expand     DeltaInv = blockdiag(1/delta_k I, Kmm/delta_GP), upper + diagonal.
#include <algorithm>

#include "dmma_common.cuh"
#include "gpl_internal.cuh"

namespace gpl {

// Squared-distance sum of one point pair: all latent dimensions (periodic dim 0, ARD dims
// >= 1; getKernelMatsWithPer) when lv < 0, dimension lv alone otherwise
// (getKernelMatsWithPerSpecificLV, kernel_funcs.cu:101-135), in the reference's order.
__device__ __forceinline__ double kern_sum(const double* __restrict__ A, size_t lda, int a,
                                           const double* __restrict__ B, int ldb, int b,
                                           const double* __restrict__ rho, int Q, int lv) {
  double sum = 0.0, t;
  if (lv <= 0) {
    t = sin((A[a] - B[b]) / 2.0);
    sum += t * t / rho[0];
  }
  const int k0 = lv < 0 ? 1 : lv, k1 = lv < 0 ? Q : (lv == 0 ? 0 : lv + 1);
  for (int k = k0; k < k1; k++) {
    t = A[a + k * lda] - B[b + k * ldb];
    sum += t * t / 2.0 / rho[k];
  }
  return sum;
}

__global__ void k_knm(int N, int ldN, int M, int Q, int lv, const double* __restrict__ X,
                      const double* __restrict__ T, const double* __restrict__ rho, double* __restrict__ Knm) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y;
  if (i >= N) return;
  Knm[i + (size_t)j * ldN] = exp(-kern_sum(X, (size_t)N, i, T, M, j, rho, Q, lv));
}

__global__ void k_kmm(int M, int Q, int lv, const double* __restrict__ T, const double* __restrict__ rho,
                      double* __restrict__ K, double* __restrict__ Kinv) {
  const int ii = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y;
  if (ii >= M) return;
  double val;
  if (ii == j) val = 1.0;
  else if (ii > j) val = 0.0;
  else val = exp(-kern_sum(T, (size_t)M, ii, T, M, j, rho, Q, lv));
  K[ii + j * M] = val;
  if (Kinv) Kinv[ii + j * M] = val;  // no copy when the caller needs Kmm once (Kinv == nullptr)
}

// The DE driver's null model as a design whose GP block is inert: Knm = 0, Kmm = Kinv = I,
// Kmm^{-1} k_n = 0, titsias = 0 (initTitsias). The GP columns then decouple from the rest of
// every Psi_j (their Gram entries vanish, DeltaInv holds 1/delta_GP on their diagonal), and
// their coefficients stay 0.
__global__ void k_gp_null(int N, int ldN, int M, double* __restrict__ Knm, double* __restrict__ KinvKmn,
                          double* __restrict__ titsias, double* __restrict__ K, double* __restrict__ Kinv) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < ldN)
    for (int m = 0; m < M; m++) {
      Knm[i + (size_t)m * ldN] = 0.0;
      KinvKmn[i + (size_t)m * ldN] = 0.0;
    }
  if (i < N) titsias[i] = 0.0;
  if (i < M * M) K[i] = Kinv[i] = (i % M == i / M) ? 1.0 : 0.0;
}

// x_i = (L L^T)^{-1} b_i for many right-hand sides (one per cell), L the lower factor in A's lower
// triangle (M x M, column-major): a cell per thread, 32 rows of its solution in registers, so that two
// multiply-adds come from one broadcast load of L and every finished Y is read once per later block
// of rows instead of once per row. Bound: N M^2 FP64 operations; a row-at-a-time substitution re-read
// Y through L2 for every multiply-add (13 GB at N = 100,000, M = 128). kUnit: b_i = the i-th unit
// vector (Kmm^{-1} of getC2, ggplvm.cu:93-95, the solution's column i at Y + i * ldY); else b_i =
// column i of Knm^T, and titsias_i = (1 - k_i . x_i)/2.
// kExact (M <= 32, one block): the sums keep cholslg's order (chol.cu:86-97) without contracted
// multiply-adds, so that with few inducing points, where Kmm (no jitter in the reference) is often
// nearly singular, the solution has the reference's bits. Otherwise multiply-adds in ascending order
// and reciprocals of the diagonal: the error against extended precision is the row-at-a-time form's
// (it is set by the factor, which keeps choldc's order): 2.7e-12 of the solution at cond(Kmm) = 5e5
// against 3.0e-12, 1e-13 at 1e4 for both. At N = 100,000, M = 128: 1.58 -> 0.43 ms.
constexpr int kSolveCells = 64, kSolveAhead = 8;
template <bool kUnit, bool kExact>
__global__ void __launch_bounds__(kSolveCells, 8)
    k_kmm_solve(int N, int64_t ldN, int M, const double* __restrict__ A, const double* __restrict__ B, double* Y,
                double* __restrict__ titsias) {
  __shared__ __align__(16) double Ls[2][32][32];  // [k][row of the block]
  __shared__ double Rd[32];
  const int tid = threadIdx.x;
  const int i = blockIdx.x * kSolveCells + tid;
  const bool on = i < N;
  // element (row r, cell i) of Y; threads past N follow cell N - 1 and store nothing
  const size_t rs = kUnit ? 1 : (size_t)ldN, cs = kUnit ? (size_t)ldN : 1;
  double* y = Y + (size_t)min(i, N - 1) * cs;
  const double* b = kUnit ? nullptr : B + min(i, N - 1);
  const int nb = (M + 31) / 32;
  double d = 0.0;

  for (int pass = 0; pass < 2; pass++) {
    for (int q = 0; q < nb; q++) {
      const int ib = pass == 0 ? q : nb - 1 - q;
      const int r0 = ib * 32, nr = min(32, M - r0);
      // rows of L (forward) or columns of L (backward) of this block against the finished ones
      const int kbeg = pass == 0 ? 0 : r0 + 32, kend = pass == 0 ? r0 : M;
      auto stage = [&](int k0, int buf) {
        for (int e = tid; e < 1024; e += kSolveCells) {
          const int r = pass == 0 ? e & 31 : e >> 5, k = pass == 0 ? e >> 5 : e & 31;
          const bool in = k0 + k < kend && r < nr;
          const size_t at = pass == 0 ? (size_t)(r0 + r) + (size_t)(k0 + k) * M : (size_t)(k0 + k) + (size_t)(r0 + r) * M;
          Ls[buf][k][r] = in ? A[at] : 0.0;
        }
      };
      // eight finished values, zeros from kend on
      auto ahead = [&](int k0, double (&v)[kSolveAhead]) {
#pragma unroll
        for (int u = 0; u < kSolveAhead; u++) v[u] = k0 + u < kend ? y[(size_t)(k0 + u) * rs] : 0.0;
      };
      double x[32];
#pragma unroll
      for (int r = 0; r < 32; r++) {
        if (pass == 0) x[r] = r >= nr ? 0.0 : kUnit ? (r0 + r == i ? 1.0 : 0.0) : b[(size_t)(r0 + r) * ldN];
        else x[r] = r < nr ? y[(size_t)(r0 + r) * rs] : 0.0;
      }
      int buf = 0;
      double next[kSolveAhead];
      if (kbeg < kend) {
        stage(kbeg, 0);
        ahead(kbeg, next);
      }
      for (int k0 = kbeg; k0 < kend; k0 += 32, buf ^= 1) {
        __syncthreads();
        if (k0 + 32 < kend) stage(k0 + 32, buf ^ 1);
#pragma unroll 1
        for (int k = 0; k < 32; k += kSolveAhead) {
          double v[kSolveAhead];
#pragma unroll
          for (int u = 0; u < kSolveAhead; u++) v[u] = next[u];
          ahead(k0 + k + kSolveAhead, next);
#pragma unroll
          for (int u = 0; u < kSolveAhead; u++) {
            const double2* l = reinterpret_cast<const double2*>(Ls[buf][k + u]);
#pragma unroll
            for (int r = 0; r < 16; r++) {
              const double2 w = l[r];
              x[2 * r] = fma(-w.x, v[u], x[2 * r]);
              x[2 * r + 1] = fma(-w.y, v[u], x[2 * r + 1]);
            }
          }
        }
      }
      // the 32 x 32 diagonal block: Ls[0][k][r] = L[r][k], k < r (forward), or L[k][r], k > r (backward)
      __syncthreads();
      for (int e = tid; e < 1024; e += kSolveCells) {
        const int r = pass == 0 ? e & 31 : e >> 5, k = pass == 0 ? e >> 5 : e & 31;
        const bool in = r < nr && k < nr && (pass == 0 ? r > k : k > r);
        const size_t at = pass == 0 ? (size_t)(r0 + r) + (size_t)(r0 + k) * M : (size_t)(r0 + k) + (size_t)(r0 + r) * M;
        Ls[0][k][r] = in ? A[at] : 0.0;
      }
      if (tid < 32) {
        const double v = tid < nr ? A[(size_t)(r0 + tid) * (M + 1)] : 1.0;
        Rd[tid] = kExact ? v : 1.0 / v;
      }
      __syncthreads();
      if (kExact && pass == 0) {
#pragma unroll
        for (int r = 0; r < 32; r++) {
          if (r < nr) {
#pragma unroll
            for (int k = r - 1; k >= 0; k--) x[r] = __dsub_rn(x[r], __dmul_rn(Ls[0][k][r], x[k]));
            x[r] = __ddiv_rn(x[r], Rd[r]);
          }
        }
      } else if (kExact) {
#pragma unroll
        for (int r = 31; r >= 0; r--) {
          if (r < nr) {
#pragma unroll
            for (int k = r + 1; k < 32; k++)
              if (k < nr) x[r] = __dsub_rn(x[r], __dmul_rn(Ls[0][k][r], x[k]));
            x[r] = __ddiv_rn(x[r], Rd[r]);
          }
        }
      } else if (pass == 0) {
#pragma unroll
        for (int k = 0; k < 32; k++) {
          x[k] *= Rd[k];
#pragma unroll
          for (int r = k + 1; r < 32; r++) x[r] = fma(-Ls[0][k][r], x[k], x[r]);
        }
      } else {
#pragma unroll
        for (int k = 31; k >= 0; k--) {
          x[k] *= Rd[k];
#pragma unroll
          for (int r = 0; r < k; r++) x[r] = fma(-Ls[0][k][r], x[k], x[r]);
        }
      }
#pragma unroll
      for (int r = 0; r < 32; r++)
        if (r < nr && on) y[(size_t)(r0 + r) * rs] = x[r];
      __syncthreads();  // Ls is refilled
    }
  }
  if (!kUnit && on) {
    for (int k = 0; k < M; k++) d = __dadd_rn(d, __dmul_rn(b[(size_t)k * ldN], y[(size_t)k * rs]));
    titsias[i] = (1.0 - d) / 2.0;
  }
}

// The same in cholslg's order for any M, a row at a time, where the order is kept (OrderScope,
// gpl_internal.cuh). A cell per thread, its solution in shared memory, the factor's next row (forward) or column
// (backward) copied there while the last one is used. Bound: the chain of M^2 subtractions per cell with few
// cells, the reads of the solution (two wavefronts a step and warp) with many. At N = 20,003, M = 128: 1.04 ms from
// global memory throughout, 0.33 ms so (k_kmm_solve: 0.15).
constexpr int kRowsCells = 64;
__global__ void __launch_bounds__(kRowsCells) k_kmm_solve_rows(int N, int ldN, int M, const double* __restrict__ L,
                                                               const double* __restrict__ Knm, double* __restrict__ Y,
                                                               double* __restrict__ titsias) {
  extern __shared__ __align__(16) double rows_sm[];
  double* ys = rows_sm + threadIdx.x;                // [M][kRowsCells]
  double* Ls = rows_sm + (size_t)M * kRowsCells;     // [2][M]
  const int i = blockIdx.x * kRowsCells + threadIdx.x;
  const bool on = i < N;
  const double* b = Knm + min(i, N - 1);
  // row r: L[r, 0 .. r]; column r: L[r .. M - 1, r] at its own rows
  auto stage = [&](int r, bool forward, int buf) {
    double* d = Ls + (size_t)buf * M;
    if (forward) {
      for (int k = threadIdx.x; k <= r; k += kRowsCells) cp_async8(d + k, L + r + (size_t)k * M, 8);
    } else {
      for (int k = r + threadIdx.x; k < M; k += kRowsCells) cp_async8(d + k, L + k + (size_t)r * M, 8);
    }
  };
  stage(0, true, 0);
  cp_async_commit();
  for (int step = 0; step < 2 * M; step++) {
    const bool forward = step < M;
    const int r = forward ? step : 2 * M - 1 - step;
    cp_async_wait<0>();
    __syncthreads();  // this row is there, and the buffer loaded next is no longer read
    if (step + 1 < 2 * M) stage(step + 1 < M ? step + 1 : 2 * M - 2 - step, step + 1 < M, (step + 1) & 1);
    cp_async_commit();
    const double* l = Ls + (size_t)(step & 1) * M;
    double sum = forward ? b[(size_t)r * ldN] : ys[(size_t)r * kRowsCells];
    if (forward) {
#pragma unroll 8
      for (int k = r - 1; k >= 0; k--) sum = __dsub_rn(sum, __dmul_rn(l[k], ys[(size_t)k * kRowsCells]));
    } else {
#pragma unroll 8
      for (int k = r + 1; k < M; k++) sum = __dsub_rn(sum, __dmul_rn(l[k], ys[(size_t)k * kRowsCells]));
    }
    sum = __ddiv_rn(sum, l[r]);
    ys[(size_t)r * kRowsCells] = sum;
    if (!forward && on) Y[i + (size_t)r * ldN] = sum;
  }
  if (!on) return;
  double d = 0.0;
  for (int k = 0; k < M; k++) d = __dadd_rn(d, __dmul_rn(b[(size_t)k * ldN], ys[(size_t)k * kRowsCells]));
  titsias[i] = (1.0 - d) / 2.0;
}
// The same with the solution in global memory, for more inducing points than that one holds.
__global__ void k_kmm_solve_rows_any(int N, int ldN, int M, const double* __restrict__ L,
                                     const double* __restrict__ Knm, double* __restrict__ Y,
                                     double* __restrict__ titsias) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  for (int r = 0; r < M; r++) {
    double sum = Knm[i + (size_t)r * ldN];
    for (int k = r - 1; k >= 0; k--) sum = __dsub_rn(sum, __dmul_rn(L[r + k * M], Y[i + (size_t)k * ldN]));
    Y[i + (size_t)r * ldN] = __ddiv_rn(sum, L[r + r * M]);
  }
  for (int r = M - 1; r >= 0; r--) {
    double sum = Y[i + (size_t)r * ldN];
    for (int k = r + 1; k < M; k++) sum = __dsub_rn(sum, __dmul_rn(L[k + r * M], Y[i + (size_t)k * ldN]));
    Y[i + (size_t)r * ldN] = __ddiv_rn(sum, L[r + r * M]);
  }
  double d = 0.0;
  for (int k = 0; k < M; k++) d = __dadd_rn(d, __dmul_rn(Knm[i + (size_t)k * ldN], Y[i + (size_t)k * ldN]));
  titsias[i] = (1.0 - d) / 2.0;
}

int launch_cholinv(Ctx* c, const double* L, int n, double* out) {
  auto fn = n <= 32 ? k_kmm_solve<true, true> : k_kmm_solve<true, false>;
  fn<<<div_up(n, kSolveCells), kSolveCells, 0, c->stream>>>(n, n, n, L, nullptr, out, nullptr);
  GPL_LAUNCHED(c, "k_kmm_solve");
  return GPL_OK;
}

__global__ void k_expand(int P, int p, int g0, int M, const int* __restrict__ mk, const double* __restrict__ delta,
                         const double* __restrict__ K, double* __restrict__ D) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  const int col = blockIdx.y;
  if (r >= P) return;
  double v = 0.0;
  if (r <= col) {
    if (r >= g0) v = K[(r - g0) + (col - g0) * M] / delta[p - 1];
    else if (r == col) v = 1.0 / delta[mk[r]];
  }
  D[r + (size_t)col * P] = v;
}

// Knm, Kmm and its factor, Kmm^{-1} k_n and titsias over the latent dimensions of c->kernel_lv.
int launch_kernel_mats(Ctx* c) {
  const int lv = c->kernel_lv;
  c->Dg_done = false;  // the kernel columns of Dm are written
  double* Knm = c->Dm + (size_t)c->dg0 * c->ldN;
  if (lv == kLvNone) {
    ProfScope ps(c, "kernel_mats");
    const int n = std::max(c->ldN, c->M * c->M);
    k_gp_null<<<div_up(n, 256), 256, 0, c->stream>>>(c->N, c->ldN, c->M, Knm, c->KinvKmn, c->titsias, c->Kmm,
                                                     c->Kinv);
    GPL_LAUNCHED(c, "k_gp_null");
    return GPL_OK;
  }
  {
    ProfScope ps(c, "kernel_mats");
    dim3 g2(div_up(c->M, 64), c->M);
    k_kmm<<<g2, 64, 0, c->stream>>>(c->M, c->Q, lv, c->T, c->rho, c->Kmm, c->Kinv);
    GPL_LAUNCHED(c, "k_kmm");
  }
  const int rc = launch_chol_single(c, c->Kinv, c->M);
  return rc ? rc : launch_kernel_cells(c);
}

int launch_kernel_cells(Ctx* c) {
  double* Knm = c->Dm + (size_t)c->dg0 * c->ldN;
  {
    ProfScope ps(c, "kernel_mats");
    dim3 g(div_up(c->N, 128), c->M);
    k_knm<<<g, 128, 0, c->stream>>>(c->N, c->ldN, c->M, c->Q, c->kernel_lv, c->X, c->T, c->rho, Knm);
    GPL_LAUNCHED(c, "k_knm");
  }
  ProfScope ps(c, "kinvkmn");
  if ((c->one_order || c->de) && c->M > 32) {  // the undamped drivers' contexts
    const size_t smem = sizeof(double) * c->M * (kRowsCells + 2);
    if (smem > 220 * 1024) {  // more than 426 inducing points
      k_kmm_solve_rows_any<<<div_up(c->N, 128), 128, 0, c->stream>>>(c->N, c->ldN, c->M, c->Kinv, Knm, c->KinvKmn,
                                                                     c->titsias);
      GPL_LAUNCHED(c, "k_kmm_solve_rows_any");
      return GPL_OK;
    }
    GPL_TRY(c, cudaFuncSetAttribute(k_kmm_solve_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k_kmm_solve_rows<<<div_up(c->N, kRowsCells), kRowsCells, smem, c->stream>>>(c->N, c->ldN, c->M, c->Kinv, Knm,
                                                                               c->KinvKmn, c->titsias);
    GPL_LAUNCHED(c, "k_kmm_solve_rows");
    return GPL_OK;
  }
  auto fn = c->M <= 32 ? k_kmm_solve<false, true> : k_kmm_solve<false, false>;
  fn<<<div_up(c->N, kSolveCells), kSolveCells, 0, c->stream>>>(c->N, c->ldN, c->M, c->Kinv, Knm, c->KinvKmn,
                                                               c->titsias);
  GPL_LAUNCHED(c, "k_kmm_solve");
  return GPL_OK;
}

int launch_expand_delta(Ctx* c) {
  ProfScope ps(c, "expand_delta");
  dim3 g(div_up(c->P, 128), c->P);
  k_expand<<<g, 128, 0, c->stream>>>(c->P, c->p, c->nh[c->p - 1], c->M, c->mk_d, c->delta, c->Kmm, c->DeltaInv);
  GPL_LAUNCHED(c, "k_expand");
  return GPL_OK;
}

// The kernel-matrix sequence on caller-supplied buffers, without a context: Knm and the
// cell-fastest Kmm^{-1} k_n (both N x M, ld N), titsias (N), and an M x M work matrix that
// receives Kmm and then its factor. Each launch goes through cudaLaunchKernel, whose return
// value is that launch's own status (an error left on the thread by earlier, unrelated work is
// neither reported nor cleared). Returns the first failing launch's cudaError_t, else
// cudaSuccess.
int launch_kernel_mats_raw(cudaStream_t st, int N, int M, int Q, const double* X, const double* T,
                           const double* rho, double* Knm, double* KinvKmn, double* titsias, double* Lwork) {
  int ldN = N, lv = kLvAll;
  double* no_copy = nullptr;
  void* a_knm[] = {&N, &ldN, &M, &Q, &lv, &X, &T, &rho, &Knm};
  cudaError_t e = cudaLaunchKernel((const void*)k_knm, dim3(div_up(N, 128), M), dim3(128), a_knm, 0, st);
  if (e != cudaSuccess) return (int)e;
  void* a_kmm[] = {&M, &Q, &lv, &T, &rho, &Lwork, &no_copy};
  e = cudaLaunchKernel((const void*)k_kmm, dim3(div_up(M, 64), M), dim3(64), a_kmm, 0, st);
  if (e != cudaSuccess) return (int)e;
  e = launch_chol_exact_raw(st, Lwork, M);
  if (e != cudaSuccess) return (int)e;
  const double* L = Lwork;
  int64_t ld = N;
  void* a_kk[] = {&N, &ld, &M, &L, &Knm, &KinvKmn, &titsias};
  auto fn = M <= 32 ? k_kmm_solve<false, true> : k_kmm_solve<false, false>;
  e = cudaLaunchKernel((const void*)fn, dim3(div_up(N, kSolveCells)), dim3(kSolveCells), a_kk, 0, st);
  return (int)e;
}

}  // namespace gpl
