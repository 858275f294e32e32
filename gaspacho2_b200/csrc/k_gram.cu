// Per-gene Gram matrices and their factorisations (replaces getPsi ggplvm.cu:621-680,
// cholPsi :683-692, cholDeltaInv :695-700, cholKmm kernel_funcs.cu:139-143, solvePsi
// ggplvm.cu:46-53, choldc/cholsl chol.cu:19-97, initPsi init.cu:125-181).
//
//   k_chol_exact  one matrix in choldc's operation order (Kmm, the prior, the GLM Gram).
//   k_chol      one matrix wider than that kernel's row slots, or a batch within an OrderScope,
//               left-looking by columns: the update of column j reads row j of the factor
//               (broadcast) and the rows below it (coalesced). A non-positive pivot zero-fills
//               the matrix, as choldc does.
//   k_solve     batched (L L^T) x = b, one warp per system: forward substitution column-
//               oriented (coalesced), back substitution as warp dot products.
//   k_trtri     V = L^{-1} (row-major scratch), one thread per column of V.
//   k_lauum     Psi^{-1} = V^T V, full symmetric, column-major.
#include "gpl_internal.cuh"

namespace gpl {

// Left-looking Cholesky of n x n matrices A_b = A + b*stride (col-major, ld n). The input is
// read from the upper triangle (src_upper) or the lower one; the factor overwrites the
// lower triangle and the diagonal; the strict upper triangle is left as it was.
__global__ void __launch_bounds__(256) k_chol(double* __restrict__ A, int n, int64_t stride, int src_upper) {
  __shared__ double sh[32];
  __shared__ int fail;
  double* a = A + (size_t)blockIdx.x * stride;
  const int tid = threadIdx.x;
  if (tid == 0) fail = 0;
  __syncthreads();
  for (int j = 0; j < n; j++) {
    // pivot: d = A(j,j) - sum_k L(j,k)^2
    double part = 0.0;
    for (int k = tid; k < j; k += blockDim.x) {
      const double l = a[j + (size_t)k * n];
      part = fma(l, l, part);
    }
    const double s = block_sum(part, sh);
    const double d = a[j + (size_t)j * n] - s;
    if (d <= 0.0) fail = 1;  // a NaN pivot passes, as in choldc, and yields a NaN factor
    __syncthreads();
    if (fail) break;
    const double ljj = sqrt(d);
    for (int i = j + 1 + tid; i < n; i += blockDim.x) {
      double acc = src_upper ? a[j + (size_t)i * n] : a[i + (size_t)j * n];
      for (int k = j - 1; k >= 0; k--) acc -= a[i + (size_t)k * n] * a[j + (size_t)k * n];
      a[i + (size_t)j * n] = acc / ljj;
    }
    __syncthreads();
    if (tid == 0) a[j + (size_t)j * n] = ljj;
    __syncthreads();
  }
  if (fail) {
    for (int e = tid; e < n * n; e += blockDim.x) a[e] = 0.0;
  }
}

// Single-matrix Cholesky in choldc's exact operation order (chol.cu:19-43): row i of the
// factor is finished before row i+1, each entry's sum runs k = i-1 .. 0, and no multiply-add
// is contracted, so identical inputs give the host reference's bits (sqrt and division are
// correctly rounded on both). Used for the small, often ill-conditioned matrices: Kmm (no
// jitter in the reference), the prior precision DeltaInv and the GLM initialisation Gram.
// Reads the upper triangle, writes the factor into the lower one; zero-fills on a
// non-positive pivot. One CTA: the bound is the dependent chain of n^2/2 subtractions. The factor's
// columns k >= k0 stay in shared memory (packed, rows j >= k contiguous), the ones that do not fit
// are read back from global memory at the end of each chain. At n = 128: 0.58 ms from global
// memory throughout, 0.18 ms so.
// The first `diag` rows hold nothing off the diagonal (the prior's covariate part): their factor is
// the square root of the diagonal, the products they contribute to later rows are exact zeros and
// are left out, unless a diagonal entry is not finite.
constexpr int kCholThreads = 256;
__global__ void __launch_bounds__(kCholThreads) k_chol_exact(double* __restrict__ a, int n, int diag, int k0) {
  extern __shared__ double ls[];  // column k >= k0, row j at off(k) + j
  __shared__ int fail, odd;
  __shared__ double piv;
  const int tid = threadIdx.x;
  if (tid == 0) fail = odd = 0;
  __syncthreads();
  for (int k = tid; k < diag; k += kCholThreads) {
    const double d = a[k + (size_t)k * n];
    if (d <= 0.0) fail = 1;
    if (!isfinite(d)) odd = 1;
  }
  __syncthreads();
  const bool bad = fail != 0;
  const int i_first = bad ? n : odd ? 0 : diag;
  if (!bad && !odd)
    for (int e = tid; e < diag * n; e += kCholThreads) {  // the lower triangle of the diagonal rows' columns
      const int k = e / n, j = e - k * n;
      if (j == k) a[e] = __dsqrt_rn(a[e]);
      else if (j > k) a[e] = 0.0;
    }
  __syncthreads();
  const int k_low = odd ? 0 : diag;  // first column whose products are taken
  auto off = [&](int k) { return (k - k0) * n - (k * (k - 1) / 2 - k0 * (k0 - 1) / 2) - k; };
  // a thread keeps its columns j = tid, tid + 256, ..; the next row's entries are loaded one row ahead
  double sums[4], next[4];
#pragma unroll
  for (int c = 0; c < 4; c++) {
    const int j = tid + c * kCholThreads;
    next[c] = i_first < n && j >= i_first && j < n ? a[i_first + (size_t)j * n] : 0.0;
  }
  for (int i = i_first; i < n; i++) {
    // sums for j = i .. n-1 (j = i is the pivot)
#pragma unroll
    for (int c = 0; c < 4; c++) {
      const int j = tid + c * kCholThreads;
      if (j < i || j >= n) continue;
      double sum = next[c];
      next[c] = j > i ? a[i + 1 + (size_t)j * n] : 0.0;
      int k = i - 1;
      const int ks = max(k0, k_low);
      const double *li = ls + (k >= ks ? off(k) + i : 0), *lj = li + (j - i);
#pragma unroll 8
      for (; k >= ks; k--) {
        sum = __dsub_rn(sum, __dmul_rn(*li, *lj));
        li -= n - k;  // off(k - 1) = off(k) - (n - k)
        lj -= n - k;
      }
#pragma unroll 8
      for (; k >= k_low; k--) sum = __dsub_rn(sum, __dmul_rn(a[i + (size_t)k * n], a[j + (size_t)k * n]));
      sums[c] = sum;
      if (j == i) {
        if (sum <= 0.0) fail = 1;
        else piv = __dsqrt_rn(sum);
      }
    }
    __syncthreads();
    if (fail) break;
    const double lii = piv;
#pragma unroll
    for (int c = 0; c < 4; c++) {
      const int j = tid + c * kCholThreads;
      if (j < i || j >= n) continue;
      const double v = j > i ? __ddiv_rn(sums[c], lii) : lii;
      a[j + (size_t)i * n] = v;
      if (i >= k0) ls[off(i) + j] = v;
    }
    __syncthreads();
  }
  __syncthreads();
  if (fail)
    for (int e = tid; e < n * n; e += kCholThreads) a[e] = 0.0;
}

// (L L^T) x = b for `batch` systems, one warp each; y in shared memory, the factor's next columns in
// registers two steps ahead (NR rows per lane), so that the dependent chain does not wait on a load
// per step. The same operations in the same order for every NR. 3,000 systems of 236: 0.70 ms with the
// loads in the chain, 0.37 ms so.
template <int NR>
__global__ void __launch_bounds__(128) k_solve(const double* __restrict__ L, int n, int64_t lstride,
                                               const double* __restrict__ B, int64_t bstride, double* __restrict__ X,
                                               int64_t xstride, int batch) {
  extern __shared__ double sy[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int b = blockIdx.x * (blockDim.x >> 5) + warp;
  if (b >= batch) return;
  double* y = sy + (size_t)warp * 2 * n;
  double* dg = y + n;  // the factor's diagonal
  const double* a = L + (size_t)b * lstride;
  const double* rhs = B + (size_t)b * bstride;
  double* x = X + (size_t)b * xstride;
  for (int i = lane; i < n; i += 32) {
    y[i] = rhs[i];
    dg[i] = a[i + (size_t)i * n];
  }
  // rows k + 1 + lane + 32 m of column k
  auto col = [&](int k, double (&c)[NR]) {
#pragma unroll
    for (int m = 0; m < NR; m++) {
      const int i = k + 1 + lane + 32 * m;
      c[m] = k >= 0 && i < n ? a[i + (size_t)k * n] : 0.0;
    }
  };
  double c0[NR], c1[NR], c2[NR];
  col(0, c0);
  col(1, c1);
  __syncwarp();
  for (int k = 0; k < n; k++) {
    col(k + 2, c2);
    const double xk = y[k] / dg[k];
    __syncwarp();
    if (lane == 0) y[k] = xk;
#pragma unroll
    for (int m = 0; m < NR; m++) {
      const int i = k + 1 + lane + 32 * m;
      if (i < n) y[i] -= c0[m] * xk;
    }
    __syncwarp();
#pragma unroll
    for (int m = 0; m < NR; m++) {
      c0[m] = c1[m];
      c1[m] = c2[m];
    }
  }
  col(n - 1, c0);
  col(n - 2, c1);
  for (int i = n - 1; i >= 0; i--) {
    col(i - 2, c2);
    double part = 0.0;
#pragma unroll
    for (int m = 0; m < NR; m++) {
      const int k = i + 1 + lane + 32 * m;
      if (k < n) part += c0[m] * y[k];
    }
    part = warp_sum(part);
    const double xi = (y[i] - part) / dg[i];
    __syncwarp();
    if (lane == 0) y[i] = xi;
    __syncwarp();
#pragma unroll
    for (int m = 0; m < NR; m++) {
      c0[m] = c1[m];
      c1[m] = c2[m];
    }
  }
  for (int i = lane; i < n; i += 32) x[i] = y[i];
}

// The same for any n, the factor read where it is used.
__global__ void k_solve_any(const double* __restrict__ L, int n, int64_t lstride, const double* __restrict__ B,
                            int64_t bstride, double* __restrict__ X, int64_t xstride, int batch) {
  extern __shared__ double sy[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int b = blockIdx.x * (blockDim.x >> 5) + warp;
  if (b >= batch) return;
  double* y = sy + (size_t)warp * n;
  const double* a = L + (size_t)b * lstride;
  const double* rhs = B + (size_t)b * bstride;
  double* x = X + (size_t)b * xstride;
  for (int i = lane; i < n; i += 32) y[i] = rhs[i];
  __syncwarp();
  for (int k = 0; k < n; k++) {
    const double xk = y[k] / a[k + (size_t)k * n];
    __syncwarp();
    if (lane == 0) y[k] = xk;
    for (int i = k + 1 + lane; i < n; i += 32) y[i] -= a[i + (size_t)k * n] * xk;
    __syncwarp();
  }
  for (int i = n - 1; i >= 0; i--) {
    double part = 0.0;
    for (int k = i + 1 + lane; k < n; k += 32) part += a[k + (size_t)i * n] * y[k];
    part = warp_sum(part);
    const double xi = (y[i] - part) / a[i + (size_t)i * n];
    __syncwarp();
    if (lane == 0) y[i] = xi;
    __syncwarp();
  }
  for (int i = lane; i < n; i += 32) x[i] = y[i];
}

// V = L^{-1}, row-major into Vrm (V[m][k] at m*n + k); thread per column k of V.
__global__ void k_trtri(const double* __restrict__ L, int n, int64_t stride, double* __restrict__ Vrm) {
  const double* a = L + (size_t)blockIdx.x * stride;
  double* v = Vrm + (size_t)blockIdx.x * stride;
  for (int k = threadIdx.x; k < n; k += blockDim.x) {
    for (int i = 0; i < k; i++) v[(size_t)i * n + k] = 0.0;
    v[(size_t)k * n + k] = 1.0 / a[k + (size_t)k * n];
    for (int i = k + 1; i < n; i++) {
      double acc = 0.0;
      for (int m = k; m < i; m++) acc = fma(a[i + (size_t)m * n], v[(size_t)m * n + k], acc);
      v[(size_t)i * n + k] = -acc / a[i + (size_t)i * n];
    }
  }
}

// S = V^T V with V lower triangular (row-major); S full symmetric col-major.
__global__ void k_lauum(const double* __restrict__ Vrm, int n, int64_t stride, double* __restrict__ S) {
  const double* v = Vrm + (size_t)blockIdx.x * stride;
  double* s = S + (size_t)blockIdx.x * stride;
  for (int b = threadIdx.x; b < n; b += blockDim.x) {
    for (int a = 0; a <= b; a++) {
      double acc = 0.0;
      for (int i = b; i < n; i++) acc = fma(v[(size_t)i * n + a], v[(size_t)i * n + b], acc);
      s[a + (size_t)b * n] = acc;
      s[b + (size_t)a * n] = acc;
    }
  }
}

int launch_gram(Ctx* c, bool unweighted) {
  const int J = unweighted ? 1 : c->J;
  int rc;
  if (unweighted) {  // the Gram of the GLM initialisation, one for all genes
    ProfScope ps(c, "gram");
    rc = dgen_unweighted_gram(c);
  } else {
    rc = c->precision == GPL_PREC_BF16X3 ? launch_tc_gram(c) : launch_pair_gram(c);
  }
  if (rc != GPL_OK) return rc;
  rc = launch_group_sums(c, unweighted ? 1 : 0);
  if (rc) return rc;
  return launch_assemble_psi(c, J);
}

int launch_chol_batched(Ctx* c, double* A, int n, int batch, int64_t stride) {
  ProfScope ps(c, "chol");
  const int rc = launch_potrf_panels(c, A, n, batch, stride);
  if (rc != GPL_ERR_ARG) return rc;
  k_chol<<<batch, 256, 0, c->stream>>>(A, n, stride, 0);
  GPL_LAUNCHED(c, "k_chol");
  return GPL_OK;
}

int launch_chol_single(Ctx* c, double* A, int n) {
  ProfScope ps(c, "chol_small");
  if (n > 4 * kCholThreads) {  // wider than the exact kernel's per-thread row slots
    k_chol<<<1, 256, 0, c->stream>>>(A, n, 0, 1);
    GPL_LAUNCHED(c, "k_chol");
    return GPL_OK;
  }
  c->launches++;
  GPL_TRY(c, launch_chol_exact_raw(c->stream, A, n));
  return GPL_OK;
}

int launch_chol_prior(Ctx* c) {
  if (c->P > 4 * kCholThreads) return launch_chol_single(c, c->DeltaInv, c->P);
  ProfScope ps(c, "chol_small");
  c->launches++;
  GPL_TRY(c, launch_chol_exact_raw(c->stream, c->DeltaInv, c->P, c->nh[c->p - 1]));
  return GPL_OK;
}

cudaError_t launch_chol_exact_raw(cudaStream_t st, double* A, int n, int diag) {
  constexpr size_t most = 224 * 1024;
  int k0 = diag;  // the diagonal rows' columns are not read
  while ((size_t)(n - k0) * (n - k0 + 1) / 2 * sizeof(double) > most) k0++;
  const size_t smem = (size_t)(n - k0) * (n - k0 + 1) / 2 * sizeof(double);
  const cudaError_t e = cudaFuncSetAttribute((const void*)k_chol_exact, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)most);
  if (e != cudaSuccess) return e;
  void* args[] = {&A, &n, &diag, &k0};
  return cudaLaunchKernel((const void*)k_chol_exact, dim3(1), dim3(kCholThreads), args, smem, st);
}

int launch_solve_batched(Ctx* c, const double* L, int n, int64_t lstride, const double* B, int64_t bstride,
                         double* X, int64_t xstride, int batch) {
  ProfScope ps(c, "solve");
  const int warps = 4;
  const bool any = n > 576;
  const size_t shm = sizeof(double) * (size_t)n * warps * (any ? 1 : 2);
  auto* fn = n <= 64 ? k_solve<2> : n <= 128 ? k_solve<4> : n <= 288 ? k_solve<9> : any ? k_solve_any : k_solve<18>;
  if (shm > 48 * 1024) GPL_TRY(c, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shm));
  fn<<<div_up(batch, warps), 32 * warps, shm, c->stream>>>(L, n, lstride, B, bstride, X, xstride, batch);
  GPL_LAUNCHED(c, "k_solve");
  return GPL_OK;
}

int launch_inverse_batched(Ctx* c) {
  const int64_t st = (int64_t)c->P * c->P;
  ProfScope ps(c, "inverse");
  {
    const int rc = launch_inverse_panels(c);
    if (rc != GPL_ERR_ARG) return rc;  // GPL_ERR_ARG: P beyond the panel kernels' checked range
  }
  k_trtri<<<c->J, 256, 0, c->stream>>>(c->Psi, c->P, st, c->scratch);
  GPL_LAUNCHED(c, "k_trtri");
  k_lauum<<<c->J, 256, 0, c->stream>>>(c->scratch, c->P, st, c->PsiInv);
  GPL_LAUNCHED(c, "k_lauum");
  return GPL_OK;
}


}  // namespace gpl
