// Genotype score statistics against the fitted model (getScoreStats, ggplvm_de.cu:489-535;
// launched after the fit over a J x L grid, :1205-1209). For gene j and genotype column g_l:
//   t = Z^T diag(W_j/Omega) g_l,  v = sum_i g_il^2 W_ij / Omega_i - t^T Psi_j^{-1} t,
//   s = sum_i g_il / Omega_i (y_ij - W_ij)  (matched counts; -g W / Omega elsewhere),
//   S[j, l] = s / sqrt(phi_j v).
// Here the dense rows of t are the Z^T u GEMM with a per-cell u, its categorical rows come from the
// group sums of every column at once (the columns in the place of the dense ones), t^T Psi_j^{-1} t is
// |L_j^{-1} t|^2 by one forward substitution of all columns (k_fwd_quad), the two sums over all cells one
// split-K DMMA GEMM of W against [g^2/Omega | g/Omega], and the count sum a walk over each gene's
// matched prefix with a lane per column.
#include <algorithm>

#include "gpl_internal.cuh"

namespace gpl {

// G2[c][i] = g_il^2 / Omega_i (c = l < L) and g_il / Omega_i (c = L + l); Gt[i][l] = g_il / Omega_i
__global__ void k_score_cols(int N, int L, const double* __restrict__ G, const double* __restrict__ Omega,
                             double* __restrict__ G2, double* __restrict__ Gt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, l = blockIdx.y;
  if (i >= N) return;
  const double g = G[(size_t)l * N + i];
  G2[(size_t)l * N + i] = g * g / Omega[i];
  G2[(size_t)(L + l) * N + i] = g / Omega[i];
  Gt[(size_t)i * L + l] = g / Omega[i];
}

// dst[l * ldN + pos] = G[l * N + cell(pos)]: the columns in group order
__global__ void k_score_order(int N, int ldN, int L, const int* __restrict__ gcells, const double* __restrict__ G,
                              double* __restrict__ dst) {
  const int pos = blockIdx.x * blockDim.x + threadIdx.x, l = blockIdx.y;
  if (pos < N) dst[(size_t)l * ldN + pos] = G[(size_t)l * N + gcells[pos]];
}

// The categorical rows of every t: T[l][j][cc] = sum over the groups at the level of Sg[j][g][l]
__global__ void __launch_bounds__(256) k_score_levels(int J, int P, int L, int n_lvl, int n_grp,
                                                      const int* __restrict__ lvl_cc, const int* __restrict__ lvl_ptr,
                                                      const int* __restrict__ lvl_grp, const double* __restrict__ Sg,
                                                      double* __restrict__ T) {
  const int j = blockIdx.x;
  const double* s = Sg + (size_t)j * n_grp * (L + 1);
  for (int e = threadIdx.x; e < n_lvl * L; e += blockDim.x) {
    const int c = e / L, l = e - c * L;
    double v = 0.0;
    for (int q = lvl_ptr[c]; q < lvl_ptr[c + 1]; q++) v += s[(size_t)lvl_grp[q] * (L + 1) + l];
    T[((size_t)l * J + j) * P + lvl_cc[c]] = v;
  }
}

// q[j + v*J] = |L_j^{-1} t_jv|^2 for the right-hand sides t_jv at T + j sj + v sv: a block per gene and
// kQuadV right-hand sides, which stay in shared memory; 16 columns of the factor at a time (their
// diagonal block by a thread per right-hand side, the rows below by a thread per row and eight right-
// hand sides), so that the factor is read once for all of them and the chain has P / 16 steps. 20
// columns of 1,000 genes at P = 236 took 13 ms as one solve per column, 0.5 ms so.
constexpr int kQuadV = 16, kQuadRows = 128, kQuadS = kQuadV + 2;
__global__ void __launch_bounds__(256) k_fwd_quad(int J, int P, int V, const double* __restrict__ Psi,
                                                  const double* __restrict__ T, size_t sj, size_t sv,
                                                  double* __restrict__ q) {
  extern __shared__ __align__(16) double ys[];  // [P][kQuadS]
  __shared__ double lp[16][kQuadRows + 4];
  __shared__ double ld[16][17];
  const int j = blockIdx.x, v0 = blockIdx.y * kQuadV, nv = min(kQuadV, V - v0), tid = threadIdx.x;
  const double* L = Psi + (size_t)j * P * P;
  for (int e = tid; e < P * kQuadV; e += 256) {
    const int v = e / P, r = e - v * P;
    ys[r * kQuadS + v] = v < nv ? T[j * sj + (v0 + v) * sv + r] : 0.0;
  }
  for (int k0 = 0; k0 < P; k0 += 16) {
    const int kn = min(16, P - k0);
    {
      const int r = tid & 15, k = tid >> 4;
      ld[k][r] = r < kn && k <= r ? L[(size_t)(k0 + r) + (size_t)(k0 + k) * P] : 0.0;
    }
    __syncthreads();
    if (tid < kQuadV) {
      double y[16];
#pragma unroll
      for (int k = 0; k < 16; k++) y[k] = k < kn ? ys[(k0 + k) * kQuadS + tid] : 0.0;
#pragma unroll
      for (int k = 0; k < 16; k++) {
        if (k < kn) {
          y[k] = y[k] / ld[k][k];
#pragma unroll
          for (int r = k + 1; r < 16; r++) y[r] = fma(-ld[k][r], y[k], y[r]);
          ys[(k0 + k) * kQuadS + tid] = y[k];
        }
      }
    }
    for (int r0 = k0 + 16; r0 < P; r0 += kQuadRows) {
      __syncthreads();  // the diagonal rows are solved, lp is free
      for (int e = tid; e < 16 * kQuadRows; e += 256) {
        const int k = e / kQuadRows, r = e - k * kQuadRows;
        lp[k][r] = r0 + r < P ? L[(size_t)(r0 + r) + (size_t)(k0 + k) * P] : 0.0;
      }
      __syncthreads();
      const int r = tid & (kQuadRows - 1), h = (tid >> 7) * 8;
      if (r0 + r < P) {
        double* y = ys + (size_t)(r0 + r) * kQuadS + h;
        double a[8];
#pragma unroll
        for (int v = 0; v < 8; v++) a[v] = y[v];
#pragma unroll
        for (int k = 0; k < 16; k++) {
          const double l = lp[k][r];
          const double2* x = reinterpret_cast<const double2*>(ys + (size_t)(k0 + k) * kQuadS + h);
#pragma unroll
          for (int v = 0; v < 4; v++) {
            const double2 w = x[v];
            a[2 * v] = fma(-l, w.x, a[2 * v]);
            a[2 * v + 1] = fma(-l, w.y, a[2 * v + 1]);
          }
        }
#pragma unroll
        for (int v = 0; v < 8; v++) y[v] = a[v];
      }
    }
    __syncthreads();
  }
  // two right-hand sides per warp
  const int warp = tid >> 5, lane = tid & 31;
  for (int v = warp; v < nv; v += 8) {
    double s = 0.0;
    for (int r = lane; r < P; r += 32) s = fma(ys[r * kQuadS + v], ys[r * kQuadS + v], s);
    s = warp_sum(s);
    if (lane == 0) q[j + (size_t)(v0 + v) * J] = s;
  }
}

// q[j] = t_j . x_j, one warp per gene
__global__ void k_quad_dot(int J, int P, const double* __restrict__ t, size_t sj, const double* __restrict__ x,
                           double* __restrict__ q) {
  const int j = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (j >= J) return;
  double s = 0.0;
  for (int k = lane; k < P; k += 32) s += t[j * sj + k] * x[(size_t)j * P + k];
  s = warp_sum(s);
  if (lane == 0) q[j] = s;
}

// t^T Psi_j^{-1} t of every right-hand side; beyond k_fwd_quad's shared memory by a solve and a product each
int launch_quad(Ctx* c, int J, int V, const double* Psi, const double* T, size_t sj, size_t sv, double* q) {
  const size_t smem = sizeof(double) * (size_t)c->P * kQuadS;
  if (smem > 200 * 1024) {
    for (int v = 0; v < V; v++) {
      const int rc = launch_solve_batched(c, Psi, c->P, (int64_t)c->P * c->P, T + v * sv, (int64_t)sj, c->rres, c->P, J);
      if (rc) return rc;
      k_quad_dot<<<div_up(J, 8), 256, 0, c->stream>>>(J, c->P, T + v * sv, sj, c->rres, q + (size_t)v * J);
      GPL_LAUNCHED(c, "k_quad_dot");
    }
    return GPL_OK;
  }
  GPL_TRY(c, cudaFuncSetAttribute(k_fwd_quad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  k_fwd_quad<<<dim3(J, div_up(V, kQuadV)), 256, smem, c->stream>>>(J, c->P, V, Psi, T, sj, sv, q);
  GPL_LAUNCHED(c, "k_fwd_quad");
  return GPL_OK;
}

// sp[j + l*J] = sum over gene j's matched counts of g_il y / Omega_i, one CTA per gene: a lane per column
// (two beyond 32), so that a count's row of Gt is read once, contiguous.
__global__ void __launch_bounds__(256) k_score_counts(int J, int L, const int32_t* __restrict__ cell,
                                                      const int64_t* __restrict__ gptr,
                                                      const int32_t* __restrict__ gvalid,
                                                      const double* __restrict__ cnt, const double* __restrict__ Gt,
                                                      double* __restrict__ sp) {
  __shared__ double sh[8][64];
  const int j = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t b = gptr[j], e = gptr[j] + gvalid[j];
  const bool on0 = lane < L, on1 = lane + 32 < L;
  double s0 = 0.0, s1 = 0.0;
#pragma unroll 4
  for (int64_t q = b + warp; q < e; q += 8) {
    const double y = cnt[q];
    const double* g = Gt + (size_t)cell[q] * L + lane;
    if (on0) s0 = fma(g[0], y, s0);
    if (on1) s1 = fma(g[32], y, s1);
  }
  sh[warp][lane] = s0;
  sh[warp][lane + 32] = s1;
  __syncthreads();
  for (int l = threadIdx.x; l < L; l += 256) {
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < 8; k++) s += sh[k][l];
    sp[j + (size_t)l * J] = s;
  }
}

// S = (sp - sum W g/Omega) / sqrt(phi (sum W g^2/Omega - td))
__global__ void k_score_final(int J, int L, const double* __restrict__ sp, const double* __restrict__ C,
                              const double* __restrict__ td, const double* __restrict__ phi,
                              double* __restrict__ S) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x, l = blockIdx.y;
  if (j >= J) return;
  const size_t e = j + (size_t)l * J;
  const double v = C[e] - td[e];
  S[e] = (sp[e] - C[j + (size_t)(L + l) * J]) / sqrt(phi[j] * v);
}

// Columns per pass: the GEMM tile takes two per column, the group sums' buffer the dense columns' count,
// and the vectors t of a pass stay within 256 MiB.
int score_columns(const Ctx* c, int L) {
  const int64_t per = (int64_t)c->J * c->P * (int64_t)sizeof(double);
  return (int)std::max<int64_t>(1, std::min<int64_t>({L, 64, c->n_grp ? c->n_d : 64, ((int64_t)256 << 20) / per}));
}

// values of scratch that a pass of L columns takes
size_t score_work(const Ctx* c, int L) {
  return (size_t)L * ((size_t)3 * c->N + c->ldN + (size_t)4 * c->J + (size_t)c->J * c->P) + 1;
}

// crt: scratch goes on with crt_columns_work values for the integer form
int launch_score_stats(Ctx* c, int L, const double* G, double* S, double* scratch, bool crt) {
  const size_t N = c->N, J = c->J, P = c->P;
  // scratch: G2 (2L x N), Gt (N x L), C (J x 2L), td (J x L), sp (J x L), G in group order, t (L x J x P)
  double* G2 = scratch;
  double* Gt = G2 + 2 * L * N;
  double* C = Gt + L * N;
  double* td = C + 2 * L * J;
  double* sp = td + L * J;
  double* Gg = sp + L * J;
  double* T = Gg + (size_t)L * c->ldN;
  T += (T - scratch) & 1;
  int rc;
  k_score_cols<<<dim3(div_up(c->N, 256), L), 256, 0, c->stream>>>(c->N, L, G, c->Omega, G2, Gt);
  GPL_LAUNCHED(c, "k_score_cols");
  if ((rc = dgen_weighted_colsums(c, G2, 2 * L, C))) return rc;
  int left = 2;
  if (crt && (rc = launch_crt_columns(c, L, G, C, T, scratch + score_work(c, L), &left))) return rc;
  for (int l = 0; l < L && left; l++)
    if ((rc = dgen_zt_u(c, 2, G + (size_t)l * N, T + (size_t)l * J * P, left == 1 ? c->pr.crt.cols + 1 : nullptr))) {
      if (rc == GPL_ERR_ARG) c->err = "per-cell Z^T u takes at most 144 dense columns";
      return rc;
    }
  if (c->n_grp) {
    k_score_order<<<dim3(div_up(N, 256), L), 256, 0, c->stream>>>(c->N, c->ldN, L, c->gcells_d, G, Gg);
    GPL_LAUNCHED(c, "k_score_order");
    if ((rc = dgen_group_sums_of(c, Gg, L))) return rc;
    k_score_levels<<<c->J, 256, 0, c->stream>>>(c->J, c->P, L, c->n_lvl, c->n_grp, c->lvl_cc_d, c->lvl_ptr_d,
                                                c->lvl_grp_d, c->gsum, T);
    GPL_LAUNCHED(c, "k_score_levels");
  }
  if ((rc = launch_quad(c, c->J, L, c->Psi, T, P, J * P, td))) return rc;
  k_score_counts<<<c->J, 256, 0, c->stream>>>(c->J, L, c->cell, c->gptr, c->gvalid, c->cnt, Gt, sp);
  GPL_LAUNCHED(c, "k_score_counts");
  k_score_final<<<dim3(div_up(c->J, 256), L), 256, 0, c->stream>>>(c->J, L, sp, C, td, c->phi, S);
  GPL_LAUNCHED(c, "k_score_final");
  return GPL_OK;
}

}  // namespace gpl
