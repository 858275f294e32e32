// Cis genotype statistics per (gene, variant): the efficient score of adding one genotype column to
// a gene's fitted model, as getScoreStats of the reference's differential-expression driver computes
// it for genotype columns shared by all genes (ggplvm_de.cu:489-535), here for a separate set of
// variants per gene whose dosages are constant within a donor (genotypes are per donor; every cell
// carries its donor's). For gene j and a dosage column g (g_i = G[donor(i)]):
//     s = sum_i g_i (y_ij - W_ij) / Omega_i
//     v = g^T diag(W_j / Omega) g - t^T Psi_j^{-1} t,   t = Z^T diag(W_j / Omega) g
//     S = s / sqrt(phi_j v),   LR = S^2
// LR is the likelihood ratio of the IRLS working model (Gaussian in nu with weights W/Omega and
// dispersion phi) for adding the column with every other coefficient re-estimated: the
// per-(gene, variant) likelihood-ratio statistic against the fitted GP.
//
// Because g is constant within a donor, every sum over cells reduces to sums over the cell groups
// (the combinations of categorical levels, which include the donor):
//     s     = sum_g G[donor(g)] R_jg,          R_jg = sum_{i in g} (y_ij - W_ij) / Omega_i
//     t_a   = sum_g G[donor(g)] S_j[g][a]       (dense column a; S = the Gram's group sums)
//     t_c   = sum_{g at level c} G[donor(g)] S_j[g][intercept]   (categorical column c)
//     g^T diag(w) g = sum_g G[donor(g)]^2 S_j[g][intercept]
// and t^T Psi_j^{-1} t = |L_j^{-1} t|^2 with the factor L_j of Psi_j. The counts enter through W
// and nu of the last W/nu pass (y = W (nu - eta + 1) for the matched counts and 0 = W (nu - eta + 1)
// for the others, with eta = log W - log s - wt delta_GP titsias).
//
//   k_group_resid  R_jg, one warp per (gene, group), the group's cells in order
//   k_cis_t        per gene: t, s and g^T diag(w) g for 16 of its variants at a time
//   k_fwd_quad     |L^{-1} t|^2 of all variants by one forward substitution (k_score.cu)
#include <math.h>

#include <algorithm>
#include <vector>

#include "gpl_internal.cuh"

namespace gpl {

namespace {

__global__ void k_group_resid(int N, int ldN, int J, int n_grp, int pvars, const int* __restrict__ gcells,
                              const int* __restrict__ gstart, const double* __restrict__ W,
                              const double* __restrict__ Nu, const double* __restrict__ Omega,
                              const double* __restrict__ ls, const double* __restrict__ delta,
                              const double* __restrict__ titsias, double* __restrict__ R) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  const int j = warp / n_grp, g = warp - j * n_grp;
  if (j >= J) return;
  const double dgp = delta[pvars - 1];
  const double* Wj = W + (size_t)j * ldN;
  const double* nj = Nu + (size_t)j * ldN;
  double s = 0.0;
  for (int k = gstart[g] + lane; k < gstart[g + 1]; k += 32) {
    const int i = gcells[k];
    const double w = Wj[i];
    const double eta = log(w) - log(ls[i]) - dgp * titsias[i] * kWt;
    s += w * (nj[i] - eta) / Omega[i];  // (y - W) / Omega with y = W (nu - eta + 1)
  }
  s = warp_sum(s);
  if (lane == 0) R[(size_t)j * n_grp + g] = s;
}

// One gene's t vectors, scores and dosage sums for kCisV of its variants: a thread per dense column takes
// every group's sum once for all of them (the dosages of kCisGroups groups at a time in shared memory;
// two halves of them per block, added in order, where the threads allow), a thread per level and variant
// its level's groups, a warp per variant the sums over all groups. T[(j - j0) V + v][P];
// num[j + v J] = s, gw[j + v J] = g^T diag(w) g. A block per gene that walked the groups once per variant
// and column, and the levels in one thread, took 10.7 ms for 1,000 genes x 20 variants with the
// substitution (400 groups, P = 236); this kernel and k_fwd_quad take 0.54 + 0.5 ms.
constexpr int kCisV = 16, kCisGroups = 128;
__global__ void __launch_bounds__(1024) k_cis_t(int j0, int J, int P, int n_d, int n_dp, int n_grp, int n_lvl, int V,
                                                const int* __restrict__ dcol, const int* __restrict__ lvl_cc,
                                                const int* __restrict__ lvl_ptr, const int* __restrict__ lvl_grp,
                                                const int* __restrict__ gdonor, const int8_t* __restrict__ dos,
                                                const double* __restrict__ gsum, const double* __restrict__ R,
                                                double* __restrict__ T, double* __restrict__ num,
                                                double* __restrict__ gw) {
  extern __shared__ __align__(16) double sm[];
  double* Gg = sm;                             // [kCisGroups][kCisV]
  double* half = Gg + kCisGroups * kCisV;      // [n_dp][kCisV] the second half's sums
  const int j = j0 + blockIdx.x, v0 = blockIdx.y * kCisV, nv = min(kCisV, V - v0), tid = threadIdx.x;
  const int ld = n_d + 1;
  const double* Sj = gsum + (size_t)j * n_grp * ld;
  const double* Rj = R + (size_t)j * n_grp;
  double* Tj = T + ((size_t)blockIdx.x * V + v0) * P;
  auto dosage = [&](int g, int v) { return (double)dos[((size_t)gdonor[g] * J + j) * V + v0 + v]; };
  const int parts = blockDim.x / n_dp, part = tid / n_dp, a0 = tid - part * n_dp;  // one or two
  for (int ab = 0; ab < n_d; ab += n_dp) {
    const int a = ab + a0;
    double acc[kCisV];
#pragma unroll
    for (int v = 0; v < kCisV; v++) acc[v] = 0.0;
    for (int b0 = 0; b0 < n_grp; b0 += kCisGroups) {
      const int nb = min(kCisGroups, n_grp - b0);
      __syncthreads();
      for (int e = tid; e < nb * kCisV; e += blockDim.x) {
        const int g = e / kCisV, v = e - g * kCisV;
        Gg[e] = v < nv ? dosage(b0 + g, v) : 0.0;
      }
      __syncthreads();
      if (a < n_d) {
        const int per = (nb + parts - 1) / parts, g1 = min(nb, (part + 1) * per);
#pragma unroll 2
        for (int g = part * per; g < g1; g++) {
          const double s = Sj[(size_t)(b0 + g) * ld + a];
          const double2* x = reinterpret_cast<const double2*>(Gg + (size_t)g * kCisV);
#pragma unroll
          for (int v = 0; v < kCisV / 2; v++) {
            const double2 w = x[v];
            acc[2 * v] = fma(w.x, s, acc[2 * v]);
            acc[2 * v + 1] = fma(w.y, s, acc[2 * v + 1]);
          }
        }
      }
    }
    if (part == 1)
#pragma unroll
      for (int v = 0; v < kCisV; v++) half[(size_t)a0 * kCisV + v] = acc[v];
    __syncthreads();
    if (a < n_d && part == 0) {
#pragma unroll
      for (int v = 0; v < kCisV; v++)
        if (v < nv) Tj[(size_t)v * P + dcol[a]] = acc[v] + (parts > 1 ? half[(size_t)a0 * kCisV + v] : 0.0);
    }
  }
  for (int e = tid; e < n_lvl * nv; e += blockDim.x) {
    const int c = e / nv, v = e - c * nv;
    double s = 0.0;
    for (int q = lvl_ptr[c]; q < lvl_ptr[c + 1]; q++) {
      const int g = lvl_grp[q];
      s += dosage(g, v) * Sj[(size_t)g * ld];
    }
    Tj[(size_t)v * P + lvl_cc[c]] = s;
  }
  const int warp = tid >> 5, lane = tid & 31;
  for (int v = warp; v < nv; v += blockDim.x >> 5) {
    double sp = 0.0, w = 0.0;
    for (int g = lane; g < n_grp; g += 32) {
      const double x = dosage(g, v);
      sp = fma(x, Rj[g], sp);
      w = fma(x * x, Sj[(size_t)g * ld], w);
    }
    sp = warp_sum(sp);
    w = warp_sum(w);
    if (lane == 0) {
      num[j + (size_t)(v0 + v) * J] = sp;
      gw[j + (size_t)(v0 + v) * J] = w;
    }
  }
}

// S = num / sqrt(phi (gw - q)), LR = S^2; q[(j - j0) + v nj] = t^T Psi_j^{-1} t
__global__ void k_cis_final(int j0, int nj, int J, const double* __restrict__ q, const double* __restrict__ phi,
                            double* __restrict__ S, double* __restrict__ LR) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x, v = blockIdx.y;
  if (r >= nj) return;
  const size_t e = j0 + r + (size_t)v * J;
  const double st = S[e] / sqrt(phi[j0 + r] * (LR[e] - q[r + (size_t)v * nj]));
  S[e] = st;
  LR[e] = st * st;
}

}  // namespace

int cis_stats(Ctx* c, int donor_var, int n_donors, int V, const int8_t* dos_host, double* S_host, double* LR_host) {
  if (c->n_grp == 0 || c->n_cv == 0) {
    c->err = "cis statistics need the categorical variables handled by cell groups";
    return GPL_ERR_ARG;
  }
  if (donor_var < 0 || donor_var >= c->n_var || c->vc[donor_var + 1] == 1) {
    c->err = "donor_var must name a categorical design variable";
    return GPL_ERR_ARG;
  }
  const int col = c->nh[donor_var + 1];
  int vd = -1;
  for (int v = 0; v < c->n_cv; v++)
    if (c->cv_nh[v] == col) vd = v;
  if (vd < 0 || n_donors != c->cv_nlev[vd]) {
    c->err = "n_donors must equal the donor variable's level count";
    return GPL_ERR_ARG;
  }
  const int J = c->J, n_grp = c->n_grp, n_cv = c->n_cv, P = c->P;
  const size_t smem = sizeof(double) * ((size_t)n_grp + (size_t)P * V);
  if (smem > 200 * 1024 || V < 1 || V > 256) {
    c->err = "too many variants or cell groups for the per-gene statistics";
    return GPL_ERR_ARG;
  }
  std::vector<int> glev((size_t)n_grp * n_cv), gdon(n_grp);
  GPL_TRY(c, cudaMemcpy(glev.data(), c->glev_d, sizeof(int) * glev.size(), cudaMemcpyDeviceToHost));
  for (int g = 0; g < n_grp; g++) gdon[g] = glev[(size_t)g * n_cv + vd];
  // work: R (J x n_grp), S and LR (J x V), the t vectors and quadratic forms of a range of genes (at most
  // 256 MiB), the groups' donors, the dosages
  const size_t nd = (size_t)n_donors * J * V;
  const int nj = (int)std::max<int64_t>(1, std::min<int64_t>(J, ((int64_t)32 << 20) / ((int64_t)V * P)));
  const size_t n_t = (size_t)nj * V * P;
  int rc = ensure_work(c, (size_t)J * n_grp + 2 * (size_t)J * V + n_t + (size_t)nj * V + (n_grp + 1) / 2 + nd / 8 + 1);
  if (rc) return rc;
  double *R = c->work, *Sd = R + (size_t)J * n_grp, *LRd = Sd + (size_t)J * V, *T = LRd + (size_t)J * V, *q = T + n_t;
  int* gdon_d = reinterpret_cast<int*>(q + (size_t)nj * V);
  int8_t* dos_d = reinterpret_cast<int8_t*>(q + (size_t)nj * V + (n_grp + 1) / 2);
  GPL_TRY(c, cudaMemcpyAsync(gdon_d, gdon.data(), sizeof(int) * n_grp, cudaMemcpyHostToDevice, c->stream));
  GPL_TRY(c, cudaMemcpyAsync(dos_d, dos_host, nd, cudaMemcpyHostToDevice, c->stream));
  if ((rc = launch_group_sums(c, 0))) return rc;  // S_j[g][a] with w = W/Omega at the current state
  const int64_t warps = (int64_t)J * n_grp;
  k_group_resid<<<div_up(warps * 32, 256), 256, 0, c->stream>>>(c->N, c->ldN, J, n_grp, c->p, c->gcells_d,
                                                                 c->gstart_d, c->W, c->Nu, c->Omega, c->ls, c->delta,
                                                                 c->titsias, R);
  GPL_LAUNCHED(c, "k_group_resid");
  const int n_dp = std::min(512, (c->n_d + 31) / 32 * 32);
  const size_t smem_t = sizeof(double) * (size_t)(kCisGroups + n_dp) * kCisV;
  GPL_TRY(c, cudaFuncSetAttribute(k_cis_t, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_t));
  for (int j0 = 0; j0 < J; j0 += nj) {
    const int n = std::min(nj, J - j0);
    k_cis_t<<<dim3(n, div_up(V, kCisV)), 2 * n_dp, smem_t, c->stream>>>(
        j0, J, P, c->n_d, n_dp, n_grp, c->n_lvl, V, c->dcol_d, c->lvl_cc_d, c->lvl_ptr_d, c->lvl_grp_d, gdon_d, dos_d,
        c->gsum, R, T, Sd, LRd);
    GPL_LAUNCHED(c, "k_cis_t");
    if ((rc = launch_quad(c, n, V, c->Psi + (size_t)j0 * P * P, T, (size_t)V * P, P, q))) return rc;
    k_cis_final<<<dim3(div_up(n, 256), V), 256, 0, c->stream>>>(j0, n, J, q, c->phi, Sd, LRd);
    GPL_LAUNCHED(c, "k_cis_final");
  }
  GPL_TRY(c, cudaMemcpyAsync(S_host, Sd, sizeof(double) * (size_t)J * V, cudaMemcpyDeviceToHost, c->stream));
  if (LR_host)
    GPL_TRY(c, cudaMemcpyAsync(LR_host, LRd, sizeof(double) * (size_t)J * V, cudaMemcpyDeviceToHost, c->stream));
  GPL_TRY(c, cudaStreamSynchronize(c->stream));
  return GPL_OK;
}

}  // namespace gpl
