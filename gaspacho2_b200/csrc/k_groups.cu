// Categorical covariates through cell groups.
//
// A categorical variable contributes one-hot columns to the model matrix (getModelMatrix,
// DataFrame.cu:72-82), and the reference's Gram treats them case by case
// (ggplvm.cu:628-674): level x numeric sums, level x level co-occurrence sums. Here every
// cell belongs to the group of its combination of levels (400 groups for batch x donor at
// config 2), and everything categorical reduces to per-(gene, group) sums over the cells of
// a group:
//
//   S[j][g][a] = sum_{i in g} w_ij D[i, a]       (dense column a; a = intercept gives sum w)
//   T[j][g]    = sum_{i in g} w_ij u_ij          (u = nu for Z^T diag(w) nu, y0 for initBeta)
//
// from which the categorical rows of Psi_j and of Z^T diag(w) nu are assembled exactly as the
// reference's case analysis defines them. In the gradient the same layout holds the
// categorical blocks of Psi_j^{-1} seen by each group:
//
//   h[j][g][a] = sum_{c in cats(g)} S_j[dcol[a], c],  kappa[j][g] = sum_{c,c' in cats(g)} S_j[c, c']
//
// so that z_i^T S_j z_i = d_i^T S_DD d_i + 2 d_i . h + kappa for a cell of group g.
// The group sums and HK are FP64 GEMMs over the cells of one group (k_dgen.cu), N*J*n_d
// multiply-adds each.
#include <algorithm>

#include "gpl_internal.cuh"

namespace gpl {

// T[j][g] = sum_{i in g} w_ij u_ij, one warp per (gene, group); mode 0: w = W/Omega, u = nu (W and
// 1/Omega read in group order); mode 2: w = 1, u = y0 (scratch).
template <int MODE>
__global__ void k_group_t(int ldN, int J, int n_grp, const int* __restrict__ gcells, const int* __restrict__ gstart,
                          const double* __restrict__ Wg, const double* __restrict__ rOmg,
                          const double* __restrict__ U, double* __restrict__ T) {
  const int g = blockIdx.x;
  const int j = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (j >= J) return;
  const int c0 = gstart[g], c1 = gstart[g + 1];
  const double *Wj = Wg + (size_t)j * ldN, *Uj = U + (size_t)j * ldN;
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  for (int k0 = c0 + lane; k0 < c1; k0 += 128) {
    double v[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int k = k0 + 32 * u;
      v[u] = k < c1 ? (MODE == 2 ? Uj[gcells[k]] : Wj[k] * rOmg[k] * Uj[gcells[k]]) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 4; u++) s[u] += v[u];
  }
  const double t = warp_sum((s[0] + s[1]) + (s[2] + s[3]));
  if (lane == 0) T[(size_t)j * n_grp + g] = t;
}

// The same sums within an OrderScope (gpl_internal.cuh): a lane's cells in one chain, W / Omega by division.
template <int MODE>
__global__ void k_group_t_chain(int ldN, int J, int n_grp, const int* __restrict__ gcells,
                                const int* __restrict__ gstart, const double* __restrict__ Wg,
                                const double* __restrict__ Omega, const double* __restrict__ U,
                                double* __restrict__ T) {
  const int g = blockIdx.x;
  const int j = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (j >= J) return;
  const double *Wj = Wg + (size_t)j * ldN, *Uj = U + (size_t)j * ldN;
  double s = 0.0;
#pragma unroll 4
  for (int k = gstart[g] + lane; k < gstart[g + 1]; k += 32) {
    const int i = gcells[k];
    if (MODE == 2) s += Uj[i];
    else s += Wj[k] / Omega[i] * Uj[i];
  }
  s = warp_sum(s);
  if (lane == 0) T[(size_t)j * n_grp + g] = s;
}

// mode 0: S with w = W/Omega (Gram of the objective and the IRLS); 1: S of gene 0 with w = 1
// (GLM initialisation Gram); 2: T with w = 1, u = y0 (GLM initialisation right-hand side);
// 3: T with w = W/Omega, u = nu (Z^T diag(W/Omega) nu).
int launch_group_sums(Ctx* c, int mode) {
  if (c->n_grp == 0) return GPL_OK;
  if (mode == 0 || mode == 1) {
    ProfScope ps(c, "group_sums");
    return dgen_group_sums(c, mode);
  }
  ProfScope pt(c, "group_t");
  dim3 g(c->n_grp, div_up(c->J, 8));
  if (c->one_order) {
    auto fn = mode == 2 ? k_group_t_chain<2> : k_group_t_chain<0>;
    fn<<<g, 256, 0, c->stream>>>(c->ldN, c->J, c->n_grp, c->gcells_d, c->gstart_d, c->Wg, c->Omega,
                                 mode == 2 ? c->scratch : c->zt_u_src ? c->zt_u_src : c->Nu, c->gT);
    GPL_LAUNCHED(c, "k_group_t_chain");
    return GPL_OK;
  }
  if (mode != 2) {
    const int rc = recip_omega_grouped(c);
    if (rc) return rc;
  }
  if (mode == 2)
    k_group_t<2><<<g, 256, 0, c->stream>>>(c->ldN, c->J, c->n_grp, c->gcells_d, c->gstart_d, c->Wg, c->rOmg,
                                           c->scratch, c->gT);
  else
    k_group_t<0><<<g, 256, 0, c->stream>>>(c->ldN, c->J, c->n_grp, c->gcells_d, c->gstart_d, c->Wg, c->rOmg,
                                           c->zt_u_src ? c->zt_u_src : c->Nu, c->gT);
  GPL_LAUNCHED(c, "k_group_t");
  return GPL_OK;
}

// Categorical rows and columns of Psi_j (both triangles) from the group sums, plus the
// prior's diagonal on them; the dense x dense entries are written by the Gram kernel. Every
// categorical entry is written once, as a sum over the groups at its level(s) taken in group
// order (the order of getPsi's case analysis, ggplvm.cu:628-674, over the cells of each group):
//   (level l, dense column a)   sum_{g at l} S[g][a]
//   (level l, level l)          sum_{g at l} S[g][0] + DeltaInv (S[.][0]: the intercept = sum w)
//   (level l, other level of the same variable)   0
//   (level l of v, level l2 of v2 != v)           sum_{g at l and l2} S[g][0]
__global__ void __launch_bounds__(256) k_assemble_psi(int P, int n_d, int NL, int n_cv, int n_grp,
                                                      const int* __restrict__ dcol, const int* __restrict__ lvl_cc,
                                                      const int* __restrict__ lvl_v, const int* __restrict__ lvl_ptr,
                                                      const int* __restrict__ lvl_grp, const int* __restrict__ cv_nh,
                                                      const int* __restrict__ glev, const double* __restrict__ S,
                                                      const double* __restrict__ Dinv, double* __restrict__ Psi) {
  const int j = blockIdx.x;
  double* Pj = Psi + (size_t)j * P * P;
  const double* Sj = S + (size_t)j * n_grp * (n_d + 1);
  const int ld = n_d + 1;
  for (int e = threadIdx.x; e < NL * n_d; e += blockDim.x) {
    const int l = e / n_d, a = e - l * n_d;
    double s = 0.0;
    int q = lvl_ptr[l];
    const int q1 = lvl_ptr[l + 1];
    for (; q + 4 <= q1; q += 4) {  // four loads in flight, added in order
      double v[4];
#pragma unroll
      for (int u = 0; u < 4; u++) v[u] = Sj[(size_t)lvl_grp[q + u] * ld + a];
#pragma unroll
      for (int u = 0; u < 4; u++) s += v[u];
    }
    for (; q < q1; q++) s += Sj[(size_t)lvl_grp[q] * ld + a];
    const size_t cc = lvl_cc[l], dc = dcol[a];
    Pj[cc + dc * P] = s;
    Pj[dc + cc * P] = s;
  }
  for (int e = threadIdx.x; e < NL * NL; e += blockDim.x) {
    const int l1 = e / NL, l2 = e - l1 * NL;
    const int v1 = lvl_v[l1], v2 = lvl_v[l2];
    const size_t c1 = lvl_cc[l1], c2 = lvl_cc[l2];
    double s = 0.0;
    if (v1 == v2) {
      if (l1 == l2) {
        for (int q = lvl_ptr[l1]; q < lvl_ptr[l1 + 1]; q++) s += Sj[(size_t)lvl_grp[q] * ld];
        s += Dinv[c1 + c1 * P];
      }
    } else {
      const int L2 = (int)c2 - cv_nh[v2];
      for (int q = lvl_ptr[l1]; q < lvl_ptr[l1 + 1]; q++) {
        const int g = lvl_grp[q];
        if (glev[(size_t)g * n_cv + v2] == L2) s += Sj[(size_t)g * ld];
      }
    }
    Pj[c1 + c2 * P] = s;
  }
}

// dst[col * ldN + pos] = src[col * ldN + cell(pos)]: the cells in group order (gcells)
__global__ void k_group_order(int N, int ldN, int ncols, const int* __restrict__ gcells, const double* __restrict__ src,
                              double* __restrict__ dst) {
  const int pos = blockIdx.x * blockDim.x + threadIdx.x;
  if (pos >= N) return;
  const int i = gcells[pos];
  for (int col = blockIdx.y; col < ncols; col += gridDim.y) dst[(size_t)col * ldN + pos] = src[(size_t)col * ldN + i];
}

int launch_group_order(Ctx* c, const double* src, int ncols, double* dst) {
  dim3 g(div_up(c->N, 256), std::min(ncols, 65535));
  k_group_order<<<g, 256, 0, c->stream>>>(c->N, c->ldN, ncols, c->gcells_d, src, dst);
  GPL_LAUNCHED(c, "k_group_order");
  return GPL_OK;
}

int launch_assemble_psi(Ctx* c, int J) {
  if (c->n_grp == 0) return GPL_OK;
  ProfScope ps(c, "assemble_psi");
  k_assemble_psi<<<J, 256, 0, c->stream>>>(c->P, c->n_d, c->n_lvl, c->n_cv, c->n_grp, c->dcol_d, c->lvl_cc_d,
                                           c->lvl_v_d, c->lvl_ptr_d, c->lvl_grp_d, c->cv_nh_d, c->glev_d, c->gsum,
                                           c->DeltaInv, c->Psi);
  GPL_LAUNCHED(c, "k_assemble_psi");
  return GPL_OK;
}

// Categorical entries of bvec (P x J): sum over the groups at each level of T[j][g], in group order;
// a block per gene with its row of T in shared memory, a thread per level.
__global__ void __launch_bounds__(128) k_assemble_b(int P, int n_lvl, int n_grp, const int* __restrict__ lvl_cc,
                                                    const int* __restrict__ lvl_ptr, const int* __restrict__ lvl_grp,
                                                    const double* __restrict__ T, double* __restrict__ b) {
  extern __shared__ double ts[];
  const int j = blockIdx.x;
  for (int g = threadIdx.x; g < n_grp; g += blockDim.x) ts[g] = T[(size_t)j * n_grp + g];
  __syncthreads();
  for (int l = threadIdx.x; l < n_lvl; l += blockDim.x) {
    double s = 0.0;
    for (int q = lvl_ptr[l]; q < lvl_ptr[l + 1]; q++) s += ts[lvl_grp[q]];
    b[(size_t)j * P + lvl_cc[l]] = s;
  }
}

int launch_assemble_b(Ctx* c, double* out) {
  if (c->n_grp == 0) return GPL_OK;
  ProfScope ps(c, "assemble_b");
  const size_t smem = sizeof(double) * c->n_grp;  // at most 8,192 groups
  if (smem > 48 * 1024)
    GPL_TRY(c, cudaFuncSetAttribute(k_assemble_b, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  k_assemble_b<<<c->J, 128, smem, c->stream>>>(c->P, c->n_lvl, c->n_grp, c->lvl_cc_d, c->lvl_ptr_d, c->lvl_grp_d, c->gT,
                                               out);
  GPL_LAUNCHED(c, "k_assemble_b");
  return GPL_OK;
}

// h and kappa per (gene, group) from Psi_j^{-1}
__global__ void k_group_tables(int P, int n_d, int n_cv, int n_grp, const int* __restrict__ dcol,
                               const int* __restrict__ cv_nh, const int* __restrict__ glev,
                               const double* __restrict__ S, double* __restrict__ tab) {
  const int j = blockIdx.x;
  const double* Sj = S + (size_t)j * P * P;
  const int ld = n_d + 1;
  double* tj = tab + (size_t)j * n_grp * ld;
  for (int e = threadIdx.x; e < n_grp * ld; e += blockDim.x) {
    const int g = e / ld, a = e % ld;
    const int* lv = glev + g * n_cv;
    double s = 0.0;
    if (a < n_d) {
      const size_t r = dcol[a];
      for (int v = 0; v < n_cv; v++) s += Sj[r + (size_t)(cv_nh[v] + lv[v]) * P];
    } else {
      for (int v = 0; v < n_cv; v++)
        for (int v2 = 0; v2 < n_cv; v2++) s += Sj[(cv_nh[v] + lv[v]) + (size_t)(cv_nh[v2] + lv[v2]) * P];
    }
    tj[e] = s;
  }
}

int launch_group_tables(Ctx* c) {
  if (c->n_grp == 0) return GPL_OK;
  ProfScope ps(c, "group_tables");
  k_group_tables<<<c->J, 256, 0, c->stream>>>(c->P, c->n_d, c->n_cv, c->n_grp, c->dcol_d, c->cv_nh_d, c->glev_d,
                                              c->PsiInv, c->gsum);
  GPL_LAUNCHED(c, "k_group_tables");
  return GPL_OK;
}

int launch_hk(Ctx* c) {
  if (c->n_grp == 0) return GPL_OK;
  ProfScope ps(c, "hk");
  return dgen_hk(c);
}

}  // namespace gpl
