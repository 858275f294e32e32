// Gradient of the objective (replaces getGradLogDelta/collectGradLogDelta ggplvm.cu:210-281,
// getGradLogOmega :301-376, getC2 :57-100, getGradTau :103-145, getGradLogRho/collect
// :148-205).
//
// The reference solves Psi_j z_i for every (cell, gene) pair (N*J solves of size P). Here
// the explicit inverses S_j = Psi_j^{-1} are formed once per gene and the per-cell sums
// over genes become one contraction over the dense columns d_i of z_i,
//     A[i, a] = sum_j O_ij (S_j[DD] d_i)_a = sum_{j,b} (O_ij d_ib) S_j[b, a],   O = W / Omega
// plus per-group terms for the categorical levels (k_groups.cu), over the unique column pairs
// (launch_pair_uq).
#include "gpl_internal.cuh"

namespace gpl {

// ---- d/d log delta ------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_grad_delta(int P, int M, int g0, const int* __restrict__ mk,
                                                    const double* __restrict__ delta, const double* __restrict__ K,
                                                    const double* __restrict__ S, const double* __restrict__ tBeta,
                                                    const double* __restrict__ phi, int J, int pvars,
                                                    const int* __restrict__ nh, double* __restrict__ gdtmp) {
  extern __shared__ double gd[];  // [P] the columns' terms
  __shared__ double sh[32];
  __shared__ double sq;
  const int j = blockIdx.x;
  const double* Sj = S + (size_t)j * P * P;
  const double* tb = tBeta + (size_t)j * P;
  // tb_GP^T Kmm tb_GP (quadform, util_cuda.cu:442-451)
  double part = 0.0;
  for (int a = threadIdx.x; a < M; a += blockDim.x) {
    double t = K[a + a * M] * tb[g0 + a];
    for (int b = a + 1; b < M; b++) t += 2.0 * K[a + b * M] * tb[g0 + b];
    part += tb[g0 + a] * t;
  }
  const double q = block_sum(part, sh);
  if (threadIdx.x == 0) sq = q;
  __syncthreads();
  const double phij = phi[j];
  for (int k = threadIdx.x; k < P; k += blockDim.x) {
    const double dk = delta[mk[k]];
    double psikk;
    if (k < g0) {
      psikk = Sj[k + (size_t)k * P];
    } else {  // (S_j Kmm[:, kk])_k over the GP block
      const int kk = k - g0;
      psikk = 0.0;
      for (int l = 0; l < M; l++) {
        const double kv = l < kk ? K[l + kk * M] : K[kk + l * M];
        psikk += Sj[k + (size_t)(g0 + l) * P] * kv;
      }
    }
    double sum = -(dk - psikk) / dk / dk / 2.0;
    if (k < g0) sum += tb[k] * tb[k] / dk / dk / phij / 2.0;
    else if (k == g0) sum += sq / dk / dk / phij / 2.0;
    gd[k] = sum * dk;
  }
  __syncthreads();
  // the gene's sum over each variable's columns, a warp per variable
  for (int l = threadIdx.x >> 5; l < pvars; l += blockDim.x >> 5) {
    double s = 0.0;
    for (int k = nh[l] + (threadIdx.x & 31); k < nh[l + 1]; k += 32) s += gd[k];
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) gdtmp[(size_t)l * J + j] = s;
  }
}

__global__ void __launch_bounds__(256) k_collect_delta(int J, int N, int pvars, const double* __restrict__ gdtmp,
                                                       const double* __restrict__ sums,
                                                       const double* __restrict__ delta, double* __restrict__ grad) {
  __shared__ double sh[32];
  const int l = blockIdx.x;
  double s = 0.0, t = 0.0;
  for (int j = threadIdx.x; j < J; j += blockDim.x) s += gdtmp[(size_t)l * J + j];
  if (l == pvars - 1 && threadIdx.x < kStateParts) t = sums[2 * kStateParts + threadIdx.x];
  s = block_sum(s, sh);
  t = block_sum(t, sh);
  if (threadIdx.x == 0) grad[N + l] = s - kWt * t * delta[pvars - 1];
}

int launch_grad_delta(Ctx* c) {
  ProfScope ps(c, "grad_delta");
  const int g0 = c->nh[c->p - 1];
  const int rc = launch_state_sums(c);
  if (rc) return rc;
  k_grad_delta<<<c->J, 256, sizeof(double) * c->P, c->stream>>>(c->P, c->M, g0, c->mk_d, c->delta, c->Kmm, c->PsiInv,
                                                                c->tBeta, c->phi, c->J, c->p, c->nh_d, c->gdtmp);
  GPL_LAUNCHED(c, "k_grad_delta");
  k_collect_delta<<<c->p, 256, 0, c->stream>>>(c->J, c->N, c->p, c->gdtmp, c->state_sums, c->delta, c->grad);
  GPL_LAUNCHED(c, "k_collect_delta");
  return GPL_OK;
}

__global__ void k_recip(int n, const double* __restrict__ x, double* __restrict__ r) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) r[i] = 1.0 / x[i];
}

// per-cell epilogue of getGradLogOmega (ggplvm.cu:352-374). With A = U (dense rows of
// sum_j O_ij S_j z_i without the level terms) and HK = [sum_j O_ij h_{j,g(i)} | sum_j O_ij
// kappa_{j,g(i)}] (absent when no variable is grouped):
//   sum_j O_ij z_i^T S_j z_i = d_i . (A_i + 2 H_i) + K_i,   sum_j O_ij (S_j z_i)_GP = A_i[GP] + H_i[GP]
__global__ void k_grad_omega_cell(int N, int ldN, int n_d, int dg0, int J, int M, int Q, int pvars,
                                  const double* __restrict__ D, const double* __restrict__ U,
                                  const double* __restrict__ HK, const double* __restrict__ tnsum,
                                  const double* __restrict__ W, const double* __restrict__ Omega,
                                  const double* __restrict__ delta, const double* __restrict__ titsias,
                                  const double* __restrict__ KinvKmn, const double* __restrict__ X,
                                  const double* __restrict__ T, const double* __restrict__ rho,
                                  double* __restrict__ C1, double* __restrict__ grad) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const double om = Omega[i];
  const double Oii = W[(size_t)J * ldN + i];
  double q = 0.0;
  for (int a = 0; a < n_d; a++) {
    double u = U[i + (size_t)a * ldN];
    if (HK) u += 2.0 * HK[i + (size_t)a * ldN];
    q += D[(size_t)a * ldN + i] * u;
  }
  if (HK) q += HK[i + (size_t)n_d * ldN];
  const double dgp = delta[pvars - 1];
  double sum = -((double)J) / om / 2.0 + q / om / 2.0 + tnsum[i];
  sum += kWt * dgp * Oii / om * titsias[i];
  grad[i] = sum * om + kIgb / om - kIgap1;
  double* gX = grad + N + pvars;
  double ci1 = 0.0, g0x = 0.0;
  for (int k = 0; k < M; k++) {
    double v = U[i + (size_t)(dg0 + k) * ldN];
    if (HK) v += HK[i + (size_t)(dg0 + k) * ldN];
    double cik = C1[i + (size_t)k * ldN] - v;
    cik += kWt * dgp * Oii * KinvKmn[i + (size_t)k * ldN];
    cik *= D[(size_t)(dg0 + k) * ldN + i];
    C1[i + (size_t)k * ldN] = cik;
    ci1 += cik;
    const double t = (X[i] - T[k]) / 2.0;
    g0x -= cik * sin(t) * cos(t) / rho[0];
  }
  gX[i] = g0x;
  for (int qd = 1; qd < Q; qd++) {
    double d = 0.0;
    for (int k = 0; k < M; k++) d += C1[i + (size_t)k * ldN] * T[k + qd * M];
    gX[i + (size_t)qd * N] = (d - ci1 * X[i + (size_t)qd * N]) / rho[qd];
  }
}

int launch_grad_omega(Ctx* c) {
  int rc = launch_zbeta(c, c->tBeta, c->scratch);  // E = Z tBeta
  if (rc) return rc;
  {
    ProfScope ps(c, "tn_sum");
    k_recip<<<div_up(c->J, 256), 256, 0, c->stream>>>(c->J, c->phi, c->rphi);
    GPL_LAUNCHED(c, "k_recip");
    if ((rc = launch_tn_sum(c, c->scratch, c->red))) return rc;
  }
  rc = launch_c1_tn(c);  // C1 = sum_j tn/phi tBeta_GP
  if (rc) return rc;
  if (c->precision == GPL_PREC_BF16X3 && c->tc_grad) {
    rc = launch_tc_grad(c);
    if (rc) return rc;
  } else if ((rc = launch_pair_uq(c))) {
    return rc;
  }
  rc = launch_group_tables(c);
  if (rc) return rc;
  rc = launch_hk(c);
  if (rc) return rc;
  ProfScope ps(c, "grad_omega_cell");
  k_grad_omega_cell<<<div_up(c->N, 128), 128, 0, c->stream>>>(
      c->N, c->ldN, c->n_d, c->dg0, c->J, c->M, c->Q, c->p, c->Dm, c->U, c->n_grp ? c->HK : nullptr, c->red, c->W,
      c->Omega, c->delta, c->titsias, c->KinvKmn, c->X, c->T, c->rho, c->C1, c->grad);
  GPL_LAUNCHED(c, "k_grad_omega_cell");
  return GPL_OK;
}

// ---- C2 (M x M adjoint of Kmm) --------------------------------------------------------------
int launch_c2(Ctx* c) {
  ProfScope ps(c, "c2");
  // Kmm^{-1} from the factor in Kinv's lower triangle (column k = cholsl(Kinv, e_k))
  const int rc = launch_cholinv(c, c->Kinv, c->M, c->KmmInv);
  return rc ? rc : dgen_c2(c);
}

// ---- d/dT and d/dlog rho -------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_grad_tau_rho(int N, int ldN, int M, int Q, int pvars,
                                                      const double* __restrict__ X, const double* __restrict__ T,
                                                      const double* __restrict__ rho, const double* __restrict__ C1,
                                                      const double* __restrict__ C2, double* __restrict__ grad,
                                                      double* __restrict__ grtmp) {
  __shared__ double sh[32];
  const int m = blockIdx.x, q = blockIdx.y;
  const double rq = rho[q];
  const double* c1 = C1 + (size_t)m * ldN;
  double a1 = 0.0, a2 = 0.0, r1 = 0.0;  // tau sums over cells, rho sum over cells
  double b1 = 0.0, b2 = 0.0, r2 = 0.0;  // the same over inducing points
  if (q == 0) {
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
      const double t = (X[i] - T[m]) / 2.0;
      const double st = sin(t);
      a1 += c1[i] * st * cos(t);
      r1 += c1[i] * st * st / rq / rq;
    }
    for (int i = threadIdx.x; i < M; i += blockDim.x) {
      const double t = (T[i] - T[m]) / 2.0;
      const double st = sin(t);
      b1 += C2[m + i * M] * st * cos(t);
      r2 += C2[i + m * M] * st * st / rq / rq;
    }
  } else {
    const double tm = T[m + q * M];
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
      const double xi = X[i + (size_t)q * N];
      a1 += c1[i] * xi;
      a2 += c1[i];
      const double d = xi - tm;
      r1 += c1[i] * d * d / rq / rq / 2.0;
    }
    for (int i = threadIdx.x; i < M; i += blockDim.x) {
      b1 += C2[m + i * M] * T[i + q * M];
      b2 += C2[m + i * M];
      const double d = T[i + q * M] - tm;
      r2 += C2[i + m * M] * d * d / rq / rq / 2.0;
    }
  }
  a1 = block_sum(a1, sh);
  a2 = block_sum(a2, sh);
  b1 = block_sum(b1, sh);
  b2 = block_sum(b2, sh);
  r1 = block_sum(r1, sh);
  r2 = block_sum(r2, sh);
  if (threadIdx.x == 0) {
    double* gT = grad + N + pvars + (size_t)N * Q;
    if (q == 0) {
      gT[m] = a1 / rho[0] + 2.0 * b1 / rho[0];
    } else {
      const double tm = T[m + q * M];
      gT[m + q * M] = (a1 - a2 * tm) / rq + 2.0 * (b1 - b2 * tm) / rq;
    }
    grtmp[q + m * Q] = (r1 + r2) * rq;
  }
}

__global__ void k_collect_rho(int N, int M, int Q, int pvars, const double* __restrict__ grtmp,
                              double* __restrict__ grad) {
  const int q = threadIdx.x;
  if (q >= Q) return;
  double s = 0.0;
  for (int k = 0; k < M; k++) s += grtmp[q + k * Q];
  grad[N + pvars + (size_t)N * Q + (size_t)M * Q + q] = s;
}

int launch_grad_tau_rho(Ctx* c) {
  ProfScope ps(c, "grad_tau_rho");
  dim3 g(c->M, c->Q);
  k_grad_tau_rho<<<g, 256, 0, c->stream>>>(c->N, c->ldN, c->M, c->Q, c->p, c->X, c->T, c->rho, c->C1, c->C2,
                                           c->grad, c->grtmp);
  GPL_LAUNCHED(c, "k_grad_tau_rho");
  k_collect_rho<<<1, 32 * div_up(c->Q, 32), 0, c->stream>>>(c->N, c->M, c->Q, c->p, c->grtmp, c->grad);
  GPL_LAUNCHED(c, "k_collect_rho");
  return GPL_OK;
}

}  // namespace gpl
