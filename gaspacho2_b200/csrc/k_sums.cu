// Sums over genes for every cell and sums over cells that several phases share.
//
//   k_cell_sums    per cell, over all genes: sum_j W_ij (getOinvt, ggplvm.cu:284-294) or the gradient's
//                  sum_j tn_ij^2 / W_ij / phi_j (getGradLogOmega, ggplvm.cu:301-376). Bound: one or three
//                  reads of cells x genes. A block takes 64 cells (two per lane, 16-byte loads) and its
//                  eight warps every eighth gene; with few cells the genes are split over grid y, so that
//                  the blocks fill the SMs, and k_cell_sums_add adds the parts in order.
//   k_state_sums   sum_i log Omega_i, sum_i 1/Omega_i and sum_i Oinvt_i titsias_i as kStateParts partial
//                  sums each, for the likelihoods, their collection and the gradient of log delta.
// All sums have a fixed order (deterministic).
#include <algorithm>

#include "gpl_internal.cuh"

namespace gpl {

// Gene ranges of a sum per cell over all genes in blocks of 64 cells: about six blocks per SM, 32 genes at least.
int cell_sum_ranges(const Ctx* c) {
  return std::max(1, std::min(6 * c->sm_count / div_up(c->N, 64), c->J / 32));
}

namespace {
constexpr int kOinvt = 0, kTn = 1;

template <int MODE>
__device__ __forceinline__ double cell_sum_out(double s, double om) {
  // tn^2 / W / phi / 2 with tn = (W/Omega)(nu - E) is W (nu - E)^2 / (2 phi Omega^2)
  return MODE == kOinvt ? s / om : s / (2.0 * om * om);
}

template <int MODE>
__global__ void __launch_bounds__(256) k_cell_sums(int N, int ldN, int J, int jper, const double* __restrict__ W,
                                                   const double* __restrict__ Nu, const double* __restrict__ E,
                                                   const double* __restrict__ Omega, const double* __restrict__ rphi,
                                                   double* __restrict__ part, double* __restrict__ out) {
  __shared__ double sh[8][64];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i = blockIdx.x * 64 + 2 * lane;  // even; ldN is a multiple of 32, so a pair lies in the column
  const int j1 = min(J, (int)(blockIdx.y + 1) * jper);
  double2 s = make_double2(0.0, 0.0);
  if (i < N) {
#pragma unroll 4
    for (int j = blockIdx.y * jper + warp; j < j1; j += 8) {
      const size_t e = (size_t)j * ldN + i;
      const double2 w = *reinterpret_cast<const double2*>(W + e);
      if (MODE == kOinvt) {
        s.x += w.x;
        s.y += w.y;
      } else {
        const double2 u = *reinterpret_cast<const double2*>(Nu + e), v = *reinterpret_cast<const double2*>(E + e);
        const double r = rphi[j], dx = u.x - v.x, dy = u.y - v.y;
        s.x += w.x * dx * dx * r;
        s.y += w.y * dy * dy * r;
      }
    }
  }
  sh[warp][2 * lane] = s.x;
  sh[warp][2 * lane + 1] = s.y;
  __syncthreads();
  const int c = blockIdx.x * 64 + threadIdx.x;
  if (threadIdx.x < 64 && c < N) {
    double t = 0.0;
#pragma unroll
    for (int k = 0; k < 8; k++) t += sh[k][threadIdx.x];
    if (gridDim.y == 1) out[c] = cell_sum_out<MODE>(t, Omega[c]);
    else part[(size_t)blockIdx.y * ldN + c] = t;
  }
}

template <int MODE>
__global__ void k_cell_sums_add(int N, int ldN, int ns, const double* __restrict__ part,
                                const double* __restrict__ Omega, double* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  double s = 0.0;
  for (int k = 0; k < ns; k++) s += part[(size_t)k * ldN + i];
  out[i] = cell_sum_out<MODE>(s, Omega[i]);
}

template <int MODE>
int launch_cell_sums(Ctx* c, const double* E, double* out) {
  const int bx = div_up(c->N, 64), ns = cell_sum_ranges(c);
  if (ns > 1) {
    const int rc = ensure_part(c, (size_t)ns * c->ldN);
    if (rc) return rc;
  }
  k_cell_sums<MODE><<<dim3(bx, ns), 256, 0, c->stream>>>(c->N, c->ldN, c->J, div_up(c->J, ns), c->W, c->Nu, E,
                                                         c->Omega, c->rphi, c->part, out);
  GPL_LAUNCHED(c, "k_cell_sums");
  if (ns > 1) {
    k_cell_sums_add<MODE><<<div_up(c->N, 256), 256, 0, c->stream>>>(c->N, c->ldN, ns, c->part, c->Omega, out);
    GPL_LAUNCHED(c, "k_cell_sums_add");
  }
  return GPL_OK;
}

__global__ void __launch_bounds__(256) k_state_sums(int N, const double* __restrict__ Omega,
                                                    const double* __restrict__ Oinvt,
                                                    const double* __restrict__ titsias, double* __restrict__ out) {
  __shared__ double sh[32];
  double a = 0.0, b = 0.0, t = 0.0;
  for (int i = blockIdx.x * 256 + threadIdx.x; i < N; i += kStateParts * 256) {
    const double om = Omega[i];
    a += log(om);
    b += 1.0 / om;
    t += Oinvt[i] * titsias[i];
  }
  a = block_sum(a, sh);
  b = block_sum(b, sh);
  t = block_sum(t, sh);
  if (threadIdx.x == 0) {
    out[blockIdx.x] = a;
    out[kStateParts + blockIdx.x] = b;
    out[2 * kStateParts + blockIdx.x] = t;
  }
}
}  // namespace

size_t cell_sums_part(const Ctx* c) { return (size_t)cell_sum_ranges(c) * c->ldN; }

int launch_oinvt(Ctx* c) {
  ProfScope ps(c, "oinvt");
  return launch_cell_sums<kOinvt>(c, nullptr, c->W + (size_t)c->J * c->ldN);
}

int launch_tn_sum(Ctx* c, const double* E, double* out) { return launch_cell_sums<kTn>(c, E, out); }

int launch_state_sums(Ctx* c) {
  k_state_sums<<<kStateParts, 256, 0, c->stream>>>(c->N, c->Omega, c->W + (size_t)c->J * c->ldN, c->titsias,
                                                   c->state_sums);
  GPL_LAUNCHED(c, "k_state_sums");
  return GPL_OK;
}

}  // namespace gpl
