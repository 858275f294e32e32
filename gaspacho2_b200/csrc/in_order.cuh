// Sums over a thread's elements in their order, with the loads of K elements issued before the first
// use: the per-gene reductions over cells and counts are bound by the latency of their loads (a gene per
// block, some 80 elements a thread), not by the sums. Same values, same order as an element at a time.
// 20,000 cells x 1,001 genes: k_de_lkhd 188 -> 117 us. (Where every element ends in a division, as in
// the residual sums of k_beta_phi, the divisions count and a plain loop is as fast: 62 / 72 us.)
#pragma once

#include <type_traits>
#include <utility>

namespace gpl {

// use(load(i)) for i = b, b + step, ... below e
template <int K, class I, class Load, class Use>
__device__ __forceinline__ void in_order(I b, I e, int step, Load load, Use use) {
  for (I i = b; i < e; i += (I)K * step) {
    typename std::decay<decltype(load(b))>::type v[K];
#pragma unroll
    for (int k = 0; k < K; k++)
      if (i + (I)k * step < e) v[k] = load(i + (I)k * step);
#pragma unroll
    for (int k = 0; k < K; k++)
      if (i + (I)k * step < e) use(v[k]);
  }
}

// use(x, gather(x)) with x = load(i): the gathers are issued before the first use too
template <int K, class I, class Load, class Gather, class Use>
__device__ __forceinline__ void in_order(I b, I e, int step, Load load, Gather gather, Use use) {
  using X = typename std::decay<decltype(load(b))>::type;
  using Y = typename std::decay<decltype(gather(std::declval<X>()))>::type;
  for (I i = b; i < e; i += (I)K * step) {
    X x[K];
    Y y[K];
#pragma unroll
    for (int k = 0; k < K; k++)
      if (i + (I)k * step < e) x[k] = load(i + (I)k * step);
#pragma unroll
    for (int k = 0; k < K; k++)
      if (i + (I)k * step < e) y[k] = gather(x[k]);
#pragma unroll
    for (int k = 0; k < K; k++)
      if (i + (I)k * step < e) use(x[k], y[k]);
  }
}

struct CountAt {
  int cell;
  double y;
};

}  // namespace gpl
