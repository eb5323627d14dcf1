// Shared pieces of the interpolation passes between levels (M2M in upward.cu,
// L2L in downward.cu) for orders that fit registers.
//
// Lane = one (parent, column) unit; a CTA holds U neighbouring units and N
// threads per unit.  The tensor-product transforms of a unit run on registers:
// thread l1 takes the N x N row (l2, l3) through the z and y passes, the x pass
// runs over N of the N x N (l2, l3) pairs per thread, with one array between
// them in shared memory as [element][unit] (conflict-free).  The passes follow
// the octree: children that share a coordinate share that coordinate's pass (14
// one-dimensional passes per parent instead of 24).  The operators are kernel
// parameters, so every multiply-add takes its coefficient from the constant
// bank.  Bound: HBM and shared memory; with one warp per (parent, column),
// coefficients read from shared memory, the shared-memory pipe was 94 % busy.
// Measured, M2M and L2L of 1M uniform points at order 5, 8 columns: float32
// 1.05 and 1.20 -> 0.40 and 0.58 ms, float64 2.45 and 2.27 -> 0.80 and 1.29 ms; 1
// column, float32 0.167 and 0.190 -> 0.107 and 0.139 ms.  (The rows are copied a
// warp per unit: with a unit and element computed per value, the copies' index
// arithmetic made both passes slower than before.)
#pragma once
#include "fmm.cuh"

namespace pbbfmm {

template <int N, typename T>
struct InterpOps {
  T w[2][N * N];  // child 0 / 1 of a coordinate
};

template <int N, typename T>
struct InterpCfg {
  static constexpr int n2 = N * N, n3 = n2 * N;
  static constexpr bool use = N <= (sizeof(T) == 4 ? 6 : 5);
  // three arrays of n^3 x U (and padding): four CTAs per SM or so
  static constexpr int U = 3 * n3 * 33 * (int)sizeof(T) <= 56 * 1024 ? 32 : 16;
  static constexpr int threads = (N * U + 31) / 32 * 32;
  static constexpr size_t smem = sizeof(T) * (size_t)n3 * 3 * (U + 1);
};

template <int N, typename T>
inline InterpOps<N, T> interp_ops(const pbbfmm_tree* t) {
  InterpOps<N, T> o;
  for (int i = 0; i < 2 * N * N; ++i) o.w[i / (N * N)][i % (N * N)] = (T)t->w.Cweights[i];
  return o;
}

}  // namespace pbbfmm
