// Dense levels of the Chebyshev M2L: combinations of a parent's children with
// three products per child coordinate instead of four.  For one parent offset
// D the block E_{2D + s - t} of (target child t, source child s) is Toeplitz in
// each coordinate, so per coordinate
//   y0 = E0 (x0 + x1) + (E+ - E0) x1,   y1 = E0 (x0 + x1) + (E- - E0) x0.
// Combination j = 9 jx + 3 jy + jz, per coordinate 0: both children, 1: child
// 1, 2: child 0; outputs y0 = [0] + [1], y1 = [0] + [2] per coordinate.
#pragma once
#include "fmm.cuh"

namespace pbbfmm {

// A level takes the combinations when its parents are nearly full: with a
// target and b source children per parent the direct list has 26 x 0.91 a b
// products per parent, the combinations 26 x 27; the line is drawn at a b > 36
// (27 / 0.91 = 29.7, and a fifth for forming the combinations).
inline bool cheb_kara_level(const pbbfmm_tree* t, int l) {
  if (l < 3) return false;
  const double np = t->lists.ntgt[l - 1], ns = t->lists.nsrc[l - 1];
  return (double)t->lists.ntgt[l] * t->lists.nsrc[l] > 36.0 * np * ns;
}

template <typename T, class Out>
__device__ __forceinline__ void kara_combine(const T* v, Out out) {
#pragma unroll
  for (int jz = 0; jz < 3; ++jz) {
    T u[4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      u[q] = jz == 0 ? v[2 * q] + v[2 * q + 1] : v[2 * q + (jz == 1 ? 1 : 0)];
#pragma unroll
    for (int jy = 0; jy < 3; ++jy) {
      T w[2];
#pragma unroll
      for (int q = 0; q < 2; ++q)
        w[q] = jy == 0 ? u[2 * q] + u[2 * q + 1] : u[2 * q + (jy == 1 ? 1 : 0)];
#pragma unroll
      for (int jx = 0; jx < 3; ++jx)
        out(9 * jx + 3 * jy + jz, jx == 0 ? w[0] + w[1] : w[jx == 1 ? 1 : 0]);
    }
  }
}

// which of parent p's children hold points (warp-collective)
__device__ __forceinline__ unsigned children_present(const int* __restrict__ start, int64_t p,
                                                     int span) {
  const int lane = threadIdx.x & 31;
  int bound = 0;
  if (lane <= 8) bound = start[(8 * p + lane) * span];
  unsigned present = 0;
#pragma unroll
  for (int ch = 0; ch < 8; ++ch)
    present |= (__shfl_sync(0xffffffffu, bound, ch + 1) != __shfl_sync(0xffffffffu, bound, ch))
                   ? 1u << ch : 0u;
  return present;
}

// pf of the children of the listed target parents, from ky[(parent 27 + j) C +
// column][rf]: warp per (parent, column).
template <typename T>
__global__ void k_kara_out(const int* __restrict__ parents, int np, const T* __restrict__ ky,
                           T* __restrict__ pf, int C, int rf) {
  const int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= (int64_t)np * C) return;
  const int64_t p = parents[w / C];
  const int c = (int)(w % C);
  for (int f = lane; f < rf; f += 32) {
    T y[kKaraJ];
#pragma unroll
    for (int j = 0; j < kKaraJ; ++j) y[j] = ky[((p * kKaraJ + j) * C + c) * rf + f];
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const int jx = 9 * (1 + ((t >> 2) & 1)), jy = 3 * (1 + ((t >> 1) & 1)), jz = 1 + (t & 1);
      pf[((8 * p + t) * C + c) * rf + f] = ((y[0] + y[jz]) + (y[jy] + y[jy + jz])) +
                                           ((y[jx] + y[jx + jz]) + (y[jx + jy] + y[jx + jy + jz]));
    }
  }
}

}  // namespace pbbfmm
