// Dense levels of the Chebyshev M2L: combinations of a parent's children with
// three products per child coordinate instead of four.  For one parent offset
// D the block E_{2D + s - t} of (target child t, source child s) is Toeplitz in
// each coordinate, so per coordinate
//   y0 = E0 (x0 + x1) + (E+ - E0) x1,   y1 = E0 (x0 + x1) + (E- - E0) x0.
// Combination j = 9 jx + 3 jy + jz, per coordinate 0: both children, 1: child
// 1, 2: child 0; outputs y0 = [0] + [1], y1 = [0] + [2] per coordinate.
#pragma once
#include <algorithm>
#include <vector>

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

// The far field's launches.  A part is a level on its direct lists (nj = 0), or
// columns [c0, c0 + nc) of combinations [j0, j0 + nj) of a dense level; a launch
// holds the parts whose arrays are there together.
struct ChebPart {
  int level, c0, nc, j0, nj;
  int64_t x, y;  // byte offsets of its combined proxies and sums (direct: of its split proxies)
};
struct ChebPlan {
  std::vector<std::vector<ChebPart>> launches;
  int64_t x_bytes = 0, y_bytes = 0, direct_bytes = 0;
};
// Parts of one launch at most (the level tables of the kernels).
constexpr int kChebParts = kMaxLevel - 1;

// dense[l], used[l] (has targets) for levels 2..L; xrow, yrow: bytes of one
// combined proxy and one sum; drow: of one split proxy of a direct level (0:
// none).  The combinations of all columns of all dense levels take 27 / 8 times
// the levels' own proxies and sums, so they get at most `bound` bytes at a time:
// columns are independent of each other, and the combinations that differ in jx
// only meet in the output step (k_kara_out9), so a level whose arrays are larger
// runs in groups of columns, if need be in three groups of 9 combinations, and on
// its direct list where one column of 9 does not fit either.
inline ChebPlan cheb_plan(const bool* dense, const bool* used, int L, int C, int64_t xrow,
                          int64_t yrow, int64_t drow, int64_t bound) {
  auto pad = [](int64_t b) { return (b + 255) / 256 * 256; };
  ChebPlan p;
  std::vector<ChebPart> cur;
  int64_t cx = 0, cy = 0, cd = 0, dcap = bound;
  for (int l = 2; l <= L; ++l) dcap = std::max(dcap, pad(cells_at(l) * C * drow));
  auto add = [&](ChebPart q, int64_t x, int64_t y, int64_t d) {
    if (!cur.empty() &&
        (cx + cy + x + y > bound || cd + d > dcap || (int)cur.size() == kChebParts)) {
      p.launches.push_back(cur);
      cur.clear();
      cx = cy = cd = 0;
    }
    q.x = q.nj ? cx : cd;
    q.y = cy;
    cur.push_back(q);
    cx += x, cy += y, cd += d;
    p.x_bytes = std::max(p.x_bytes, cx);
    p.y_bytes = std::max(p.y_bytes, cy);
    p.direct_bytes = std::max(p.direct_bytes, cd);
  };
  // deepest level first: the shallow levels' few items fill the last wave
  for (int l = L; l >= 2; --l) {
    if (!used[l]) continue;
    const int64_t parents = cells_at(l - 1);
    int nj = kKaraJ, nc = 0;
    if (dense[l])
      for (;; nj = kKaraJ / 3) {
        nc = (int)std::min<int64_t>(C, std::max<int64_t>(bound - 512, 0) / (nj * parents * (xrow + yrow)));
        if (nc > 0 || nj < kKaraJ) break;
      }
    if (nc == 0) {
      add({l, 0, C, 0, 0, 0, 0}, 0, 0, pad(cells_at(l) * C * drow));
      continue;
    }
    const int groups = (C + nc - 1) / nc;
    for (int g = 0; g < groups; ++g) {
      const int c0 = (int)((int64_t)C * g / groups), n = (int)((int64_t)C * (g + 1) / groups) - c0;
      for (int j0 = 0; j0 < kKaraJ; j0 += nj)
        add({l, c0, n, j0, nj, 0, 0}, pad(parents * nj * n * xrow), pad(parents * nj * n * yrow), 0);
    }
  }
  if (!cur.empty()) p.launches.push_back(cur);
  return p;
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

// pf of the children of the listed target parents, columns [c0, c0 + nc) of C,
// from ky[(parent 27 + j) nc + column][rf]: warp per (parent, column).
template <typename T>
__global__ void k_kara_out(const int* __restrict__ parents, int np, const T* __restrict__ ky,
                           T* __restrict__ pf, int C, int c0, int nc, int rf) {
  const int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= (int64_t)np * nc) return;
  const int64_t p = parents[w / nc];
  const int c = (int)(w % nc);
  for (int f = lane; f < rf; f += 32) {
    T y[kKaraJ];
#pragma unroll
    for (int j = 0; j < kKaraJ; ++j) y[j] = ky[((p * kKaraJ + j) * nc + c) * rf + f];
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const int jx = 9 * (1 + ((t >> 2) & 1)), jy = 3 * (1 + ((t >> 1) & 1)), jz = 1 + (t & 1);
      pf[((8 * p + t) * C + c0 + c) * rf + f] =
          ((y[0] + y[jz]) + (y[jy] + y[jy + jz])) +
          ((y[jx] + y[jx + jz]) + (y[jx + jy] + y[jx + jy + jz]));
    }
  }
}

// The same in three steps, jx = 0, 1, 2, from ky[(parent 9 + j % 9) nc + column]
// of the combinations 9 jx + ...: jx = 0 writes all children, 1 and 2 add to those
// of bx = 0 and 1 (the sums of k_kara_out in the same order).
template <typename T>
__global__ void k_kara_out9(const int* __restrict__ parents, int np, const T* __restrict__ ky,
                            T* __restrict__ pf, int C, int c0, int nc, int rf, int jx) {
  const int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= (int64_t)np * nc) return;
  const int64_t p = parents[w / nc];
  const int c = (int)(w % nc);
  for (int f = lane; f < rf; f += 32) {
    T y[9];
#pragma unroll
    for (int j = 0; j < 9; ++j) y[j] = ky[((p * 9 + j) * nc + c) * rf + f];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int jy = 3 * (1 + (t >> 1)), jz = 1 + (t & 1);
      const T v = (y[0] + y[jz]) + (y[jy] + y[jy + jz]);
      T* d = pf + ((8 * p + t) * C + c0 + c) * rf + f;
      const int64_t bx = (int64_t)4 * C * rf;  // to the child of bx = 1
      if (jx == 0) {
        d[0] = v;
        d[bx] = v;
      } else {
        d[jx == 1 ? 0 : bx] += v;
      }
    }
  }
}

// k_kara_out of one part (lists: the level's target parents).
template <typename T>
inline int launch_kara_out(const pbbfmm_tree* t, const ChebPart& q, const T* ky, T* pf, int C,
                           int rf, cudaStream_t st) {
  const int np = t->lists.ntgt[q.level - 1];
  const int* parents = t->ws.lists.as<int>() + t->lists.tgt_off[q.level - 1];
  const unsigned g = (unsigned)(((int64_t)np * q.nc + 7) / 8);
  if (q.nj == kKaraJ)
    k_kara_out<T><<<g, 256, 0, st>>>(parents, np, ky, pf, C, q.c0, q.nc, rf);
  else
    k_kara_out9<T><<<g, 256, 0, st>>>(parents, np, ky, pf, C, q.c0, q.nc, rf, q.j0 / 9);
  PB_LAUNCH("kara_out");
  return PBBFMM_OK;
}

}  // namespace pbbfmm
