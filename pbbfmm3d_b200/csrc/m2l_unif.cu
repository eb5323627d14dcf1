// Uniform-grid far field: FFT of the padded moments, the
// frequency-domain M2L, and the inverse FFT to local coefficients.
//
// Reference: UpwardPass padding + R2HC (include/compute.hpp:337-372),
// FarFieldInteractions / FrequencyProduct / HC2R (include/compute.hpp:
// 488-544, 930-943) and the stencils of ComputeKernelUnif
// (src/H2_3D_Tree.cpp:585-648).
//
// The reference embeds the n^3 moments in a length-(2n-1)^3 vector at offset
// (P-1)/2 and uses a 1-D circular correlation of length P; because the offset
// digits never carry, that equals the 3-D Toeplitz product
//     y[a] = sum_b A[n-1+b-a] x[b],   a, b in [0,n)^3,  A the (2n-1)^3 stencil,
// which is what runs here, as a 3-D real DFT on the m^3 grid (m = 2n-1):
// x placed at grid position b, y read at grid position (a + n) mod m, and
// the operator spectra stored as conj(DFT3(A)).  Only the k3 < n half of each
// spectrum is computed (Hermitian symmetry), and of its k3 = 0 plane, which is
// Hermitian in itself, one half: nk = (m^3 + 1) / 2 complex values per cell
// and column (365 instead of m*m*n = 405 at order 5).  Same sums as the
// reference, different rounding.
//
// Frequency slots.  Jobs j number the kept (k2, k3): first k3 = 1..n-1 for
// every k2, then k3 = 0 for k2 = 1..(m-1)/2, last (0, 0); slot j m + k1, of
// the last job only k1 <= (m-1)/2.
#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <vector>

#include "fmm.cuh"
#include "tcgen05.cuh"
#include "unif_tc.cuh"

namespace pbbfmm {

// ----------------------------------------------------------------- FFT
// Each thread computes one whole 1-D transform of a stage: its n (or m)
// inputs are read once from shared memory and every output is accumulated in
// registers, with the loops fully unrolled so that every twiddle index
// (k l mod m) is a compile-time constant into the __constant__ tables below
// (constant-bank operands of the FMAs, no loads).

// cos / sin of 2 pi j / m for m = 2n - 1, n = 2..kMaxOrder, back to back.
constexpr int kTwTotal = kMaxOrder * kMaxOrder - 1;  // sum_{n=2}^{N} (2n - 1)
__host__ __device__ constexpr int tw_off(int n) { return n <= 2 ? 0 : tw_off(n - 1) + 2 * n - 3; }
__constant__ double c_tw_cos_d[kTwTotal];
__constant__ double c_tw_sin_d[kTwTotal];
__constant__ float c_tw_cos_f[kTwTotal];
__constant__ float c_tw_sin_f[kTwTotal];

template <int n, typename T>
struct Tw {
  static constexpr int m = 2 * n - 1, off = tw_off(n);
  static __device__ __forceinline__ T c(int j) {
    if constexpr (sizeof(T) == 8) return c_tw_cos_d[off + j];
    else return c_tw_cos_f[off + j];
  }
  static __device__ __forceinline__ T s(int j) {
    if constexpr (sizeof(T) == 8) return c_tw_sin_d[off + j];
    else return c_tw_sin_f[off + j];
  }
};

// Fill the tables on the current device (once per device).
int init_fft_twiddles() {
  static std::mutex mu;
  static bool done[64] = {};
  int dev = 0;
  PB_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  if (dev < 64 && done[dev]) return PBBFMM_OK;
  double cd[kTwTotal], sd[kTwTotal];
  float cf[kTwTotal], sf[kTwTotal];
  for (int n = 2; n <= kMaxOrder; ++n) {
    const int m = 2 * n - 1;
    for (int j = 0; j < m; ++j) {
      cd[tw_off(n) + j] = cos(2.0 * M_PI * j / m);
      sd[tw_off(n) + j] = sin(2.0 * M_PI * j / m);
      cf[tw_off(n) + j] = (float)cd[tw_off(n) + j];
      sf[tw_off(n) + j] = (float)sd[tw_off(n) + j];
    }
  }
  PB_CUDA(cudaMemcpyToSymbol(c_tw_cos_d, cd, sizeof(cd)));
  PB_CUDA(cudaMemcpyToSymbol(c_tw_sin_d, sd, sizeof(sd)));
  PB_CUDA(cudaMemcpyToSymbol(c_tw_cos_f, cf, sizeof(cf)));
  PB_CUDA(cudaMemcpyToSymbol(c_tw_sin_f, sf, sizeof(sf)));
  if (dev < 64) done[dev] = true;
  return PBBFMM_OK;
}

// Length-9 transforms (order 5) by one radix-3 step, with l = b + 3a:
//   forward, 5 inputs:  X[k] = U0[k%3] + w^k U1[k%3] + w^2k v2,
//     U0[j] = v0 + v3 w^3j, U1[j] = v1 + v4 w^3j;
//   inverse, 9 inputs:  X[t] = sum_b w^-bt V_b[t%3], V_b[j] = sum_a v[b+3a] w^-3aj,
// for w = e^{-2 pi i / 9}; about half the multiply-adds of the direct sums.
// (a + ib) w^j = (a c + b s) + i (b c - a s), (a + ib) w^-j = (a c - b s) + i (b c + a s).
template <int n, typename T>
__device__ __forceinline__ cplx_t<T> mul_w(cplx_t<T> x, int j) {
  using W = Tw<n, T>;
  return make_cplx<T>(fma(x.x, W::c(j), x.y * W::s(j)), fma(x.y, W::c(j), -x.x * W::s(j)));
}
template <int n, typename T>
__device__ __forceinline__ cplx_t<T> mul_wc(cplx_t<T> x, int j) {
  using W = Tw<n, T>;
  return make_cplx<T>(fma(x.x, W::c(j), -x.y * W::s(j)), fma(x.y, W::c(j), x.x * W::s(j)));
}
// forward 5 -> 9, out(k, X[k]) for k = 0..8
template <int n, typename T, class Out>
__device__ __forceinline__ void dft_5_to_9(const cplx_t<T>* v, Out out) {
  static_assert(2 * n - 1 == 9, "length-9 transform");
  using W = Tw<n, T>;
  cplx_t<T> u0[3], u1[3];
  u0[0] = make_cplx<T>(v[0].x + v[3].x, v[0].y + v[3].y);
  u1[0] = make_cplx<T>(v[1].x + v[4].x, v[1].y + v[4].y);
#pragma unroll
  for (int j = 1; j < 3; ++j) {
    const cplx_t<T> a = mul_w<n, T>(v[3], 3 * j), b = mul_w<n, T>(v[4], 3 * j);
    u0[j] = make_cplx<T>(v[0].x + a.x, v[0].y + a.y);
    u1[j] = make_cplx<T>(v[1].x + b.x, v[1].y + b.y);
  }
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const cplx_t<T> a = u0[k % 3], b = u1[k % 3], c = v[2];
    const int j1 = k, j2 = (2 * k) % 9;
    T re = fma(c.x, W::c(j2), fma(c.y, W::s(j2), a.x));
    re = fma(b.x, W::c(j1), fma(b.y, W::s(j1), re));
    T im = fma(c.y, W::c(j2), fma(-c.x, W::s(j2), a.y));
    im = fma(b.y, W::c(j1), fma(-b.x, W::s(j1), im));
    out(k, make_cplx<T>(re, im));
  }
}
// inverse 9 -> 5 at t = (a + 5) mod 9, out(a, X[t]) for a = 0..4
template <int n, typename T, class Out>
__device__ __forceinline__ void idft_9_to_5(const cplx_t<T>* v, Out out) {
  static_assert(2 * n - 1 == 9, "length-9 transform");
  using W = Tw<n, T>;
  cplx_t<T> vb[3][3];  // [b][j]
#pragma unroll
  for (int b = 0; b < 3; ++b) {
    const cplx_t<T> x0 = v[b], x1 = v[b + 3], x2 = v[b + 6];
    vb[b][0] = make_cplx<T>(x0.x + x1.x + x2.x, x0.y + x1.y + x2.y);
#pragma unroll
    for (int j = 1; j < 3; ++j) {
      const cplx_t<T> p = mul_wc<n, T>(x1, 3 * j), q = mul_wc<n, T>(x2, (6 * j) % 9);
      vb[b][j] = make_cplx<T>(x0.x + p.x + q.x, x0.y + p.y + q.y);
    }
  }
#pragma unroll
  for (int a = 0; a < 5; ++a) {
    const int t = (a + 5) % 9, j = t % 3;
    const cplx_t<T> y0 = vb[0][j], y1 = vb[1][j], y2 = vb[2][j];
    const int j1 = t, j2 = (2 * t) % 9;
    T re = fma(y2.x, W::c(j2), fma(-y2.y, W::s(j2), y0.x));
    re = fma(y1.x, W::c(j1), fma(-y1.y, W::s(j1), re));
    T im = fma(y2.y, W::c(j2), fma(y2.x, W::s(j2), y0.y));
    im = fma(y1.y, W::c(j1), fma(y1.x, W::s(j1), im));
    out(a, make_cplx<T>(re, im));
  }
}

__host__ __device__ inline constexpr int unif_jobs(int n) {
  return (2 * n - 1) * (n - 1) + (n - 1) + 1;
}
__host__ __device__ inline void unif_job(int n, int j, int* k2, int* k3) {
  const int m = 2 * n - 1, full = m * (n - 1);
  if (j < full) {
    *k2 = j / (n - 1);
    *k3 = j % (n - 1) + 1;
  } else {  // k3 = 0: k2 = 1..n-1 = (m-1)/2, then 0
    *k2 = j < full + n - 1 ? j - full + 1 : 0;
    *k3 = 0;
  }
}
// job of (k2, k3); k3 = 0: k2 < n
__host__ __device__ inline constexpr int unif_job_of(int n, int k2, int k3) {
  const int full = (2 * n - 1) * (n - 1);
  return k3 > 0 ? k2 * (n - 1) + k3 - 1 : k2 > 0 ? full + k2 - 1 : full + n - 1;
}
int unif_slots(int n) { return (unif_jobs(n) - 1) * (2 * n - 1) + n; }
int unif_slot_freq(int n, int slot) {
  const int m = 2 * n - 1;
  int k2, k3;
  unif_job(n, slot / m, &k2, &k3);
  return ((slot % m) * m + k2) * n + k3;
}

// Spectra of a level are stored frequency-major: X[(slot * ncells + cell) * C + col]
// (ncells = 8^level), so that one frequency plane of a level is contiguous.

// Both transforms run one unit = (cell, column) per lane: the U units of a CTA
// are neighbours in memory, so that a warp's loads and stores of a frequency
// cover consecutive words, and every thread computes whole 1-D transforms of
// its unit.  Two stages with one array between them in shared memory
// ([element][unit], conflict-free):
//   forward: thread (l1): the n^2 moments of its row; for each k3 the z
//            transform of the n lines l2 and the y transform of the results;
//            thread (j): the x transform of (k2, k3), straight to global memory;
//   inverse: thread (j): the x transform, straight from global memory; thread
//            (a1), of the largest orders several (qparts): for each k3 the y
//            transform, added into the n^2 outputs of its row by the z
//            transform; the outputs leave through shared memory in coalesced
//            rows.
// Spectra between the stages: the jobs (k2, k3) that are kept, n nj elements per
// unit.  Bound: HBM and the latency of the stages (shared memory admits two to
// four CTAs per SM).  Measured, 1M points at order 5, forward + inverse, against one
// cell per CTA with a column per lane: 1 column, float32 2.57 + 1.56 -> 0.38 +
// 0.34 ms (its stores covered 8 bytes of each frequency plane); 8 columns,
// float64 4.43 + 5.26 -> 2.75 + 3.31 ms, float32 with the split 3.32 + 3.10 -> 2.57 +
// 2.19 ms, and with four CTAs per SM instead of three (the conjugate elements not
// stored, the forward's moments under its spectra) 2.27 + 1.99 ms.
template <int n, typename T>
struct FftCfg {
  static constexpr int m = 2 * n - 1, n3 = n * n * n, nj = unif_jobs(n), nym = n * nj;
  static constexpr int unit = (n3 + 2 * nym) * (int)sizeof(T);  // bytes per unit (forward)
  static constexpr int U = unit * 32 <= 110 * 1024   ? 32
                           : unit * 16 <= 110 * 1024 ? 16
                           : unit * 8 <= 226 * 1024  ? 8
                                                     : 4;
  // the rows of the k3 loop: one thread per (row, part of k3) where one per row leaves warps idle
  static constexpr int parts = n * U < 128 ? 2 : 1;
  static constexpr int threads = n * U * parts <= 128 ? 128 : (n * U * parts + 31) / 32 * 32;
  // forward: the moments take the place of the spectra until every thread has
  // its row in registers
  static constexpr bool alias = parts == 1 && sizeof(T) == 4 && n <= 5;
  static constexpr size_t smem_y = 2 * sizeof(T) * (size_t)nym * U;
  static constexpr size_t smem_s = sizeof(T) * (size_t)n3 * (U + 1);
  static constexpr size_t smem_fwd = alias ? (smem_y > smem_s ? smem_y : smem_s) : smem_y + smem_s + 16;
  static constexpr size_t out_bytes = sizeof(T) * (size_t)U * (n3 | 1);
  // inverse: plain levels of 32 units per CTA, four of which would fit an SM (order
  // 4 in float64, 5 in float32), ask for so much that three do: 1M points, 1 column,
  // order 5, float32 0.356 -> 0.334 ms; 800,000 points, 3 columns, order 4, float64
  // 0.702 -> 0.653 ms.  The other plans lose by it (order 6, 120,000 points, 3
  // columns: float64 0.369 -> 0.494, float32 0.227 -> 0.277 ms) or do not notice, and
  // the split levels gain from four (2.20 -> 1.99 ms).
  static constexpr size_t smem_inv(bool split) {
    constexpr size_t sm = 228 * 1024, cta = smem_y + 1024;  // (1 KB is the system's)
    const bool three = !split && U == 32 && 4 * cta <= sm && 5 * cta > sm;
    const size_t b = three ? (size_t)60 * 1024 : smem_y;
    return b > out_bytes ? b : out_bytes;
  }
  static constexpr int unroll = n <= 6 ? n : 1;  // the k3 loops: larger orders keep the code small
  // inverse: threads of a row of outputs.  From order 8 (float32 9) on a thread's n^2
  // outputs and the m inputs of a transform do not fit its registers (spills of
  // up to 1 KB), and a thread per row leaves half of the warps idle: each then
  // takes n / qparts of the outputs a2 and reads its inputs from shared memory as it
  // uses them.  20,000 points on 4 levels, inverse of all levels, 1 column: float64,
  // orders 8, 9, 10: 0.188, 0.466, 0.698 -> 0.101, 0.186, 0.310 ms (2, 3, 2 parts:
  // 0.127, 0.186, 0.341); float32, orders 9, 10: 0.187, 0.264 -> 0.101, 0.184 ms.
  static constexpr int qparts = sizeof(T) == 8 ? (n == 8 ? 4 : n == 9 ? 3 : n == 10 ? 5 : 1)
                                               : (n == 9 ? 3 : n == 10 ? 2 : 1);
  static_assert(n % qparts == 0, "equal parts");
  static constexpr int threads_inv =
      n * U * qparts <= threads ? threads : (n * U * qparts + 31) / 32 * 32;
};

// The z and y transforms of row l1 of one unit, for k3 = K0, K0 + STEP, ...
template <int n, typename T, int U, int K0, int STEP, int PITCH>
__device__ __forceinline__ void fwd_row(const T* __restrict__ s, cplx_t<T>* __restrict__ y) {
  using W = Tw<n, T>;
  constexpr int m = 2 * n - 1;
  using Cfg = FftCfg<n, T>;
#pragma unroll Cfg::unroll
  for (int k3 = K0; k3 < n; k3 += STEP) {
    cplx_t<T> v[n];
#pragma unroll
    for (int l2 = 0; l2 < n; ++l2) {
      T re = 0, im = 0;
#pragma unroll
      for (int l = 0; l < n; ++l) {
        const T x = s[(l2 * n + l) * PITCH];
        re = fma(x, W::c((k3 * l) % m), re);
        im = fma(-x, W::s((k3 * l) % m), im);
      }
      v[l2] = make_cplx<T>(re, im);
    }
    const int kend = k3 == 0 ? n : m;  // (k2 >= n, 0) are not kept
    if constexpr (m == 9) {
      dft_5_to_9<n, T>(v, [&](int k, cplx_t<T> r) {
        if (k < kend) y[unif_job_of(n, k, k3) * U] = r;
      });
    } else {
#pragma unroll
      for (int k = 0; k < m; ++k) {
        if (k >= kend) break;
        T re = 0, im = 0;
#pragma unroll
        for (int l = 0; l < n; ++l) {
          const T c = W::c((k * l) % m), sn = W::s((k * l) % m);
          re = fma(v[l].x, c, fma(v[l].y, sn, re));
          im = fma(v[l].y, c, fma(-v[l].x, sn, im));
        }
        y[unif_job_of(n, k, k3) * U] = make_cplx<T>(re, im);
      }
    }
  }
}

// w = e^{-2 pi i / m}; (a + ib) w^j = (a c + b s) + i (b c - a s).
// Units of a CTA: U consecutive (cell, column) pairs of the nonempty source
// cells; spectra to X[(slot ncells + cell) C + column].  SPLIT (tensor-core
// levels, one group of 8 columns from c0): units are U / 4 (parent, column)
// rows x 4 children of one half of the children; spectra scaled by 2^s with s
// from the column's bound, split into F16 hi and lo and stored in the layout
// of the tensor-core MAC (UnifPlanes); zeros for empty cells.
template <int n, typename T, bool SPLIT>
__global__ void __launch_bounds__(FftCfg<n, T>::threads)
    k_fft_fwd(const FftFwdArgs<T> a) {
  using C2 = cplx_t<T>;
  using W = Tw<n, T>;
  using Cfg = FftCfg<n, T>;
  constexpr int m = Cfg::m, n2 = n * n, n3 = Cfg::n3, U = Cfg::U, nj = unif_jobs(n);
  extern __shared__ __align__(16) unsigned char smraw[];
  C2* Y = reinterpret_cast<C2*>(smraw);                        // [l1][job][U]
  T* S = reinterpret_cast<T*>(Cfg::alias ? Y : Y + (size_t)Cfg::nym * U);  // [n^3][U + 1]
  __shared__ int64_t s_src[U];                                 // unit: its moments, or -1
  const int tid = threadIdx.x, u = tid % U, job0 = tid / U;
  constexpr int JS = Cfg::threads / U;
  int64_t dst = 0;  // this thread's unit: first output
  bool has = false, inside = true;
  int col = 0;  // SPLIT: its column of the group
  if constexpr (SPLIT) {
    // group: kplane = blockIdx.x & 1, rows (blockIdx.x >> 1) U / 4 ...
    const int kp = blockIdx.x & 1, e = u & 3;
    const int64_t row = (int64_t)(blockIdx.x >> 1) * (U / 4) + (u >> 2);
    const int S_ = a.side, c = (int)(row % 8);
    const int z = (int)(row / 8 % S_), y = (int)(row / 8 / S_ % S_), x = (int)(row / 8 / S_ / S_);
    inside = x < S_;
    col = c;
    if (inside) {
      const int64_t cell = 8 * (int64_t)morton_encode(x, y, z) + 4 * kp + e;
      has = a.occ[cell] != 0;
      dst = UnifPlanes::row_byte(S_, x, kp, y, z, c) + 4 * e;
      if (job0 == 0) s_src[u] = has ? (cell * a.C + a.c0 + c) * n3 : -1;
    } else if (job0 == 0) {
      s_src[u] = -1;
    }
  } else {
    const int64_t g = (int64_t)blockIdx.x * U + u;
    has = g < a.nunits;
    if (has) {
      const int64_t cell = a.cells[g / a.C];
      dst = cell * a.C + g % a.C;
    }
    if (job0 == 0) s_src[u] = has ? dst * n3 : -1;
  }
  const bool any = __syncthreads_or(has);
  if (any) {
    units_in<U, n3, Cfg::threads, U + 1>(S, a.S, [&](int v) { return s_src[v]; });
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads();
    if constexpr (Cfg::alias) {
      T row[n2];
      if (job0 < n) {
        const T* s = S + job0 * n2 * (U + 1) + u;
#pragma unroll
        for (int l = 0; l < n2; ++l) row[l] = s[l * (U + 1)];
      }
      __syncthreads();
      if (job0 < n) fwd_row<n, T, U, 0, 1, 1>(row, Y + job0 * nj * U + u);
    } else {
      for (int job = job0; job < n * Cfg::parts; job += JS) {
        const int l1 = job % n;
        const T* s = S + l1 * n2 * (U + 1) + u;
        C2* y = Y + l1 * nj * U + u;
        if constexpr (Cfg::parts == 1)
          fwd_row<n, T, U, 0, 1, U + 1>(s, y);
        else if (job < n)
          fwd_row<n, T, U, 0, 2, U + 1>(s, y);
        else
          fwd_row<n, T, U, 1, 2, U + 1>(s, y);
      }
    }
    __syncthreads();
  }
  float sc = 1.f;
  if constexpr (SPLIT) {
    if (!inside) return;
    sc = exp2i(unif_scale_exp(a.amax[col]));
  } else {
    if (!has) return;
  }
  for (int j = job0; j < nj; j += JS) {
    const int kend = j == nj - 1 ? n : m;  // (0, 0): the rest are conjugates
    C2 v[n];
    if (any) {
      const C2* y = Y + j * U + u;
#pragma unroll
      for (int l = 0; l < n; ++l) v[l] = y[l * nj * U];
    } else {
#pragma unroll
      for (int l = 0; l < n; ++l) v[l] = make_cplx<T>(T(0), T(0));
    }
    auto put = [&](int k, C2 r) {
      if (k >= kend) return;
      if constexpr (SPLIT) {
        const float x0 = r.x * sc, x1 = r.y * sc;
        const __half2 h = __floats2half2_rn(x0, x1);
        const float2 hf = __half22float2(h);
        const __half2 l = __floats2half2_rn(x0 - hf.x, x1 - hf.y);
        unsigned char* p = reinterpret_cast<unsigned char*>(a.X) + (j * m + k) * a.slot_stride + dst;
        *reinterpret_cast<__half2*>(p) = h;
        *reinterpret_cast<__half2*>(p + a.lo_off) = l;
      } else {
        a.X[(j * m + k) * a.slot_stride + dst] = r;
      }
    };
    if constexpr (m == 9) {
      dft_5_to_9<n, T>(v, put);
    } else {
#pragma unroll
      for (int k = 0; k < m; ++k) {
        T re = 0, im = 0;
#pragma unroll
        for (int l = 0; l < n; ++l) {
          const T c = W::c((k * l) % m), s = W::s((k * l) % m);
          re = fma(v[l].x, c, fma(v[l].y, s, re));
          im = fma(v[l].y, c, fma(-v[l].x, s, im));
        }
        put(k, make_cplx<T>(re, im));
      }
    }
  }
}

// y and z of outputs a2 = Q0 .. Q0 + QN - 1 of one row a1 of one unit (see
// k_fft_inv), the inputs read from shared memory as they are used.
template <int n, typename T, int U, int Q0, int QN>
__device__ __forceinline__ void inv_row_part(const cplx_t<T>* __restrict__ g, T (&acc)[QN][n]) {
  using W = Tw<n, T>;
  constexpr int m = 2 * n - 1;
#pragma unroll 1
  for (int k3 = 0; k3 < n; ++k3) {
    T re[QN], im[QN];
#pragma unroll
    for (int q = 0; q < QN; ++q) re[q] = im[q] = 0;
#pragma unroll
    for (int k = 0; k < m; ++k) {
      const bool mirror = k3 == 0 && k >= n;  // G(-k2, 0) = conj G(k2, 0)
      cplx_t<T> v = g[unif_job_of(n, mirror ? m - k : k, k3) * U];
      if (mirror) v.y = -v.y;
#pragma unroll
      for (int q = 0; q < QN; ++q) {
        const int t = (Q0 + q + n) % m;
        const T c = W::c((k * t) % m), s = W::s((k * t) % m);
        re[q] = fma(v.x, c, fma(-v.y, s, re[q]));
        im[q] = fma(v.y, c, fma(v.x, s, im[q]));
      }
    }
#pragma unroll
    for (int q = 0; q < QN; ++q)
#pragma unroll
      for (int a3 = 0; a3 < n; ++a3) {
        const int t = (a3 + n) % m;
        if (k3 == 0)
          acc[q][a3] = re[q];
        else
          acc[q][a3] = fma(T(2), fma(re[q], W::c((k3 * t) % m), -im[q] * W::s((k3 * t) % m)),
                           acc[q][a3]);
      }
  }
}

// F = scale * IDFT(Y)/P at grid positions (a + n) mod m;
// (a + ib) e^{+2 pi i j / m} = (a c - b s) + i (b c + a s).
// Units: U consecutive (cell, column) pairs of the nonempty target cells,
// Y[(slot ncells + cell) C + column]; SPLIT: U consecutive (parent, column)
// rows of one child, Y as the tensor-core MAC writes it (UnifPlanes).
template <int n, typename T, bool SPLIT>
__global__ void __launch_bounds__(FftCfg<n, T>::threads_inv)
    k_fft_inv(const FftInvArgs<T> a) {
  using C2 = cplx_t<T>;
  using W = Tw<n, T>;
  using Cfg = FftCfg<n, T>;
  constexpr int m = Cfg::m, n2 = n * n, n3 = Cfg::n3, U = Cfg::U, nj = unif_jobs(n);
  constexpr int OP = n3 | 1;  // pitch of a unit's outputs
  extern __shared__ __align__(16) unsigned char smraw[];
  C2* G = reinterpret_cast<C2*>(smraw);  // [a1][job][U]
  T* O = reinterpret_cast<T*>(smraw);    // [U][OP], after G
  __shared__ int64_t s_dst[U];           // unit: its locals, or -1
  const int tid = threadIdx.x, u = tid % U, job0 = tid / U;
  constexpr int JS = Cfg::threads_inv / U;
  int64_t src = 0;
  bool has;
  if constexpr (SPLIT) {
    const int t = blockIdx.x & 7, S_ = a.side;
    const int64_t row = (int64_t)(blockIdx.x >> 3) * U + u;
    const int c = (int)(row % 8);
    const int z = (int)(row / 8 % S_), y = (int)(row / 8 / S_ % S_), x = (int)(row / 8 / S_ / S_);
    has = x < S_;
    int64_t cell = 0;
    if (has) {
      cell = 8 * (int64_t)morton_encode(x, y, z) + t;
      has = a.occ[cell] != 0;
      src = UnifPlanes::out_index(S_, x, t, y, z, c);
    }
    if (job0 == 0) s_dst[u] = has ? (cell * a.C + a.c0 + c) * n3 : -1;
  } else {
    const int64_t g = (int64_t)blockIdx.x * U + u;
    has = g < a.nunits;
    if (has) src = (int64_t)a.cells[g / a.C] * a.C + g % a.C;
    if (job0 == 0) s_dst[u] = has ? src * n3 : -1;
  }
  if (!__syncthreads_or(has)) return;
  if (has) {
    // x: G[a1][k2][k3] = sum_k1 Y[k1][k2][k3] e^{+2 pi i k1 t1 / m}
    for (int j = job0; j < nj; j += JS) {
      const C2* y = a.Y + (int64_t)j * m * a.slot_stride + src;
      C2 v[m];
#pragma unroll
      for (int k = 0; k < m; ++k) {
        const bool mirror = j == nj - 1 && k >= n;  // Y(-k1, 0, 0) = conj Y(k1, 0, 0)
        v[k] = y[(mirror ? m - k : k) * a.slot_stride];
        if (mirror) v[k].y = -v[k].y;
      }
      C2* g = G + j * U + u;
      if constexpr (m == 9) {
        idft_9_to_5<n, T>(v, [&](int q, C2 r) { g[q * nj * U] = r; });
      } else {
#pragma unroll
        for (int q = 0; q < n; ++q) {
          const int t = (q + n) % m;
          T re = 0, im = 0;
#pragma unroll
          for (int k = 0; k < m; ++k) {
            const T c = W::c((k * t) % m), s = W::s((k * t) % m);
            re = fma(v[k].x, c, fma(-v[k].y, s, re));
            im = fma(v[k].y, c, fma(v[k].x, s, im));
          }
          g[q * nj * U] = make_cplx<T>(re, im);
        }
      }
    }
  }
  __syncthreads();
  // y and z of row a1: H[a2][k3] = sum_k2 G[a1][k2][k3] e^{+2 pi i k2 t2 / m},
  // out = Re H[..][0] + 2 sum_{k3>=1} Re(H[..][k3] e^{+2 pi i k3 t3 / m})
  constexpr int QP = Cfg::qparts, QN = n / QP;
  T acc[QN][n];
  const bool row = job0 < n * QP && has;
  const int a1 = job0 % n, part = job0 / n;
  const C2* grow = G + a1 * nj * U + u;
  if constexpr (QP > 1) {
    if (row) {
      if (part == 0) inv_row_part<n, T, U, 0, QN>(grow, acc);
      if (part == 1) inv_row_part<n, T, U, QN, QN>(grow, acc);
      if constexpr (QP > 2)
        if (part == 2) inv_row_part<n, T, U, 2 * QN, QN>(grow, acc);
      if constexpr (QP > 3)
        if (part == 3) inv_row_part<n, T, U, 3 * QN, QN>(grow, acc);
      if constexpr (QP > 4)
        if (part == 4) inv_row_part<n, T, U, 4 * QN, QN>(grow, acc);
    }
  } else if (row) {
    const C2* g = grow;
#pragma unroll Cfg::unroll
    for (int k3 = 0; k3 < n; ++k3) {
      C2 v[m];
#pragma unroll
      for (int k = 0; k < m; ++k) {
        const bool mirror = k3 == 0 && k >= n;  // G(-k2, 0) = conj G(k2, 0)
        v[k] = g[unif_job_of(n, mirror ? m - k : k, k3) * U];
        if (mirror) v[k].y = -v[k].y;
      }
      auto add = [&](int q, C2 h) {
#pragma unroll
        for (int a3 = 0; a3 < n; ++a3) {
          const int t = (a3 + n) % m;
          if (k3 == 0)
            acc[q][a3] = h.x;
          else
            acc[q][a3] = fma(T(2), fma(h.x, W::c((k3 * t) % m), -h.y * W::s((k3 * t) % m)),
                             acc[q][a3]);
        }
      };
      if constexpr (m == 9) {
        idft_9_to_5<n, T>(v, add);
      } else {
#pragma unroll
        for (int q = 0; q < n; ++q) {
          const int t = (q + n) % m;
          T re = 0, im = 0;
#pragma unroll
          for (int k = 0; k < m; ++k) {
            const T c = W::c((k * t) % m), s = W::s((k * t) % m);
            re = fma(v[k].x, c, fma(-v[k].y, s, re));
            im = fma(v[k].y, c, fma(v[k].x, s, im));
          }
          add(q, make_cplx<T>(re, im));
        }
      }
    }
  }
  __syncthreads();
  if (row) {
    T* o = O + u * OP + a1 * n2 + part * QN * n;
#pragma unroll
    for (int q = 0; q < QN; ++q)
#pragma unroll
      for (int a3 = 0; a3 < n; ++a3) o[q * n + a3] = a.scale * (acc[q][a3] * a.invP);
  }
  __syncthreads();
  // (a warp per unit, lanes over its row)
  for (int v = tid >> 5; v < U; v += Cfg::threads_inv / 32) {
    const int64_t o = s_dst[v];
    if (o < 0) continue;
#pragma unroll
    for (int r = 0; r < (n3 + 31) / 32; ++r) {
      const int l = (tid & 31) + 32 * r;
      if (l < n3) a.F[o + l] = O[v * OP + l];
    }
  }
}

// ----------------------------------------------------------------- MAC
// y_k(P)[t] = sum over parent offsets D in {-1, 0, 1}^3 and children s of
// E_k[2 D + s - t] x_k(P + D)[s] (E = 0 for near offsets; D = 0 has near ones
// only).  For one D this is an 8 x 8 block that is Toeplitz in each of the
// three child coordinates, so it is taken with three products per coordinate
// instead of four (Karatsuba):
//   y0 = e0 x0 + e+ x1 = e0 (x0 + x1) + (e+ - e0) x1
//   y1 = e- x0 + e0 x1 = e0 (x0 + x1) + (e- - e0) x0
// 27 complex products per parent pair instead of 56 (64 less the near ones);
// the 27 products of a target parent are summed over D before the (linear)
// output step.  Counted per target parent and frequency: 26 x (108
// multiply-adds + 38 additions) against 6048 multiply-adds.
//
// A thread owns (target parent, slot, column) and its 27 complex sums; a CTA
// owns a block of PX x PY x PZ target parents, KC slots and CG columns.  The
// source parents of the block and its one-parent halo are staged in shared
// memory as [child][parent][slot][column], so that the threads of a warp,
// which run over column, slot and z, read consecutive words; the 26 x 27
// coefficients of each slot lie behind them and are read by broadcast.  The
// loop over D is not unrolled (every D has the same body).  The slot varies
// slowest in the grid, so resident CTAs share a few frequency planes in L2.
//
// Bound: the FP64 pipe and the shared-memory reads beside it (float32: issue
// slots and shared-memory reads).  Measured, M2L of one matvec at order 5
// against the direct sum of 189 products per child and m m n frequencies:
// 1M points, 8 columns, float64 59.7 -> 47.3 ms; 250,000 points, 1 column,
// float64 1.66 -> 0.84 ms; 1M points, 1 column, float32 6.45 -> 3.96 ms;
// 200,000 points, 3 columns, float32 2.79 -> 1.61 ms.  The distance of the
// float32 pass from float64 stays where it was (2.3e-7 to 5.2e-7 over orders 3
// to 5 and 1 to 3 columns; before, 2.9e-7 to 5.2e-7).
//
// Per level, halo[b * STRIDE + r] holds for the region parents of block b their
// Morton index, then the occupancy of their 8 children (0 outside the
// domain), then the same of the block's target parents.
template <int PX, int PY, int PZ>
struct MacGeom {
  static constexpr int RX = PX + 2, RY = PY + 2, RZ = PZ + 2;
  static constexpr int RP = RX * RY * RZ;  // region parents
  static constexpr int NP = PX * PY * PZ;  // target parents
  static constexpr int STRIDE = 2 * RP + 2 * NP;
};

__device__ __forceinline__ int parent_mask(const int* __restrict__ start, int64_t p, int span) {
  int m = 0, lo = start[8 * p * span];
  for (int c = 0; c < 8; ++c) {
    const int hi = start[(8 * p + c + 1) * span];
    m |= (hi > lo ? 1 : 0) << c;
    lo = hi;
  }
  return m;
}

template <int PX, int PY, int PZ>
__global__ void k_halo_tables(const int* __restrict__ sstart, const int* __restrict__ tstart,
                              int span, int S, int nby, int nbz, int* __restrict__ halo) {
  using G = MacGeom<PX, PY, PZ>;
  const int b = blockIdx.x;
  const int x0 = PX * (b / (nby * nbz)), y0 = PY * ((b / nbz) % nby), z0 = PZ * (b % nbz);
  int* h = halo + (int64_t)b * G::STRIDE;
  for (int r = threadIdx.x; r < G::RP + G::NP; r += blockDim.x) {
    const bool src = r < G::RP;
    const int q = src ? r : r - G::RP;
    const int x = src ? x0 - 1 + q / (G::RY * G::RZ) : x0 + q / (PY * PZ);
    const int y = src ? y0 - 1 + (q / G::RZ) % G::RY : y0 + (q / PZ) % PY;
    const int z = src ? z0 - 1 + q % G::RZ : z0 + q % PZ;
    int p = 0, m = 0;
    if (x >= 0 && y >= 0 && z >= 0 && x < S && y < S && z < S) {
      p = (int)morton_encode(x, y, z);
      m = parent_mask(src ? sstart : tstart, p, span);
    }
    int* d = src ? h + q : h + 2 * G::RP + q;
    d[0] = p;
    d[src ? G::RP : G::NP] = m;
  }
}

template <int PX, int PY, int PZ, int KC, int CG, typename T>
struct MacSmem {
  using G = MacGeom<PX, PY, PZ>;
  static constexpr int Q = KC * CG;
  // stride of a child's plane: shifted against the others, so that the copies
  // of several children of one parent reach different banks
  static constexpr int CS = G::RP * Q + (CG > 4 ? CG : 4);
  static constexpr size_t bytes =
      sizeof(cplx_t<T>) * (8 * CS + KC * kKaraD * kKaraJ) + sizeof(int) * G::STRIDE;
};

template <int PX, int PY, int PZ, int KC, int CG, typename T>
__global__ void __launch_bounds__(PX* PY* PZ* KC* CG)
    k_m2l_unif_mac(const cplx_t<T>* __restrict__ X_l, cplx_t<T>* __restrict__ Y_l,
                   const cplx_t<T>* __restrict__ op,  // [slot][26][27] of this level
                   const int* __restrict__ halo, int64_t ncells, int C, int c0, int nk) {
  using G = MacGeom<PX, PY, PZ>;
  using SM = MacSmem<PX, PY, PZ, KC, CG, T>;
  using C2 = cplx_t<T>;
  constexpr int NT = G::NP * KC * CG, Q = KC * CG, CS = SM::CS, NE = kKaraD * kKaraJ;
  extern __shared__ __align__(16) unsigned char smraw[];
  C2* reg = reinterpret_cast<C2*>(smraw);  // [child][region parent][slot][col]
  C2* sop = reg + 8 * CS;                  // [slot][26][27]
  int* s_par = (int*)(sop + KC * NE);      // region parents
  int* s_msk = s_par + G::RP;              // their children with sources
  int* s_tgt = s_msk + G::RP;              // target parents, then their children with targets
  const int tid = threadIdx.x;
  const int cc = tid % CG, kc = (tid / CG) % KC, p = tid / Q;
  const int px = p / (PY * PZ), py = (p / PZ) % PY, pz = p % PZ;
  const int* hb = halo + (int64_t)blockIdx.x * G::STRIDE;
  int mine = 0;
  for (int r = tid; r < G::STRIDE; r += NT) {
    const int v = hb[r];
    s_par[r] = v;
    if (r >= 2 * G::RP + G::NP) mine |= v;
  }
  if (!__syncthreads_or(mine)) return;  // no target in the block
  const int k0 = blockIdx.y * KC;
  // all copies in flight at once; empty or out-of-domain cells are zero-filled.
  // Order (column, child, slot, parent): runs of 8 CG values are contiguous.
  for (int i = tid; i < G::RP * 8 * Q; i += NT) {
    const int c = i % CG, ch = (i / CG) % 8, kk = (i / (8 * CG)) % KC, r = i / (8 * Q);
    const bool ok = ((s_msk[r] >> ch) & 1) && k0 + kk < nk;
    const C2* g = ok ? &X_l[((int64_t)(k0 + kk) * ncells + 8 * (int64_t)s_par[r] + ch) * C + c0 + c]
                     : X_l;
    cp_async_cplx(&reg[ch * CS + r * Q + kk * CG + c], g, ok);
  }
  for (int i = tid; i < KC * NE; i += NT) {
    const bool ok = k0 + i / NE < nk;
    cp_async_cplx(&sop[i], ok ? &op[(int64_t)k0 * NE + i] : op, ok);
  }
  cp_async_commit();
  cp_async_wait_all();
  __syncthreads();
  C2 acc[kKaraJ];
#pragma unroll
  for (int j = 0; j < kKaraJ; ++j) acc[j] = make_cplx<T>(T(0), T(0));
  const C2* e = sop + kc * NE;
  auto add = [](C2 a, C2 b) { return make_cplx<T>(a.x + b.x, a.y + b.y); };
#pragma unroll 1
  for (int dx = 0; dx < 3; ++dx)
#pragma unroll 1
    for (int dy = 0; dy < 3; ++dy)
#pragma unroll 1
      for (int dz = 0; dz < 3; ++dz) {
        if (dx == 1 && dy == 1 && dz == 1) continue;
        const int r = ((px + dx) * G::RY + py + dy) * G::RZ + pz + dz;
        if (s_msk[r]) {
          const C2* xr = reg + r * Q + kc * CG + cc;
          C2 x[8];
#pragma unroll
          for (int ch = 0; ch < 8; ++ch) x[ch] = xr[ch * CS];
          // j = 9 jx + 3 jy + jz, each 0: x0 + x1, 1: x1, 2: x0
#pragma unroll
          for (int jz = 0; jz < 3; ++jz) {
            C2 u[4];  // (bx, by)
#pragma unroll
            for (int q = 0; q < 4; ++q)
              u[q] = jz == 0 ? add(x[2 * q], x[2 * q + 1]) : x[2 * q + (jz == 1 ? 1 : 0)];
#pragma unroll
            for (int jy = 0; jy < 3; ++jy) {
              C2 v[2];  // bx
#pragma unroll
              for (int q = 0; q < 2; ++q)
                v[q] = jy == 0 ? add(u[2 * q], u[2 * q + 1]) : u[2 * q + (jy == 1 ? 1 : 0)];
#pragma unroll
              for (int jx = 0; jx < 3; ++jx) {
                const C2 w = jx == 0 ? add(v[0], v[1]) : v[jx == 1 ? 1 : 0];
                const int j = 9 * jx + 3 * jy + jz;
                const C2 a = e[j];
                acc[j].x = fma(a.x, w.x, acc[j].x);
                acc[j].y = fma(a.x, w.y, acc[j].y);
                acc[j].x = fma(-a.y, w.y, acc[j].x);
                acc[j].y = fma(a.y, w.x, acc[j].y);
              }
            }
          }
        }
        e += kKaraJ;
      }
  if (k0 + kc >= nk) return;
  const int tm = s_tgt[G::NP + p];
  const int64_t tp = 8 * (int64_t)s_tgt[p];
  C2* out = Y_l + ((int64_t)(k0 + kc) * ncells + tp) * C + c0 + cc;
  // y0 = P + Q1, y1 = P + Q0 per coordinate
#pragma unroll
  for (int t = 0; t < 8; ++t) {
    const int jx = 9 * (1 + ((t >> 2) & 1)), jy = 3 * (1 + ((t >> 1) & 1)), jz = 1 + (t & 1);
    const C2 y = add(add(add(acc[0], acc[jz]), add(acc[jy], acc[jy + jz])),
                     add(add(acc[jx], acc[jx + jz]), add(acc[jx + jy], acc[jx + jy + jz])));
    if ((tm >> t) & 1) out[(int64_t)t * C] = y;
  }
}

// The coefficients [level][slot][26][27] from the spectra op[level][k][343]
// (lex-indexed offsets, inner 27 zero): per coordinate the differences above.
std::vector<double> unif_kara_operators(int n, const std::vector<double>& op, int nlev) {
  const int nk = unif_slots(n), nfull = (2 * n - 1) * (2 * n - 1) * n;
  std::vector<double> out((size_t)nlev * nk * kKaraD * kKaraJ * 2);
  parallel_for((int64_t)nlev * nk, [&](int64_t b0, int64_t b1) {
    for (int64_t b = b0; b < b1; ++b) {
      const double* E = &op[(size_t)(b / nk * nfull + unif_slot_freq(n, (int)(b % nk))) * 343 * 2];
      double* o = &out[(size_t)b * kKaraD * kKaraJ * 2];
      for (int d = 0; d < 27; ++d) {
        if (d == 13) continue;
        const int c[3] = {2 * (d / 9 - 1), 2 * (d / 3 % 3 - 1), 2 * (d % 3 - 1)};
        for (int j = 0; j < kKaraJ; ++j, o += 2) {
          const int jd[3] = {j / 9, j / 3 % 3, j % 3};
          o[0] = o[1] = 0.0;
          for (int q = 0; q < 8; ++q) {  // bit i: the subtracted term of coordinate i
            int lex = 0, sign = 1;
            bool used = true;
            for (int i = 0; i < 3; ++i) {
              const int sub = (q >> i) & 1;
              int off = c[i];
              if (jd[i] == 0)
                used &= !sub;
              else if (sub)
                sign = -sign;
              else
                off += jd[i] == 1 ? 1 : -1;
              lex = 7 * lex + off + 3;
            }
            if (!used) continue;
            o[0] += sign * E[2 * lex];
            o[1] += sign * E[2 * lex + 1];
          }
        }
      }
    }
  });
  return out;
}

// ints of the halo tables of a level with S parents per side
int64_t unif_halo_ints(int S) {
  const int64_t b4 = (S + 3) / 4, b2 = (S + 1) / 2;
  const int64_t a = b4 * b4 * b4 * MacGeom<4, 4, 4>::STRIDE, b = b4 * b4 * b2 * MacGeom<4, 4, 2>::STRIDE,
                c = b4 * b2 * b2 * MacGeom<4, 2, 2>::STRIDE;
  return std::max(a, std::max(b, c));
}

template <typename T>
struct MacLevel {
  const cplx_t<T>* X;
  cplx_t<T>* Y;
  const cplx_t<T>* op;
  int* halo;
  const int* sstart;
  const int* tstart;
  int span, lev, C, nk;
  cudaStream_t st;
  int last = 0;  // geometry that the halo tables hold

  template <int PX, int PY, int PZ, int KC, int CG>
  int run(int c0) {
    using G = MacGeom<PX, PY, PZ>;
    const int S = 1 << (lev - 1);
    const int nbx = (S + PX - 1) / PX, nby = (S + PY - 1) / PY, nbz = (S + PZ - 1) / PZ;
    const unsigned nblk = (unsigned)(nbx * nby * nbz);
    if (last != G::STRIDE) {
      k_halo_tables<PX, PY, PZ><<<nblk, 128, 0, st>>>(sstart, tstart, span, S, nby, nbz, halo);
      PB_LAUNCH("halo_tables");
      last = G::STRIDE;
    }
    auto kern = k_m2l_unif_mac<PX, PY, PZ, KC, CG, T>;
    constexpr size_t smem = MacSmem<PX, PY, PZ, KC, CG, T>::bytes;
    PB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<dim3(nblk, (unsigned)((nk + KC - 1) / KC)), G::NP * KC * CG, smem, st>>>(
        X, Y, op, halo, cells_at(lev), C, c0, nk);
    PB_LAUNCH("m2l_unif_mac");
    return PBBFMM_OK;
  }

  // Columns in groups of 8 and one smaller group, each an instance of its own
  // (no lanes on absent columns).  Blocks: the fewer the columns, the more
  // parents, so that a CTA has 4 to 10 warps and two or more CTAs share an SM.
  int columns() {
    constexpr bool f64 = sizeof(T) == 8;
    for (int c0 = 0; c0 < C; c0 += 8) {
      int rc;
      switch (std::min(8, C - c0)) {
        case 1: rc = run<4, 4, 4, f64 ? 2 : 4, 1>(c0); break;
        case 2: rc = run<4, 4, 4, f64 ? 1 : 2, 2>(c0); break;
        case 3: rc = run<4, 4, 4, 1, 3>(c0); break;
        case 4: rc = run<4, 4, f64 ? 2 : 4, 1, 4>(c0); break;
        case 5: rc = run<4, f64 ? 2 : 4, 2, 1, 5>(c0); break;
        case 6: rc = run<4, f64 ? 2 : 4, 2, 1, 6>(c0); break;
        case 7: rc = run<4, f64 ? 2 : 4, 2, 1, 7>(c0); break;
        default: rc = run<4, f64 ? 2 : 4, 2, 1, 8>(c0); break;
      }
      if (rc) return rc;
    }
    return PBBFMM_OK;
  }
};

template <typename T, bool SPLIT>
struct FftFwdLaunch {
  FftFwdArgs<T> a;
  int64_t groups4;  // SPLIT: (parent, column) rows of the level
  cudaStream_t st;
  template <int N>
  int run() {
    using Cfg = FftCfg<N, T>;
    const int64_t grid = SPLIT ? 2 * ((groups4 + Cfg::U / 4 - 1) / (Cfg::U / 4))
                               : (a.nunits + Cfg::U - 1) / Cfg::U;
    auto kern = k_fft_fwd<N, T, SPLIT>;
    PB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)Cfg::smem_fwd));
    kern<<<(unsigned)grid, Cfg::threads, Cfg::smem_fwd, st>>>(a);
    PB_LAUNCH("fft_fwd");
    return PBBFMM_OK;
  }
};

template <typename T, bool SPLIT>
struct FftInvLaunch {
  FftInvArgs<T> a;
  int64_t rows;  // SPLIT: (parent, column) rows of the level
  cudaStream_t st;
  template <int N>
  int run() {
    using Cfg = FftCfg<N, T>;
    const int64_t grid = SPLIT ? 8 * ((rows + Cfg::U - 1) / Cfg::U) : (a.nunits + Cfg::U - 1) / Cfg::U;
    auto kern = k_fft_inv<N, T, SPLIT>;
    PB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)Cfg::smem_inv(SPLIT)));
    kern<<<(unsigned)grid, Cfg::threads_inv, Cfg::smem_inv(SPLIT), st>>>(a);
    PB_LAUNCH("fft_inv");
    return PBBFMM_OK;
  }
};

// Largest sum over a cell and column of |moments|, per column of the group
// (float bits): a bound on |re| and |im| of its spectra.  Warps over cells, lanes
// over the moments, the 8 columns' loads in flight together; the 8 sums meet in
// 9 shuffles, lane l ending with column l / 4.  Bound: HBM (one read of the
// moments).  Against a column at a time with 5 shuffles each, 1M points, 8 columns:
// forward phase 2.27 -> 2.18 ms.
__global__ void k_moment_bound(const int* __restrict__ cells, int ncl, const float* __restrict__ S,
                               int C, int c0, int n3, uint32_t* __restrict__ amax) {
  const int lane = threadIdx.x & 31, nw = gridDim.x * (blockDim.x >> 5);
  float mx = 0.f;
  for (int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < ncl; i += nw) {
    const float* s = S + ((int64_t)cells[i] * C + c0) * n3;
    float v[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) v[c] = 0.f;
#pragma unroll 4
    for (int l = lane; l < n3; l += 32) {
#pragma unroll
      for (int c = 0; c < 8; ++c) v[c] += fabsf(s[c * n3 + l]);
    }
#pragma unroll
    for (int h = 4; h > 0; h >>= 1) {  // the lanes of the upper half keep the upper columns
      const bool up = (lane & (4 * h)) != 0;
#pragma unroll
      for (int c = 0; c < h; ++c) {
        const float keep = up ? v[c + h] : v[c];
        v[c] = keep + __shfl_xor_sync(0xffffffffu, up ? v[c] : v[c + h], 4 * h);
      }
    }
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
    mx = fmaxf(mx, v[0]);
  }
  if ((lane & 3) == 0 && mx > 0.f) atomicMax(&amax[lane >> 2], __float_as_uint(mx));
}

// Bytes of the spectra arrays X and Y (one level at a time uses them).
void unif_spectra_bytes(const pbbfmm_tree* t, int C, bool f64, size_t* x, size_t* y) {
  *x = *y = 16;
  for (int l = 2; l <= t->p.tree_level; ++l) {
    const bool tc = !f64 && unif_tc_eligible(t, l, C);
    const size_t plain = (size_t)cells_at(l) * C * t->nk * (f64 ? 16 : 8);
    const int S = 1 << (l - 1);
    *x = std::max(*x, tc ? (size_t)t->nk * UnifPlanes::slot_bytes(S) : plain);
    *y = std::max(*y, tc ? (size_t)t->nk * UnifPlanes::slot_outputs(S) * sizeof(float2) : plain);
  }
}

// Level by level: forward transforms, MAC, inverse transforms (the spectra
// arrays hold one level at a time).
template <typename T>
static int run_m2l_unif_t(pbbfmm_tree* t, int C, cudaStream_t st) {
  if (int rc = init_fft_twiddles()) return rc;
  using C2 = cplx_t<T>;
  const int L = t->p.tree_level, n = t->n, m = t->m, n3 = t->n3, nk = t->nk;
  Workspace& ws = t->ws;
  C2* X = ws.proxy.as<C2>();
  C2* Y = ws.pf.as<C2>();
  const int* lists = ws.lists.as<int>();
  const int* sstart = ws.sstart_p;
  const int* tstart = ws.tstart.as<int>();
  int* halo = ws.halo.as<int>();
  const OpsView<T> ov = ops_view<T>(t);
  int rc;
  for (int l = L; l >= 2; --l) {
    if (t->lists.ntgt[l] == 0) continue;
    const int lvl = t->homog ? 0 : l - 2;
    const int span = (int)cells_at(L - l);
    const T* S_l = ws.S.as<T>() + level_offset(l, (int64_t)C * n3);
    T* F_l = ws.F.as<T>() + level_offset(l, (int64_t)C * n3);
    double len = t->p.L;
    for (int i = 0; i < l; ++i) len = 0.5 * len;
    const T scale = (T)pow(1.0 / len, t->homogen_neg), invP = (T)(1.0 / (double)(m * m * m));
    // float32, 16 parents per side or more, columns in groups of 8: the
    // tensor cores (m2l_unif_tc.cu); otherwise the CUDA cores
    if constexpr (sizeof(T) == 4) {
      if (unif_tc_eligible(t, l, C)) {
        const int S = 1 << (l - 1);
        uint8_t *socc, *tocc;
        if ((rc = kt_begin(t, KS_MAC, st))) return rc;
        if ((rc = run_unif_tc_occupancy(t, l, &socc, &tocc, st))) return rc;
        if ((rc = kt_end(t, st))) return rc;
        for (int c0 = 0; c0 < C; c0 += 8) {
          uint32_t* amax = ws.amax.as<uint32_t>();
          if ((rc = kt_begin(t, KS_FFT_FWD, st))) return rc;
          PB_CUDA(cudaMemsetAsync(amax, 0, 8 * sizeof(uint32_t), st));
          if (t->lists.nsrc[l] > 0) {
            k_moment_bound<<<std::min((t->lists.nsrc[l] + 7) / 8, 4 * 148), 256, 0, st>>>(
                lists + t->lists.src_off[l], t->lists.nsrc[l], S_l, C, c0, n3, amax);
            PB_LAUNCH("moment_bound");
          }
          if ((rc = run_unif_tc_borders(t, S, reinterpret_cast<unsigned char*>(X), st))) return rc;
          const int64_t rows = (int64_t)S * S * S * 8;
          FftFwdLaunch<T, true> f{{}, rows, st};
          f.a.S = S_l;
          f.a.X = X;
          f.a.slot_stride = UnifPlanes::slot_bytes(S);
          f.a.lo_off = UnifPlanes::lo_off(S);
          f.a.C = C;
          f.a.c0 = c0;
          f.a.side = S;
          f.a.occ = socc;
          f.a.amax = amax;
          if ((rc = dispatch_order(n, f))) return rc;
          if ((rc = kt_end(t, st))) return rc;
          if ((rc = kt_begin(t, KS_MAC, st))) return rc;
          if ((rc = run_m2l_unif_tc_level(t, l, lvl, reinterpret_cast<unsigned char*>(X),
                                          reinterpret_cast<float2*>(Y), amax, tocc, st)))
            return rc;
          if ((rc = kt_end(t, st))) return rc;
          if ((rc = kt_begin(t, KS_FFT_INV, st))) return rc;
          FftInvLaunch<T, true> g{{}, rows, st};
          g.a.Y = Y;
          g.a.F = F_l;
          g.a.slot_stride = UnifPlanes::slot_outputs(S);
          g.a.C = C;
          g.a.c0 = c0;
          g.a.side = S;
          g.a.occ = tocc;
          g.a.scale = scale;
          g.a.invP = invP;
          if ((rc = dispatch_order(n, g))) return rc;
          if ((rc = kt_end(t, st))) return rc;
        }
        continue;
      }
    }
    if (t->lists.nsrc[l] > 0) {
      if ((rc = kt_begin(t, KS_FFT_FWD, st))) return rc;
      FftFwdLaunch<T, false> f{{}, 0, st};
      f.a.S = S_l;
      f.a.X = X;
      f.a.slot_stride = cells_at(l) * C;
      f.a.C = C;
      f.a.cells = lists + t->lists.src_off[l];
      f.a.nunits = (int64_t)t->lists.nsrc[l] * C;
      if ((rc = dispatch_order(n, f))) return rc;
      if ((rc = kt_end(t, st))) return rc;
    }
    if ((rc = kt_begin(t, KS_MAC, st))) return rc;
    MacLevel<T> ml{X, Y, ov.op + (int64_t)lvl * nk * kKaraD * kKaraJ, halo, sstart, tstart,
                   span, l, C, nk, st};
    if ((rc = ml.columns())) return rc;
    if ((rc = kt_end(t, st))) return rc;
    if ((rc = kt_begin(t, KS_FFT_INV, st))) return rc;
    FftInvLaunch<T, false> g{{}, 0, st};
    g.a.Y = Y;
    g.a.F = F_l;
    g.a.slot_stride = cells_at(l) * C;
    g.a.C = C;
    g.a.cells = lists + t->lists.tgt_off[l];
    g.a.nunits = (int64_t)t->lists.ntgt[l] * C;
    g.a.scale = scale;
    g.a.invP = invP;
    if ((rc = dispatch_order(n, g))) return rc;
    if ((rc = kt_end(t, st))) return rc;
  }
  return PBBFMM_OK;
}

int run_m2l_unif(pbbfmm_tree* t, int C, cudaStream_t st) {
  return t->cur_prec == PBBFMM_PREC_FP64 ? run_m2l_unif_t<double>(t, C, st)
                                         : run_m2l_unif_t<float>(t, C, st);
}

}  // namespace pbbfmm
