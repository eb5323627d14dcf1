// Downward pass (L2L) and the leaf phase (L2P + P2P + scatter to output).
//
// Reference: DownwardPass / Local2Local (include/compute.hpp:552-587,
// 799-878) and NearFieldInteractions (include/compute.hpp:591-749) with
// EvaluateField / EvaluateField_self (:761-785).  The reference's P2P uses
// the kernel's symmetry to update both leaves of a pair under an OpenMP
// critical section; here each target point gathers from its 27 neighbour
// leaves (no atomics, no symmetry assumption, sources may differ from
// targets), and the far-field interpolation, the near-field sum and the
// scatter to the caller's output are one kernel.
#include <type_traits>

#include "fmm.cuh"
#include "interp.cuh"

namespace pbbfmm {

// L2L of the higher orders (k_l2l_units: the others), one warp per nonempty
// target parent and column: the parent's local
// coefficients are staged once and pushed through the x, y and z passes for
// each nonempty child, which is updated in place (F_child += ...).
template <int N>
struct L2LCfg {
  static constexpr int n3 = N * N * N;
  static constexpr int per_warp = 3 * n3;  // parent + two pass buffers (elements)
  static constexpr int warps = 8;
};

template <int N, typename T>
__global__ void __launch_bounds__(32 * L2LCfg<N>::warps)
    k_l2l(const int* __restrict__ parents, int npar, const int* __restrict__ tstart,
          int span_child, const T* __restrict__ Fpar, T* __restrict__ Fch, int C,
          const T* __restrict__ Cw_g) {
  using G = L2LCfg<N>;
  constexpr int n2 = N * N, n3 = G::n3;
  extern __shared__ __align__(16) unsigned char smraw[];
  T* smd = reinterpret_cast<T*>(smraw);
  __shared__ T sCw[2 * N * N];
  for (int i = threadIdx.x; i < 2 * n2; i += blockDim.x) sCw[i] = Cw_g[i];
  __syncthreads();
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
  const int task = blockIdx.x * G::warps + wl;
  if (task >= npar * C) return;
  const int par = parents[task / C], col = task % C;
  T* sp = smd + wl * G::per_warp;
  T* b0 = sp + n3;
  T* b1 = b0 + n3;
  const T* src = Fpar + ((int64_t)par * C + col) * n3;
  for (int i = lane; i < n3; i += 32) sp[i] = src[i];
  // which children hold targets (lanes 0..8 read the 9 leaf-range bounds at
  // once)
  int bound = 0;
  if (lane <= 8) bound = tstart[(int64_t)(par * 8 + lane) * span_child];
  unsigned present = 0;
#pragma unroll
  for (int ch = 0; ch < 8; ++ch)
    present |= (__shfl_sync(0xffffffffu, bound, ch + 1) != __shfl_sync(0xffffffffu, bound, ch))
                   ? 1u << ch : 0u;
  __syncwarp();
  for (int ch = 0; ch < 8; ++ch) {
    const int cell = par * 8 + ch;
    if (!((present >> ch) & 1)) continue;  // child without targets
    const T* wx = sCw + (((ch >> 2) & 1) ? n2 : 0);
    const T* wy = sCw + (((ch >> 1) & 1) ? n2 : 0);
    const T* wz = sCw + ((ch & 1) ? n2 : 0);
    // x: Fx[l1 n2 + l2 n + l3] = sum_k F[k n2 + l2 n + l3] wx[l1 + k n]
    for (int i = lane; i < n3; i += 32) {
      const int l1 = i / n2, rem = i % n2;
      T v = 0;
#pragma unroll
      for (int k = 0; k < N; ++k) v += sp[k * n2 + rem] * wx[l1 + k * N];
      b0[i] = v;
    }
    __syncwarp();
    // y: Fy[l1 n2 + l2 n + l3] = sum_k Fx[l1 n2 + k n + l3] wy[l2 + k n]
    for (int i = lane; i < n3; i += 32) {
      const int l1 = i / n2, l2 = (i / N) % N, l3 = i % N;
      T v = 0;
#pragma unroll
      for (int k = 0; k < N; ++k) v += b0[l1 * n2 + k * N + l3] * wy[l2 + k * N];
      b1[i] = v;
    }
    __syncwarp();
    // z: Fchild[l1 n + l3] += sum_k Fy[l1 n + k] wz[l3 + k n]   (l1 over n^2)
    T* dst = Fch + ((int64_t)cell * C + col) * n3;
    for (int i = lane; i < n3; i += 32) {
      const int l1 = i / N, l3 = i % N;
      T v = 0;
#pragma unroll
      for (int k = 0; k < N; ++k) v += b1[l1 * N + k] * wz[l3 + k * N];
      dst[i] += v;
    }
    __syncwarp();
  }
}

// L2L for orders with InterpCfg::use (interp.cuh): the x pass once per x half,
// the y pass once per (x, y) quarter, the z pass per child.
template <int N, typename T>
__global__ void __launch_bounds__(InterpCfg<N, T>::threads)
    k_l2l_units(const int* __restrict__ parents, int64_t nunits, const int* __restrict__ tstart,
                int span_child, const T* __restrict__ Fpar, T* __restrict__ Fch, int C,
                const __grid_constant__ InterpOps<N, T> op) {
  using G = InterpCfg<N, T>;
  constexpr int n2 = G::n2, n3 = G::n3, U = G::U, NT = G::threads;
  // units per warp and values per lane of the children's updates
  constexpr int VPW = (U + NT / 32 - 1) / (NT / 32), RPU = (n3 + 31) / 32;
  extern __shared__ __align__(16) unsigned char smraw[];
  T* sp = reinterpret_cast<T*>(smraw);  // [n^3][U + 1] parent, then the children's updates
  T* mid = sp + n3 * (U + 1);           // 2 x [n^3][U] after x
  __shared__ int64_t s_row[U];    // unit: its parent's locals, or -1
  __shared__ int64_t s_child[U];  // its first child's locals
  __shared__ unsigned s_present[U];
  const int tid = threadIdx.x, u = tid % U, l1 = tid / U, warp = tid >> 5, lane = tid & 31;
  if (tid < U) {
    const int64_t g = (int64_t)blockIdx.x * U + tid;
    int64_t row = -1, child = 0;
    unsigned present = 0;
    if (g < nunits) {
      const int64_t p = parents[g / C];
      row = (p * C + g % C) * n3;
      child = (8 * p * C + g % C) * n3;
      int lo = tstart[8 * p * span_child];
      for (int ch = 0; ch < 8; ++ch) {
        const int hi = tstart[(8 * p + ch + 1) * span_child];
        present |= hi != lo ? 1u << ch : 0u;
        lo = hi;
      }
    }
    s_row[tid] = row;
    s_child[tid] = child;
    s_present[tid] = present;
  }
  __syncthreads();
  units_in<U, n3, NT, U + 1>(sp, Fpar, [&](int v) { return s_row[v]; });
  cp_async_commit();
  cp_async_wait_all();
  __syncthreads();
  if (l1 < N) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int rem = l1 + N * i;
      T x[N];
#pragma unroll
      for (int k = 0; k < N; ++k) x[k] = sp[(k * n2 + rem) * (U + 1) + u];
#pragma unroll
      for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int o = 0; o < N; ++o) {
          T v = 0;
#pragma unroll
          for (int k = 0; k < N; ++k) v = fma(x[k], op.w[b][o + k * N], v);
          mid[(b * n3 + o * n2 + rem) * U + u] = v;
        }
    }
  }
  __syncthreads();
#pragma unroll 1
  for (int bx = 0; bx < 2; ++bx)
#pragma unroll
    for (int by = 0; by < 2; ++by) {
      T y[N][N];
      if (l1 < N) {
        const T* m = mid + (bx * n3 + l1 * n2) * U + u;
#pragma unroll
        for (int l3 = 0; l3 < N; ++l3) {
          T x[N];
#pragma unroll
          for (int k = 0; k < N; ++k) x[k] = m[(k * N + l3) * U];
#pragma unroll
          for (int l2 = 0; l2 < N; ++l2) {
            T v = 0;
#pragma unroll
            for (int k = 0; k < N; ++k) v = fma(x[k], op.w[by][l2 + k * N], v);
            y[l2][l3] = v;
          }
        }
      }
#pragma unroll
      for (int bz = 0; bz < 2; ++bz) {
        const int ch = 4 * bx + 2 * by + bz;
        // the child's coefficients, loaded while its update is computed (a warp
        // per unit, lanes over its row, as units_out)
        T cur[VPW][RPU];
#pragma unroll
        for (int i = 0; i < VPW; ++i) {
          const int v = warp + i * (NT / 32);
          const bool ok = v < U && ((s_present[v] >> ch) & 1);
          const T* f = Fch + (ok ? s_child[v] + (int64_t)ch * C * n3 : 0);
#pragma unroll
          for (int r = 0; r < RPU; ++r) cur[i][r] = ok && lane + 32 * r < n3 ? f[lane + 32 * r] : T(0);
        }
        if (l1 < N) {
          T* d = sp + l1 * n2 * (U + 1) + u;
#pragma unroll
          for (int l2 = 0; l2 < N; ++l2)
#pragma unroll
            for (int l3 = 0; l3 < N; ++l3) {
              T v = 0;
#pragma unroll
              for (int k = 0; k < N; ++k) v = fma(y[l2][k], op.w[bz][l3 + k * N], v);
              d[(l2 * N + l3) * (U + 1)] = v;
            }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < VPW; ++i) {
          const int v = warp + i * (NT / 32);
          if (v < U && ((s_present[v] >> ch) & 1)) {
            T* f = Fch + s_child[v] + (int64_t)ch * C * n3;
#pragma unroll
            for (int r = 0; r < RPU; ++r) {
              const int e = lane + 32 * r;
              if (e < n3) f[e] = cur[i][r] + sp[e * (U + 1) + v];
            }
          }
        }
        __syncthreads();
      }
    }
}


template <typename T>
struct L2LLaunch {
  pbbfmm_tree* t;
  int C, l;  // child level
  cudaStream_t st;
  template <int N>
  int run() {
    const int L = t->p.tree_level;
    Workspace& ws = t->ws;
    const int64_t per = (int64_t)C * N * N * N;
    const int np = t->lists.ntgt[l - 1];
    if constexpr (InterpCfg<N, T>::use) {
      using I = InterpCfg<N, T>;
      const int64_t units = (int64_t)np * C;
      PB_CUDA(cudaFuncSetAttribute(k_l2l_units<N, T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)I::smem));
      k_l2l_units<N, T><<<(unsigned)((units + I::U - 1) / I::U), I::threads, I::smem, st>>>(
          ws.lists.as<int>() + t->lists.tgt_off[l - 1], units, ws.tstart.as<int>(),
          (int)cells_at(L - l), ws.F.as<T>() + level_offset(l - 1, per),
          ws.F.as<T>() + level_offset(l, per), C, interp_ops<N, T>(t));
      PB_LAUNCH("l2l");
      return PBBFMM_OK;
    } else {
    using G = L2LCfg<N>;
    const int64_t tasks = (int64_t)np * C;
    const size_t smem = sizeof(T) * G::per_warp * G::warps;
    PB_CUDA(cudaFuncSetAttribute(k_l2l<N, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k_l2l<N, T><<<(unsigned)((tasks + G::warps - 1) / G::warps), 32 * G::warps, smem, st>>>(
        ws.lists.as<int>() + t->lists.tgt_off[l - 1], np, ws.tstart.as<int>(),
        (int)cells_at(L - l), ws.F.as<T>() + level_offset(l - 1, per),
        ws.F.as<T>() + level_offset(l, per), C, ops_view<T>(t).Cw);
    PB_LAUNCH("l2l");
    return PBBFMM_OK;
    }
  }
};

// The leaf kernels' arguments for this compute.  Potentials: the binning's
// leaves dense-first, with the dense leaves' first 32-target chunks (so that
// each launch's active warps are packed into the first CTAs of its grid).
// Gradients: all leaves, one warp each.
static void prepare_leaf_args(pbbfmm_tree* t, int64_t Nf, int64_t Ns, int C, double* out,
                              pbbfmm_leaf_args* a) {
  const int L = t->p.tree_level;
  const int nl = t->lists.ntgt[L];
  Workspace& ws = t->ws;
  const bool f64 = t->cur_prec == PBBFMM_PREC_FP64;
  const int64_t perS = (int64_t)C * t->n3;
  *a = pbbfmm_leaf_args{};
  a->precision = t->cur_prec;
  a->gradient = t->gl.on ? 1 : 0;
  a->leaves = ws.lists.as<int>() + t->lists.tgt_off[L];
  a->nleaves = nl;
  a->tstart = ws.tstart.as<int>();
  a->sstart = ws.sstart_p;
  a->tperm = ws.tperm.as<int>();
  a->tpos = ws.tpos.as<double>();
  a->spos = ws.spos_p;
  a->wsorted = ws.wsorted.as<double>();
  a->Nf = (int)Nf;
  a->Ns = (int)Ns;
  a->C = C;
  a->F_leaf = f64 ? (const void*)(ws.F.as<double>() + level_offset(L, perS))
                  : (const void*)(ws.F.as<float>() + level_offset(L, perS));
  a->n = t->n;
  a->cheb = t->p.use_chebyshev;
  a->Tkz = f64 ? (const void*)t->d_Tkz : (const void*)t->f_Tkz;
  a->box = t->p.L;
  a->L = L;
  a->kparam = t->d_kparam;
  if (t->gl.on) {
    a->out = t->gl.values ? out : nullptr;
    a->contract = t->gl.contract;
    a->grad_out = t->gl.grad_out;
    return;
  }
  a->out = out;
  a->leaves = ws.leafpart.as<int>();
  a->ndense = ws.ndense;
  a->chunk_prefix = ws.dense_prefix;
  // upper bound of the chunk count: Nf / 32 + one partial chunk per dense
  // leaf (at most Nf / kLaneLeafMin of them)
  a->max_chunks = Nf / 32 + (nl < Nf / kLaneLeafMin ? nl : Nf / kLaneLeafMin) + 1;
}

// Status of a leaf launcher's return value (0, a cudaError_t code, or -1 for
// a gradient pass of a kernel without gradient).
static int leaf_status(int r) {
  if (r == 0) return PBBFMM_OK;
  if (r < 0) {
    set_error("this kernel has no gradient: position gradients are not available");
    return PBBFMM_ERR_UNSUPPORTED;
  }
  return cuda_status((cudaError_t)r, "leaf kernels");
}

struct LeafBuiltin {
  const pbbfmm_leaf_args* a;
  cudaStream_t st;
  template <class KF>
  int run() {
    return leaf_status(launch_leaf_kernels<KF>(*a, st));
  }
};

template <typename T>
static int run_downward_t(pbbfmm_tree* t, int C, cudaStream_t st) {
  const int L = t->p.tree_level;
  // level-2 locals have no parent contribution (levels 0 and 1 carry none)
  for (int l = 3; l <= L; ++l) {
    if (t->lists.ntgt[l - 1] == 0) continue;
    if (int rc_ = kt_begin(t, KS_L2L, st)) return rc_;
    L2LLaunch<T> ll{t, C, l, st};
    if (int rc_ = dispatch_order(t->n, ll)) return rc_;
    if (int rc_ = kt_end(t, st)) return rc_;
  }
  return PBBFMM_OK;
}

int run_downward(pbbfmm_tree* t, int C, cudaStream_t st) {
  return t->cur_prec == PBBFMM_PREC_FP64 ? run_downward_t<double>(t, C, st)
                                         : run_downward_t<float>(t, C, st);
}

int run_leaves(pbbfmm_tree* t, int64_t Nf, int64_t Ns, int C, double* d_out, cudaStream_t st) {
  if (t->lists.ntgt[t->p.tree_level] == 0) return PBBFMM_OK;
  pbbfmm_leaf_args a;
  if (int rc = kt_begin(t, KS_LEAF, st)) return rc;
  prepare_leaf_args(t, Nf, Ns, C, d_out, &a);
  int rc;
  if (t->p.kernel == PBBFMM_KERNEL_USER) {
    if (a.gradient && !t->user.has_gradient) return leaf_status(-1);
    rc = leaf_status(t->user.launch_leaf(&a, (void*)st));
  } else {
    LeafBuiltin lb{&a, st};
    rc = dispatch_kernel(t->p.kernel, lb);
  }
  if (rc) return rc;
  count_launches(a.gradient ? 1 : 2);
  return kt_end(t, st);
}

}  // namespace pbbfmm
