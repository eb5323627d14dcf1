// Point binning on the GPU: recentring, bit-exact leaf keys, stable sort,
// leaf ranges and per-level lists of nonempty cells.
//
// Reference: H2_3D_Compute ctor recentring (include/compute.hpp:92-131) and
// DistributeFieldPoints (include/compute.hpp:1127-1203) over the octree of
// BuildFMMHierarchy (src/H2_3D_Tree.cpp:917-977).  The reference walks a
// pointer tree and compares each point against FP64 cell centres built by
// repeated +-quarter-length steps; here the same comparisons run per point on
// the device, producing the same Morton leaf index, and a stable radix sort
// keeps the reference's within-leaf order (original index order).
#include <cub/cub.cuh>

#include "fmm.cuh"

namespace pbbfmm {

constexpr int kBBoxBlocks = 296;
constexpr int kBBoxThreads = 256;

__global__ void k_bbox_partial(const double* __restrict__ p, int64_t N, double* __restrict__ part) {
  double mn[3] = {1e32, 1e32, 1e32}, mx[3] = {-1e32, -1e32, -1e32};
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < N;
       i += (int64_t)gridDim.x * blockDim.x) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      double v = p[3 * i + d];
      mn[d] = v < mn[d] ? v : mn[d];
      mx[d] = mx[d] < v ? v : mx[d];
    }
  }
  __shared__ double s[6][kBBoxThreads / 32];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    for (int o = 16; o > 0; o >>= 1) {
      double a = __shfl_down_sync(0xffffffffu, mn[d], o);
      double b = __shfl_down_sync(0xffffffffu, mx[d], o);
      mn[d] = a < mn[d] ? a : mn[d];
      mx[d] = mx[d] < b ? b : mx[d];
    }
  }
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0)
    for (int d = 0; d < 3; ++d) {
      s[d][w] = mn[d];
      s[3 + d][w] = mx[d];
    }
  __syncthreads();
  if (threadIdx.x < 3) {
    int d = threadIdx.x;
    double a = s[d][0], b = s[3 + d][0];
    for (int j = 1; j < kBBoxThreads / 32; ++j) {
      a = s[d][j] < a ? s[d][j] : a;
      b = b < s[3 + d][j] ? s[3 + d][j] : b;
    }
    part[blockIdx.x * 6 + d] = a;
    part[blockIdx.x * 6 + 3 + d] = b;
  }
}

// One warp: lanes over the partial boxes, then across the lanes.
__global__ void k_bbox_final(const double* __restrict__ part, int nb, double* __restrict__ ctr) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    double a = 1e32, b = -1e32;
    for (int j = lane; j < nb; j += 32) {
      a = part[j * 6 + d] < a ? part[j * 6 + d] : a;
      b = b < part[j * 6 + 3 + d] ? part[j * 6 + 3 + d] : b;
    }
    for (int o = 16; o > 0; o >>= 1) {
      const double a2 = __shfl_xor_sync(0xffffffffu, a, o), b2 = __shfl_xor_sync(0xffffffffu, b, o);
      a = a2 < a ? a2 : a;
      b = b < b2 ? b2 : b;
    }
    if (lane == 0) ctr[d] = 0.5 * (a + b);  // include/compute.hpp:108-111
  }
}

// Leaf key by the reference's comparison descent.
__global__ void k_keys(const double* __restrict__ p, int64_t N, const double* __restrict__ ctr,
                       double box, int L, uint32_t* __restrict__ key, int* __restrict__ idx) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= N) return;
  const double qx = p[3 * i + 0] - ctr[0];
  const double qy = p[3 * i + 1] - ctr[1];
  const double qz = p[3 * i + 2] - ctr[2];
  double cx = 0, cy = 0, cz = 0, len = box;
  uint32_t k = 0;
  for (int lev = 0; lev < L; ++lev) {
    const int bx = !(qx < cx), by = !(qy < cy), bz = !(qz < cz);
    k = k * 8u + (uint32_t)(4 * bx + 2 * by + bz);
    const double q = 0.25 * len;
    cx = bx ? __dadd_rn(cx, q) : __dsub_rn(cx, q);
    cy = by ? __dadd_rn(cy, q) : __dsub_rn(cy, q);
    cz = bz ? __dadd_rn(cz, q) : __dsub_rn(cz, q);
    len = 0.5 * len;
  }
  key[i] = k;
  idx[i] = (int)i;
}

// start[k] = first sorted position with key >= k, k in [0, nleaf].
__global__ void k_leaf_start(const uint32_t* __restrict__ ks, int N, int64_t nleaf,
                             int* __restrict__ start) {
  int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k > nleaf) return;
  int lo = 0, hi = N;
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if ((int64_t)ks[mid] < k)
      lo = mid + 1;
    else
      hi = mid;
  }
  start[k] = lo;
}

// Sorted positions (recentred, SoA) and, with w, the sorted weights.
__global__ void k_gather(const double* __restrict__ p, const int* __restrict__ perm, int N,
                         const double* __restrict__ ctr, double* __restrict__ soa,
                         const double* __restrict__ w, int C, double* __restrict__ ws) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const int j = perm[i];
#pragma unroll
  for (int d = 0; d < 3; ++d) soa[(int64_t)d * N + i] = p[3 * (int64_t)j + d] - ctr[d];
  if (w)
    for (int c = 0; c < C; ++c) ws[(int64_t)i * C + c] = w[(int64_t)c * N + j];
}

// Sorted weights, thread per (point, column): coalesced rows for several columns.
__global__ void k_gather_w(const double* __restrict__ w, const int* __restrict__ perm, int Ns,
                           int C, double* __restrict__ ws) {
  int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= (int64_t)Ns * C) return;
  int j = (int)(t / C), c = (int)(t % C);
  ws[t] = w[(int64_t)c * Ns + perm[j]];
}

// Lists of cells, all levels in three launches (counts per block of cells, a
// scan of the counts, the writes): per level the nonempty source cells and
// target cells in Morton order and the target cells ordered by (child type,
// parent); of the leaves also the dense and the sparse target leaves, back to
// back, with the first 32-target chunk of each dense one.  (A select per list
// costs two launches for each of 3 (L - 1) lists: of a 20,000-point matvec on
// 4 levels that was 0.1 of 0.64 ms, nearly all of it launches.)
enum ListKind { LIST_SRC = 0, LIST_TGT = 1, LIST_TYPED = 2, LIST_DENSE = 3, LIST_SPARSE = 4 };
constexpr int kListThreads = 256, kListItems = 4, kListBlock = kListThreads * kListItems;

constexpr int kScanItems = 16;  // counts of a thread of k_list_scan
// Blocks of a list at most: a deep level's blocks take several pieces of kListBlock
// cells each, and there are still enough to fill the chip (20,000 points at level 9,
// binning: a piece per block 5.9, so 4.8 ms; at level 8 0.79 and 0.68 ms).
constexpr int kListBlocksMax = 2048;

struct ListJob {
  int kind, shift;     // shift = 3 (L - level): leaf ranges of a cell
  int ncells, block0;  // cells (LIST_TYPED: parents), first block
  int pieces;          // of kListBlock cells per block
  int count0, ncounts; // its counts: one per block (LIST_TYPED: per child type and block)
  int* out;            // the list
  int* count;          // its length (device)
  int slot;            // index of the length in the host copy; LIST_TYPED: the first
                       // position of each child type, then the length, from slot + 1 on
};
struct ListArgs {
  ListJob job[3 * (kMaxLevel - 1) + 2];
  int njobs, nblocks, ncounts;
  const int *sstart, *tstart;
  int *bcount, *bchunk;  // the jobs' counts: cells selected, chunks of dense leaves
  int* prefix;           // first chunk of each dense leaf, then the total
  int* hcount;           // mapped host memory: the lengths and bounds
};

__device__ __forceinline__ int list_job(const ListArgs& a) {
  int j = 0;
  for (int i = 1; i < a.njobs; ++i)
    if ((int)blockIdx.x >= a.job[i].block0) j = i;
  return j;
}
// whether cell c of a job is listed; for dense leaves also their chunks of 32
// targets
__device__ __forceinline__ bool list_cell(const ListArgs& a, const ListJob& j, int64_t c,
                                          int* chunks) {
  if (c >= j.ncells) return false;
  const int* start = j.kind == LIST_SRC ? a.sstart : a.tstart;
  const int n = start[(c + 1) << j.shift] - start[c << j.shift];
  *chunks = (n + 31) / 32;
  if (j.kind == LIST_DENSE) return n >= kLaneLeafMin;
  if (j.kind == LIST_SPARSE) return n > 0 && n < kLaneLeafMin;
  return n > 0;
}

// LIST_TYPED: bit t: child t of parent p has targets.  A thread reads its parent's
// nine bounds, neighbours in memory, and serves all eight types (a cell at a time in
// the order of the list, types outermost, every sector of bounds is read eight
// times: 20,000 points at level 9, binning 8.3 ms, so 5.9).
__device__ __forceinline__ unsigned list_children(const ListArgs& a, const ListJob& j, int64_t p) {
  if (p >= j.ncells) return 0;
  unsigned m = 0;
  int lo = a.tstart[(8 * p) << j.shift];
#pragma unroll
  for (int t = 0; t < 8; ++t) {
    const int hi = a.tstart[(8 * p + t + 1) << j.shift];
    m |= hi > lo ? 1u << t : 0u;
    lo = hi;
  }
  return m;
}

// LIST_TYPED: end of block b's parents
__device__ __forceinline__ int64_t list_end(const ListJob& j, int b) {
  return min((int64_t)j.ncells, (int64_t)(b + 1) * j.pieces * kListBlock);
}

// block-wide exclusive prefix of (x, y); *tx, *ty the totals
__device__ __forceinline__ void block_scan2(int x, int y, int* ex, int* ey, int* tx, int* ty) {
  __shared__ int sx[kListThreads / 32], sy[kListThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int ix = x, iy = y;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int ax = __shfl_up_sync(0xffffffffu, ix, o), ay = __shfl_up_sync(0xffffffffu, iy, o);
    if (lane >= o) ix += ax, iy += ay;
  }
  __syncthreads();  // the previous call's readers
  if (lane == 31) sx[w] = ix, sy[w] = iy;
  __syncthreads();
  int bx = 0, by = 0;
  *tx = *ty = 0;
  for (int k = 0; k < kListThreads / 32; ++k) {
    if (k < w) bx += sx[k], by += sy[k];
    *tx += sx[k], *ty += sy[k];
  }
  *ex = bx + ix - x;
  *ey = by + iy - y;
}

__global__ void __launch_bounds__(kListThreads) k_list_count(const __grid_constant__ ListArgs a) {
  const ListJob& j = a.job[list_job(a)];
  const int b = (int)blockIdx.x - j.block0, tid = threadIdx.x;
  if (j.kind == LIST_TYPED) {
    __shared__ int s_n[8];
    if (tid < 8) s_n[tid] = 0;
    __syncthreads();
    int n[8] = {};
    for (int64_t p0 = (int64_t)b * j.pieces * kListBlock, e = list_end(j, b); p0 < e;
         p0 += kListThreads) {
      const unsigned m = list_children(a, j, p0 + tid);
#pragma unroll
      for (int t = 0; t < 8; ++t) n[t] += __popc(__ballot_sync(0xffffffffu, (m >> t) & 1u));
    }
    if ((tid & 31) == 0)
#pragma unroll
      for (int t = 0; t < 8; ++t) atomicAdd(&s_n[t], n[t]);
    __syncthreads();
    if (tid < 8) a.bcount[j.count0 + tid * (j.ncounts / 8) + b] = s_n[tid];
    return;
  }
  int n = 0, nc = 0;
  for (int k = 0; k < j.pieces; ++k) {
    const int64_t c0 = ((int64_t)b * j.pieces + k) * kListBlock + tid * kListItems;
#pragma unroll
    for (int i = 0; i < kListItems; ++i) {
      int ch;
      if (list_cell(a, j, c0 + i, &ch)) n += 1, nc += ch;
    }
  }
  int ex, ey, tx, ty;
  block_scan2(n, nc, &ex, &ey, &tx, &ty);
  if (tid == 0) a.bcount[j.count0 + b] = tx, a.bchunk[j.count0 + b] = ty;
}

// exclusive scan of a job's counts from k0 on, in place, N per thread; n, nc: the sums
// of those before
template <int N>
__device__ __forceinline__ void scan_counts(const ListArgs& a, const ListJob& j, int k0, int* n,
                                            int* nc) {
  const bool dense = j.kind == LIST_DENSE;
  const int first = k0 + threadIdx.x * N;
  int x[N], y[N], sx = 0, sy = 0;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const bool ok = first + i < j.ncounts;
    x[i] = ok ? a.bcount[j.count0 + first + i] : 0;
    y[i] = ok && dense ? a.bchunk[j.count0 + first + i] : 0;
    sx += x[i], sy += y[i];
  }
  int ex, ey, tx, ty;
  block_scan2(sx, sy, &ex, &ey, &tx, &ty);
  ex += *n, ey += *nc;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    if (first + i < j.ncounts) {
      a.bcount[j.count0 + first + i] = ex;
      if (dense) a.bchunk[j.count0 + first + i] = ey;
    }
    ex += x[i], ey += y[i];
  }
  *n += tx;
  *nc += ty;
}

// one block per list; several counts per thread and step where there are many
__global__ void __launch_bounds__(kListThreads) k_list_scan(const __grid_constant__ ListArgs a) {
  const ListJob& j = a.job[blockIdx.x];
  int n = 0, nc = 0;
  if (j.ncounts <= kListThreads)
    scan_counts<1>(a, j, 0, &n, &nc);
  else
    for (int k0 = 0; k0 < j.ncounts; k0 += kListThreads * kScanItems)
      scan_counts<kScanItems>(a, j, k0, &n, &nc);
  if (threadIdx.x == 0) {
    *j.count = n;
    if (j.kind == LIST_DENSE) a.prefix[n] = nc;
    if (j.slot >= 0) a.hcount[j.slot] = n;
    if (j.kind == LIST_TYPED) a.hcount[j.slot + 9] = n;
  }
}

__global__ void __launch_bounds__(kListThreads) k_list_write(const __grid_constant__ ListArgs a) {
  const int ji = list_job(a);
  const ListJob& j = a.job[ji];
  const int b = (int)blockIdx.x - j.block0, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (j.kind == LIST_TYPED) {
    __shared__ int s_w[2][8][kListThreads / 32];  // listed children of a type in a warp
    const int nb = j.ncounts / 8;
    const unsigned below = (1u << lane) - 1u;
    int at[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) at[t] = a.bcount[j.count0 + t * nb + b];
    if (b == 0 && tid < 8) a.hcount[j.slot + 1 + tid] = a.bcount[j.count0 + tid * nb];
    int i = 0;
    for (int64_t p0 = (int64_t)b * j.pieces * kListBlock, e = list_end(j, b); p0 < e;
         p0 += kListThreads, ++i) {
      const int64_t p = p0 + tid;
      const unsigned m = list_children(a, j, p);
      unsigned v[8];
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        v[t] = __ballot_sync(0xffffffffu, (m >> t) & 1u);
        if (lane == 0) s_w[i & 1][t][warp] = __popc(v[t]);
      }
      __syncthreads();  // (two buffers: a warp is at most one step ahead)
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        int mine = at[t] + __popc(v[t] & below), all = 0;
        for (int w = 0; w < kListThreads / 32; ++w) {
          const int x = s_w[i & 1][t][w];
          if (w < warp) mine += x;
          all += x;
        }
        if ((m >> t) & 1u) j.out[mine] = (int)(8 * p + t);
        at[t] += all;
      }
    }
    return;
  }
  // the sparse leaves follow the dense ones (the job before)
  const int base = j.kind == LIST_SPARSE ? *a.job[ji - 1].count : 0;
  int at0 = a.bcount[j.count0 + b], cat0 = j.kind == LIST_DENSE ? a.bchunk[j.count0 + b] : 0;
  for (int k = 0; k < j.pieces; ++k) {
    const int64_t c0 = ((int64_t)b * j.pieces + k) * kListBlock + tid * kListItems;
    int ch[kListItems], n = 0, nc = 0;
    bool sel[kListItems];
#pragma unroll
    for (int i = 0; i < kListItems; ++i) {
      sel[i] = list_cell(a, j, c0 + i, &ch[i]);
      if (sel[i]) n += 1, nc += ch[i];
    }
    int ex, ey, tx, ty;
    block_scan2(n, nc, &ex, &ey, &tx, &ty);
    int at = at0 + ex, cat = cat0 + ey;
#pragma unroll
    for (int i = 0; i < kListItems; ++i) {
      if (sel[i]) {
        j.out[base + at] = (int)(c0 + i);
        if (j.kind == LIST_DENSE) a.prefix[at] = cat;
        at += 1;
        cat += ch[i];
      }
    }
    at0 += tx;
    cat0 += ty;
  }
}

int run_binning(pbbfmm_tree* t, const double* d_tgt, int64_t Nf, const double* d_src, int64_t Ns,
                const double* d_w, int C, cudaStream_t st) {
  Workspace& ws = t->ws;
  const int L = t->p.tree_level;
  const int64_t nleaf = cells_at(L);
  const int64_t Nmax = Nf > Ns ? Nf : Ns;

  // CUB scratch: radix sort of Nmax keys
  size_t cub_need = 0;
  PB_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, cub_need, (const uint32_t*)nullptr,
                                          (uint32_t*)nullptr, (const int*)nullptr, (int*)nullptr,
                                          (int)Nmax, 0, 3 * L, st));
  // one buffer given as sources and targets is binned once: the sources'
  // arrays are the targets'
  const bool same = d_tgt == d_src && Nf == Ns;
  int64_t list_need = 0;
  for (int l = 2; l <= L; ++l) {
    int64_t nc = cells_at(l);
    list_need += (nc < Ns ? nc : Ns) + 2 * (nc < Nf ? nc : Nf);
  }
  int rc;
  if ((rc = grow(ws.bbox_part, 8 * 6 * kBBoxBlocks))) return rc;
  if ((rc = grow(ws.ctr, 8 * 4))) return rc;
  if ((rc = grow(ws.key, 4 * Nmax))) return rc;
  if ((rc = grow(ws.key_sorted, 4 * Nmax))) return rc;
  if ((rc = grow(ws.idx, 4 * Nmax))) return rc;
  if ((rc = grow(ws.tperm, 4 * Nf))) return rc;
  if (!same && (rc = grow(ws.sperm, 4 * Ns))) return rc;
  if ((rc = grow(ws.tstart, 4 * (nleaf + 1)))) return rc;
  if (!same && (rc = grow(ws.sstart, 4 * (nleaf + 1)))) return rc;
  if ((rc = grow(ws.tpos, 8 * 3 * Nf))) return rc;
  if (!same && (rc = grow(ws.spos, 8 * 3 * Ns))) return rc;
  if ((rc = grow(ws.wsorted, 8 * Ns * (int64_t)C))) return rc;
  if ((rc = grow(ws.cub_temp, cub_need))) return rc;
  if ((rc = grow(ws.lists, 4 * (list_need + 16)))) return rc;
  if ((rc = grow(ws.dcounts, 4 * (kMaxLevel + 1) * 3))) return rc;
  // dense and sparse target leaves, the chunk prefix, then the block counts
  const int64_t leaf_need = (nleaf < Nf ? nleaf : Nf) + 1;
  auto list_pieces = [](int64_t cells) {
    return (cells + (int64_t)kListBlock * kListBlocksMax - 1) / ((int64_t)kListBlock * kListBlocksMax);
  };
  auto list_blocks = [&](int64_t cells) {
    const int64_t per = kListBlock * list_pieces(cells);
    return (cells + per - 1) / per;
  };
  int64_t list_counts = 0;
  for (int l = 2; l <= L; ++l)
    list_counts += (l == L ? 4 : 2) * list_blocks(cells_at(l)) + 8 * list_blocks(cells_at(l - 1));
  if ((rc = grow(ws.leafpart, 4 * (2 * leaf_need + 2 * list_counts)))) return rc;
  if (!ws.h_counts) {
    PB_CUDA(cudaHostAlloc(&ws.h_counts, sizeof(int) * 12 * (kMaxLevel + 1), cudaHostAllocMapped));
    PB_CUDA(cudaHostGetDevicePointer(&ws.d_counts, ws.h_counts, 0));
  }
  double* ctr = ws.ctr.as<double>();
  uint32_t* key = ws.key.as<uint32_t>();
  uint32_t* key_sorted = ws.key_sorted.as<uint32_t>();
  int* idx = ws.idx.as<int>();
  int* lists = ws.lists.as<int>();

  // recentre on the target bounding box (an adjoint pass keeps the forward
  // targets' box, given by bbox_pts)
  const double* bpts = t->bbox_pts ? t->bbox_pts : d_tgt;
  const int64_t bn = t->bbox_pts ? t->bbox_n : Nf;
  k_bbox_partial<<<kBBoxBlocks, kBBoxThreads, 0, st>>>(bpts, bn, ws.bbox_part.as<double>());
  k_bbox_final<<<1, 32, 0, st>>>(ws.bbox_part.as<double>(), kBBoxBlocks, ctr);
  PB_LAUNCH_N("bbox", 2);

  auto bin_set = [&](const double* pts, int64_t N, int* perm, int* start) -> int {
    if (N > 0) {
      k_keys<<<(unsigned)((N + 255) / 256), 256, 0, st>>>(pts, N, ctr, t->p.L, L, key, idx);
      PB_LAUNCH("keys");
      size_t bytes = ws.cub_temp.cap;
      PB_CUDA(cub::DeviceRadixSort::SortPairs(ws.cub_temp.p, bytes, key, key_sorted, idx, perm,
                                              (int)N, 0, 3 * L, st));
      // onesweep: one histogram pass plus one pass per 8-bit digit
      count_launches(1 + (3 * L + 7) / 8);
    }
    k_leaf_start<<<(unsigned)((nleaf + 1 + 255) / 256), 256, 0, st>>>(key_sorted, (int)N, nleaf,
                                                                      start);
    PB_LAUNCH("leaf_start");
    return PBBFMM_OK;
  };
  auto gather = [&](const double* pts, const int* perm, int64_t N, double* pos, const double* w) -> int {
    if (N == 0) return PBBFMM_OK;
    const bool fused = C < 4;  // few columns: the weights with the positions
    k_gather<<<(unsigned)((N + 255) / 256), 256, 0, st>>>(pts, perm, (int)N, ctr, pos,
                                                         fused ? w : nullptr, C,
                                                         ws.wsorted.as<double>());
    PB_LAUNCH("gather");
    if (w && !fused) {
      k_gather_w<<<(unsigned)((N * C + 255) / 256), 256, 0, st>>>(w, perm, (int)N, C,
                                                                 ws.wsorted.as<double>());
      PB_LAUNCH("gather_w");
    }
    return PBBFMM_OK;
  };
  ws.sperm_p = same ? ws.tperm.as<int>() : ws.sperm.as<int>();
  ws.sstart_p = same ? ws.tstart.as<int>() : ws.sstart.as<int>();
  ws.spos_p = same ? ws.tpos.as<double>() : ws.spos.as<double>();
  if ((rc = bin_set(d_tgt, Nf, ws.tperm.as<int>(), ws.tstart.as<int>()))) return rc;
  if ((rc = gather(d_tgt, ws.tperm.as<int>(), Nf, ws.tpos.as<double>(), same ? d_w : nullptr)))
    return rc;
  if (!same) {
    if ((rc = bin_set(d_src, Ns, ws.sperm_p, ws.sstart_p))) return rc;
    if ((rc = gather(d_src, ws.sperm_p, Ns, ws.spos_p, d_w))) return rc;
  }

  LevelLists& LL = t->lists;
  ListArgs la{};
  la.sstart = ws.sstart_p;
  la.tstart = ws.tstart.as<int>();
  la.hcount = ws.d_counts;
  int* cnt = ws.dcounts.as<int>();  // [l][0]=nsrc [l][1]=ntgt [l][2]=ntyp; [0] and [1] dense, sparse
  int* part = ws.leafpart.as<int>();
  la.prefix = part + leaf_need;
  la.bcount = la.prefix + leaf_need;
  la.bchunk = la.bcount + list_counts;
  auto add = [&](int kind, int l, int* out, int* count, int slot) {
    ListJob& j = la.job[la.njobs++];
    j.kind = kind;
    j.shift = 3 * (L - l);
    j.ncells = (int)cells_at(kind == LIST_TYPED ? l - 1 : l);
    j.block0 = la.nblocks;
    j.count0 = la.ncounts;
    j.pieces = (int)list_pieces(j.ncells);
    j.ncounts = (int)list_blocks(j.ncells) * (kind == LIST_TYPED ? 8 : 1);
    j.out = out;
    j.count = count;
    j.slot = slot;
    la.nblocks += (int)list_blocks(j.ncells);
    la.ncounts += j.ncounts;
  };
  int64_t off = 0;
  for (int l = 2; l <= L; ++l) {
    const int64_t nc = cells_at(l), ms = nc < Ns ? nc : Ns, mt = nc < Nf ? nc : Nf;
    LL.src_off[l] = off;
    LL.tgt_off[l] = off + ms;
    LL.typ_off[l] = off + ms + mt;
    for (int k = 0; k < 3; ++k)
      add(k, l, lists + (k == 0 ? LL.src_off[l] : k == 1 ? LL.tgt_off[l] : LL.typ_off[l]),
          cnt + 3 * l + k, 12 * l + k);
    off += ms + 2 * mt;
  }
  add(LIST_DENSE, L, part, cnt, -1);
  add(LIST_SPARSE, L, part, cnt + 1, -1);
  ws.ndense = cnt;
  ws.dense_prefix = la.prefix;
  k_list_count<<<la.nblocks, kListThreads, 0, st>>>(la);
  k_list_scan<<<la.njobs, kListThreads, 0, st>>>(la);
  k_list_write<<<la.nblocks, kListThreads, 0, st>>>(la);
  PB_LAUNCH_N("lists", 3);
  PB_CUDA(cudaStreamSynchronize(st));
  const int* hc = ws.h_counts;
  for (int l = 2; l <= L; ++l) {
    LL.nsrc[l] = hc[12 * l + 0];
    LL.ntgt[l] = hc[12 * l + 1];
    for (int k = 0; k < 9; ++k) LL.ntyp[l][k] = hc[12 * l + 3 + k];
  }
  return PBBFMM_OK;
}

}  // namespace pbbfmm
