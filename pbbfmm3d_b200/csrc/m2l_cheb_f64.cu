// Chebyshev M2L in float64, and its pre and post transforms, on the FP64
// tensor instructions (mma.sync m8n8k4), all levels in one launch each.
//
// Reference: FarFieldInteractions / Moment2Local (include/compute.hpp:402-508,
// 881-914): pf[t][f] = sum over the 189 offsets o of child type(t) of
// sum_s E_o[f][s] proxy[t + o][s].
//
// A work item is (tile, block of up to 128 outputs f, part of the offsets).  A
// tile is 64 consecutive (target, column) rows of one level and child type, so
// that its rows share the 189 operators.  Per offset only the rows whose
// source cell is nonempty take part, compacted in row order into groups of 8
// (the M of the instruction); the product of the compacted rows with the
// operator accumulates in registers and is then added into the tile's running
// sum in shared memory under the rows' own positions.  A row appears once per
// offset, the offsets come in a fixed order and a block barrier lies between
// the adds of consecutive offsets: the result is deterministic.
//
// Why this shape.  The kernel is bound by the FP64 pipe.  mma.sync.f64 reaches
// 36-37 TFLOP/s from two accumulators per warp up, where chains of plain FMAs
// on 8 x 8 register blocks reach 27-33 (register-bank conflicts), and it reads
// an operand element once per 8 products instead of once per FMA lane.  Both
// operands lie in shared memory in the order of the instruction's fragments
// (lane-contiguous 256-byte reads, no bank conflicts); the operators are
// stored that way in global memory, so a K chunk is one contiguous copy.  A
// tile of 64 rows leaves the running sum at 68 KB or less and two CTAs per SM:
// one CTA's barriers, adds and copies hide behind the other's products.
//
// Measured, M2L of one matvec (B200), against one FMA kernel per level with
// 128-row tiles: 500,000 clustered points, r = 120, 5 levels 41.0 -> 14.7 ms
// (28 TFLOP/s of the useful rows); 20,000 points, r = 48, 3 levels 5.3 -> 0.25
// ms; 33,331 targets, r = 91, 3 columns 10.8 -> 1.8 ms.  The transforms of the
// first: 0.86 + 0.90 -> 0.21 + 0.23 ms.
//
// Dense levels run on combinations of the children (cheb_kara.cuh): k_kara_in
// forms the 27 combined proxies of each source parent, the same M2L kernel sums
// the products over the 26 parent offsets with the combined operators
// (k_kara_ops), and k_kara_out forms the 8 children's sums: 702 products per
// parent instead of 1512.  M2L of 33,331 targets and 77,777 sources, r = 91, 3
// columns: 1.79 -> 1.29 ms; of the 500,000 clustered points (dense at levels 3
// to 5): 14.7 -> 12.5 ms.
//
// Levels with few tiles are cut along the offsets as well (`nsplit` parts, the
// partial sums added in order by k_m2l_parts), since one tile's 189 offsets
// are a serial chain of ~100 us; see m2l_cheb_f64_split.
#include <algorithm>
#include <cmath>
#include <vector>

#include "cheb_kara.cuh"
#include "fmm.cuh"

namespace pbbfmm {

constexpr int FD_R = 64;         // rows of a tile
constexpr int FD_MT = FD_R / 8;  // their groups of 8
constexpr int FD_THREADS = 256;
constexpr int FD_OFFS = 189;

struct FdLevel {
  const double* E;      // operators of the level, fragment order (cheb_fragment_operators)
  const double* proxy;  // [cell * C + col][rsp]
  double* pf;           // [cell * C + col][rf]
  double* part;         // nsplit > 1: [split][row of the level][rf]
  const int* typed;     // targets ordered by (child type, parent); combined: target parents
  int lev, span;
  // 0: rows are (cell, column) of the level, types are child types, 189
  // offsets each; otherwise combined, rows are (parent, combination, column) of
  // the `mult` combinations from j0 on, types are these, 26 parent offsets each
  int mult, j0;
  int C;                // columns of the rows
  int item0, nsplit;
  int row0, rows;       // (target, column) rows of the level, and of the levels before it
  int first[8];         // first list position of each type
  int count[8];         // targets of each type
  int tile0[9];         // first tile of each type
};

struct FdArgs {
  FdLevel lv[kChebParts];
  int nlev;
  int rf, rsp;          // rsp: rs padded to a multiple of 4
  int nblk, ntb;        // column blocks, column groups of 8 per block
  const int* sstart;
  const int* offs;      // [8][189] (ox, oy, oz, operator), then [27][26] of the combinations
};

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm volatile(
      "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

// pitch of the running sum in doubles: 8 mod 16, so that the 64-byte pieces of
// neighbouring rows lie in different halves of the banks
__host__ __device__ constexpr int fd_pitch(int ntb) { return 8 * ntb + (ntb % 2 ? 0 : 8); }
__host__ __device__ constexpr size_t fd_smem(int ntb, int kc, int nst) {
  return sizeof(double) *
         ((size_t)FD_R * fd_pitch(ntb) + (size_t)nst * kc * (FD_R + 8 * ntb));
}

// two CTAs of the widest plans fit an SM's 228 KB (the row lists and masks take less
// than 5 KB, the system 1 KB per CTA)
static_assert(2 * (fd_smem(16, 8, 3) + 6 * 1024) <= 228 * 1024 &&
                  2 * (fd_smem(15, 16, 2) + 6 * 1024) <= 228 * 1024 &&
                  2 * (fd_smem(8, 16, 3) + 6 * 1024) <= 228 * 1024,
              "two CTAs per SM");

template <int N>
__device__ __forceinline__ void cp_async_wait_group() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// Warps of a CTA: NWN column slices of TN column groups x 8 / NWN row sets
// (row groups wm, wm + 8 / NWN, ...).  With NWN = 4 every SM sub-partition
// (warp % 4) holds one warp of each row set, so an odd number of row groups
// loads the four sub-partitions alike.
template <int TN, int NWN>
struct FdWarps {
  static constexpr int nwm = (FD_THREADS / 32) / NWN;
  static constexpr int mw = FD_MT / nwm;  // most row groups of a warp
};

// kn steps of 4 along K for MW row groups x tn <= TN column groups
template <int MW, int TN, int NWM, int MWX>
__device__ __forceinline__ void fd_step(const double* __restrict__ as, const double* __restrict__ bs,
                                        int kn, int bstep, int tn, double (&acc)[MWX][TN][2]) {
#pragma unroll 2
  for (int k = 0; k < kn; ++k) {
    double a[MW], b[TN];
#pragma unroll
    for (int i = 0; i < MW; ++i) a[i] = as[i * NWM * 32];
#pragma unroll
    for (int j = 0; j < TN; ++j) b[j] = j < tn ? bs[j * 32] : 0.0;
#pragma unroll
    for (int j = 0; j < TN; ++j)
      if (j < tn) {
#pragma unroll
        for (int i = 0; i < MW; ++i) dmma(acc[i][j], a[i], b[j]);
      }
    as += FD_MT * 32;
    bs += bstep;
  }
}

template <int KC, int NST, int TN, int NWN>
__global__ void __launch_bounds__(FD_THREADS, 2) k_m2l_cheb_f64(const __grid_constant__ FdArgs a) {
  extern __shared__ __align__(16) unsigned char fd_raw[];
  using W = FdWarps<TN, NWN>;
  constexpr int SL = NST + 1;  // row lists in flight: one more than the loads run ahead
  __shared__ long long s_src[SL][FD_R];  // compacted row: proxy row of its source
  __shared__ uint8_t s_row[SL][FD_R];    // compacted row: its row of the tile
  __shared__ uint32_t s_mask[FD_OFFS][FD_R / 32];  // offset: rows with a source
  __shared__ uint8_t s_oidx[FD_OFFS];  // offsets with any, in order
  __shared__ uint8_t s_cnt[FD_OFFS];   // their rows
  __shared__ int s_xyz[FD_R], s_flat[FD_R];
  __shared__ int s_nvalid;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int li = 0;
  for (int i = 1; i < a.nlev; ++i)
    if ((int)blockIdx.x >= a.lv[i].item0) li = i;
  const FdLevel& lv = a.lv[li];
  const int local = (int)blockIdx.x - lv.item0;
  const int split = local % lv.nsplit, rest = local / lv.nsplit;
  const int nb = rest % a.nblk, tile = rest / a.nblk;
  const int ntb = a.ntb;  // column groups of a block
  const int C = lv.C;
  const int4* offs = reinterpret_cast<const int4*>(a.offs);
  int type = 0, r0, nrow, first = 0, noff = FD_OFFS, mult = 1, comb = 0;
  if (lv.mult) {  // tile0[0] tiles per combination
    type = comb = tile / lv.tile0[0];
    r0 = (tile - type * lv.tile0[0]) * FD_R;  // first row within the type
    nrow = min(FD_R, lv.count[0] * C - r0);
    offs += 8 * FD_OFFS + (lv.j0 + type) * kKaraD;
    noff = kKaraD;
    mult = lv.mult;
  } else {
    for (int i = 1; i < 8; ++i)
      if (tile >= lv.tile0[i]) type = i;
    r0 = (tile - lv.tile0[type]) * FD_R;
    nrow = min(FD_R, lv.count[type] * C - r0);
    first = lv.first[type];
    offs += type * FD_OFFS;
  }
  const int nside = 1 << lv.lev, span = lv.span;
  const int o_lo = noff * split / lv.nsplit, o_hi = noff * (split + 1) / lv.nsplit;

  const int pitch = fd_pitch(ntb);
  double* Sum = reinterpret_cast<double*>(fd_raw);  // [FD_R][pitch]
  double* As = Sum + FD_R * pitch;                  // [NST][KC / 4][FD_MT][32]
  double* Bs = As + NST * KC * FD_R;                // [NST][KC / 4][ntb][32]
  const int bstep = ntb * 32, bstage = (KC / 4) * bstep;

  if (tid < FD_R) {
    int v = -1;
    if (tid < nrow) {
      int x, y, z;
      morton_decode((uint32_t)lv.typed[first + (r0 + tid) / C], &x, &y, &z);
      v = (x << 20) | (y << 10) | z;
    }
    s_xyz[tid] = v;
    s_flat[tid] = first * C + r0 + tid;
  }
  for (int i = tid; i < FD_R * pitch / 2; i += FD_THREADS)
    reinterpret_cast<double2*>(Sum)[i] = make_double2(0.0, 0.0);
  __syncthreads();
  // the rows with a source, per offset of this part: a warp per (offset, 32
  // rows), four at a time so that their lookups are in flight together
  for (int w0 = warp; w0 < (o_hi - o_lo) * (FD_R / 32); w0 += 4 * (FD_THREADS / 32)) {
    int lo[4], hi[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int w = w0 + u * (FD_THREADS / 32), o = o_lo + w / (FD_R / 32), h = w % (FD_R / 32);
      lo[u] = hi[u] = 0;
      const int xyz = s_xyz[32 * h + lane];
      if (o < o_hi && xyz >= 0) {
        const int4 d = __ldg(offs + o);
        const int x = (xyz >> 20) + d.x, y = ((xyz >> 10) & 1023) + d.y, z = (xyz & 1023) + d.z;
        if (x >= 0 && y >= 0 && z >= 0 && x < nside && y < nside && z < nside) {
          const int64_t bm = morton_encode(x, y, z);
          lo[u] = __ldg(a.sstart + bm * span);
          hi[u] = __ldg(a.sstart + (bm + 1) * span);
        }
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int w = w0 + u * (FD_THREADS / 32), o = o_lo + w / (FD_R / 32), h = w % (FD_R / 32);
      const uint32_t m = __ballot_sync(0xffffffffu, hi[u] > lo[u]);
      if (lane == 0 && o < o_hi) s_mask[o][h] = m;
    }
  }
  __syncthreads();
  if (warp == 0) {
    int n = 0;
    for (int b = o_lo; b < o_hi; b += 32) {
      const int o = b + lane;
      const int cnt = o < o_hi ? __popc(s_mask[o][0]) + __popc(s_mask[o][1]) : 0;
      const uint32_t m = __ballot_sync(0xffffffffu, cnt > 0);
      const int at = n + __popc(m & ((1u << lane) - 1u));
      if (cnt > 0) s_oidx[at] = (uint8_t)o, s_cnt[at] = (uint8_t)cnt;
      n += __popc(m);
    }
    if (lane == 0) s_nvalid = n;
  }
  __syncthreads();
  const int nvalid = s_nvalid;
  const int k4 = a.rsp / 4, kch = (k4 + KC / 4 - 1) / (KC / 4);  // K chunks of an offset
  const int niter = nvalid * kch;
  const double* const proxy = lv.proxy;
  const double* const E0 = lv.E + (int64_t)nb * k4 * bstep;  // this block of an operator
  const int64_t op_stride = (int64_t)a.nblk * k4 * bstep;

  auto lookup = [&](int q) {  // the compacted rows of valid offset q, into slot q % SL
    if (tid >= FD_R) return;
    const int o = s_oidx[q];
    const uint32_t m0 = s_mask[o][0], m1 = s_mask[o][1];
    const uint32_t mine = tid < 32 ? m0 : m1;
    if (!((mine >> lane) & 1u)) return;
    const int pos = __popc(mine & ((1u << lane) - 1u)) + (tid < 32 ? 0 : __popc(m0));
    const int4 d = __ldg(offs + o);
    const int xyz = s_xyz[tid];
    const long long cell =
        morton_encode((xyz >> 20) + d.x, ((xyz >> 10) & 1023) + d.y, (xyz & 1023) + d.z);
    s_src[q % SL][pos] = ((cell * mult + comb) * C + s_flat[tid] % C) * a.rsp;
    s_row[q % SL][pos] = (uint8_t)tid;
  };
  // the next iteration to load: chunk lc of valid offset lq, into stage lst.  A: granules
  // of 16 bytes (two values of K) scattered into fragment order; B: a straight copy.
  int lq = 0, lc = 0, lst = 0;
  constexpr int GR = KC / 2;  // granules of a row
  const int g = tid % GR, m_first = tid / GR;
  const int a_dst = ((g >> 1) * FD_MT * 32) + (g & 1) * 2;
  auto load = [&]() {
    const int kn = min(KC / 4, k4 - lc * (KC / 4));  // steps of 4 in this chunk
    const int m_o = s_cnt[lq], mpad = (m_o + 7) & ~7;
    const long long* src = s_src[lq % SL];
    double* as = As + lst * KC * FD_R + a_dst;
    const double* ps = proxy + lc * KC + 2 * g;
    if (g < 2 * kn) {
#pragma unroll
      for (int r = 0; r < FD_R * GR / FD_THREADS; ++r) {
        const int m = m_first + r * (FD_THREADS / GR);
        if (m < mpad) {
          const bool ok = m < m_o;
          cp_async16(as + (m >> 3) * 32 + (m & 7) * 4, ps + (ok ? src[m] : 0), ok ? 16 : 0);
        }
      }
    }
    const int op = __ldg(&offs[s_oidx[lq]].w);
    const double* eo = E0 + op * op_stride + lc * bstage + 2 * tid;
    double* bs = Bs + lst * bstage + 2 * tid;
    for (int n = kn * ntb * 16 - tid; n > 0; n -= FD_THREADS) {
      cp_async16(bs, eo, 16);
      bs += 2 * FD_THREADS;
      eo += 2 * FD_THREADS;
    }
    if (++lc == kch) lc = 0, ++lq;
  };

  const int wn = warp % NWN, wm = warp / NWN;
  const int tn = min(TN, ntb - TN * wn);  // column groups of this warp (<= 0: none)
  double acc[W::mw][TN][2];
#pragma unroll
  for (int i = 0; i < W::mw; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

  // loads run NST - 1 iterations ahead
  {
    int q = 0, c = 0;
#pragma unroll
    for (int s = 0; s < NST - 1; ++s)
      if (s < niter) {
        if (c == 0) lookup(q);
        if (++c == kch) c = 0, ++q;
      }
  }
  __syncthreads();
#pragma unroll
  for (int s = 0; s < NST - 1; ++s) {
    if (s < niter) {
      lst = s;
      load();
    }
    cp_async_commit();
  }
  lst = NST - 1;
  int st = 0;
  for (int q = 0; q < nvalid; ++q) {
    const int m_o = s_cnt[q], mg = (m_o + 7) >> 3;
    const int mw = tn > 0 ? (mg - wm + W::nwm - 1) / W::nwm : 0;  // this warp's row groups
    for (int c = 0; c < kch; ++c) {
      const bool more = lq < nvalid;
      if (more && lc == 0) lookup(lq);
      cp_async_wait_group<NST - 2>();
      __syncthreads();
      if (more) load();
      cp_async_commit();
      const int kn = min(KC / 4, k4 - c * (KC / 4));
      const double* as = As + st * KC * FD_R + wm * 32 + lane;
      const double* bs = Bs + st * bstage + TN * wn * 32 + lane;
      switch (mw) {  // warp-uniform; at most W::mw
        case 1: fd_step<1, TN, W::nwm, W::mw>(as, bs, kn, bstep, tn, acc); break;
        case 2:
          if constexpr (W::mw >= 2) fd_step<2, TN, W::nwm, W::mw>(as, bs, kn, bstep, tn, acc);
          break;
        case 3:
          if constexpr (W::mw >= 4) fd_step<3, TN, W::nwm, W::mw>(as, bs, kn, bstep, tn, acc);
          break;
        case 4:
          if constexpr (W::mw >= 4) fd_step<4, TN, W::nwm, W::mw>(as, bs, kn, bstep, tn, acc);
          break;
        default: break;
      }
      if (++st == NST) st = 0;
      if (++lst == NST) lst = 0;
    }
    // the offset's product into the running sum: lane holds row lane / 4 and
    // two columns of each 8 x 8 block
    const uint8_t* rows = s_row[q % SL];
#pragma unroll
    for (int i = 0; i < W::mw; ++i) {
      if (i < mw) {
        const int m = (wm + i * W::nwm) * 8 + (lane >> 2);
        if (m < m_o) {
          double2* s = reinterpret_cast<double2*>(Sum + (int)rows[m] * pitch + 8 * TN * wn +
                                                  2 * (lane & 3));
#pragma unroll
          for (int j = 0; j < TN; ++j)
            if (j < tn) {
              double2 v = s[4 * j];
              v.x += acc[i][j][0], v.y += acc[i][j][1];
              s[4 * j] = v;
            }
        }
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
      }
    }
  }
  __syncthreads();
  const int col0 = 8 * nb * ntb, ncol = min(8 * ntb, a.rf - col0);
  for (int r = warp; r < nrow; r += FD_THREADS / 32) {
    const int flat = s_flat[r];
    double* dst =
        lv.nsplit > 1
            ? lv.part + ((int64_t)split * lv.rows + (int64_t)comb * lv.count[0] * C + flat) * a.rf
            : lv.pf + (((int64_t)lv.typed[flat / C] * mult + comb) * C + flat % C) * a.rf;
    for (int n = lane; n < ncol; n += 32) dst[col0 + n] = Sum[r * pitch + n];
  }
}

// pf = the sum of the parts, in order, for every level with nsplit > 1: a warp per row.
__global__ void k_m2l_parts(const __grid_constant__ FdArgs a, int nrows) {
  const int r = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (r >= nrows) return;
  int li = 0;
  for (int i = 1; i < a.nlev; ++i)
    if (r >= a.lv[i].row0) li = i;
  const FdLevel& lv = a.lv[li];
  const int flat = r - lv.row0;
  const int per = lv.mult ? lv.count[0] * lv.C : lv.rows;  // rows of a combination
  const int comb = flat / per, f2 = flat % per;
  double* dst = lv.pf + (((int64_t)lv.typed[f2 / lv.C] * (lv.mult ? lv.mult : 1) + comb) * lv.C +
                         f2 % lv.C) * a.rf;
  for (int n = lane; n < a.rf; n += 32) {
    double v = 0.0;
    for (int s = 0; s < lv.nsplit; ++s) v += lv.part[((int64_t)s * lv.rows + flat) * a.rf + n];
    dst[n] = v;
  }
}

// Combined proxies j0 <= j < j0 + nj of columns [c0, c0 + nc) of the listed source
// parents: warp per (parent, column).  NJ = nj (27: j0 is 0), fixed so
// that the stores need no test of j.
template <int NJ>
__global__ void k_kara_in(const int* __restrict__ parents, int np, const int* __restrict__ sstart,
                          int span, const double* __restrict__ proxy, double* __restrict__ kx,
                          int C, int c0, int nc, int j0_, int rsp) {
  constexpr int nj = NJ;
  const int j0 = NJ == kKaraJ ? 0 : j0_;
  const int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= (int64_t)np * nc) return;
  const int64_t p = parents[w / nc];
  const int c = (int)(w % nc);
  const unsigned present = children_present(sstart, p, span);
  for (int k = lane; k < rsp; k += 32) {
    double v[8];
#pragma unroll
    for (int ch = 0; ch < 8; ++ch)
      v[ch] = ((present >> ch) & 1) ? proxy[((8 * p + ch) * C + c0 + c) * rsp + k] : 0.0;
    kara_combine(v, [&](int j, double x) {
      if ((unsigned)(j - j0) < (unsigned)nj) kx[((p * nj + j - j0) * nc + c) * rsp + k] = x;
    });
  }
}

// Combined operators [level][27][26] from the level's 316, element by element;
// terms[j * 26 + d][8]: +-(operator + 1), 0 for none.
__global__ void k_kara_ops(const double* __restrict__ E, const int* __restrict__ terms,
                           int64_t per_op, double* __restrict__ Ek) {
  const int64_t op = blockIdx.y, lvl = blockIdx.z;
  const double* e = E + lvl * 316 * per_op;
  double* o = Ek + (lvl * kKaraJ * kKaraD + op) * per_op;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < per_op;
       i += (int64_t)gridDim.x * blockDim.x) {
    double v = 0.0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int s = terms[op * 8 + q];
      if (s) v += s > 0 ? e[(s - 1) * per_op + i] : -e[(-s - 1) * per_op + i];
    }
    o[i] = v;
  }
}

// Offsets of the combinations, [27][26] (dx, dy, dz, j 26 + d), behind the 189
// per child type; and the operators' terms (k_kara_ops).
void cheb_kara_tables(const int* Ktable, std::vector<int>* offs, std::vector<int>* terms) {
  for (int j = 0; j < kKaraJ; ++j)
    for (int d = 0, n = 0; d < 27; ++d) {
      if (d == 13) continue;
      const int D[3] = {d / 9 - 1, d / 3 % 3 - 1, d % 3 - 1}, jd[3] = {j / 9, j / 3 % 3, j % 3};
      for (int i = 0; i < 3; ++i) offs->push_back(D[i]);
      offs->push_back(j * kKaraD + n++);
      for (int q = 0; q < 8; ++q) {  // bit i: the subtracted term of coordinate i
        int lex = 0, sign = 1;
        bool used = true;
        for (int i = 0; i < 3; ++i) {
          const int sub = (q >> i) & 1;
          int off = 2 * D[i];
          if (jd[i] == 0)
            used &= !sub;
          else if (sub)
            sign = -sign;
          else
            off += jd[i] == 1 ? 1 : -1;
          lex = 7 * lex + off + 3;
        }
        const int op = used ? Ktable[lex] : -1;  // -1: near, no operator
        terms->push_back(op < 0 ? 0 : sign * (op + 1));
      }
    }
}

int cheb_rsp(int rs) { return (rs + 3) & ~3; }

// column groups of 8 in blocks of at most 16, all blocks alike (the last one padded)
void cheb_fragment_blocks(int rf, int* nblk, int* ntb) {
  const int nt = (rf + 7) / 8;
  *nblk = (nt + 15) / 16;
  *ntb = (nt + *nblk - 1) / *nblk;
}

// Operators (column-major rf x rs blocks) in the order of the instruction's B
// fragments: [operator][column block][k / 4][f / 8][lane], lane (f % 8) 4 + k % 4
// holds E[f][k]; zero padded to 4 in k and to whole blocks in f.
std::vector<double> cheb_fragment_operators(const double* K, int64_t nops, int rf, int rs) {
  int nblk, ntb;
  cheb_fragment_blocks(rf, &nblk, &ntb);
  const int k4 = cheb_rsp(rs) / 4;
  const size_t per_blk = (size_t)k4 * ntb * 32, per_op = per_blk * nblk;
  std::vector<double> out((size_t)nops * per_op, 0.0);
  parallel_for(nops, [&](int64_t b0, int64_t b1) {
    for (int64_t b = b0; b < b1; ++b) {
      const double* E = K + (size_t)b * rf * rs;
      double* o = out.data() + (size_t)b * per_op;
      for (int k = 0; k < rs; ++k)
        for (int f = 0; f < rf; ++f)
          o[(f / 8 / ntb) * per_blk + ((size_t)(k / 4) * ntb + f / 8 % ntb) * 32 + (f % 8) * 4 +
            k % 4] = E[f + (size_t)rf * k];
    }
  });
  return out;
}

// ------------------------------------------------------------------------
// M2L pre / post transforms, all levels in one launch:
//   Out[row][m] = alpha sum_k W[m][k] X[row][k],   row = cell * C + col,
// for the listed cells (reference: include/compute.hpp:373-396 and 881-914),
// W = VT diag(Kw) or diag(Kw) U in fragment order.  A CTA takes 64 rows and
// one column block of W; the accumulators stay in registers.
struct CgLevel {
  const double* W;
  const double* X;
  double* Out;
  const int* cells;
  int rows, item0;
  double alpha;
};
struct CgArgs {
  CgLevel lv[kMaxLevel - 1];
  int nlev, C, M, K, ldo, nblk, ntb;  // ldo >= M: pitch of Out, zeros from M on
};

constexpr int CGD_KC = 16, CGD_NST = 3;

template <int TN, int NWN>
__global__ void __launch_bounds__(FD_THREADS, 2) k_colgemm_f64(const __grid_constant__ CgArgs a) {
  extern __shared__ __align__(16) unsigned char cgd_raw[];
  using W = FdWarps<TN, NWN>;
  __shared__ long long s_base[FD_R];  // row: cell * C + col, -1 past the end
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int li = 0;
  for (int i = 1; i < a.nlev; ++i)
    if ((int)blockIdx.x >= a.lv[i].item0) li = i;
  const CgLevel& lv = a.lv[li];
  const int local = (int)blockIdx.x - lv.item0;
  const int nb = local % a.nblk, r0 = (local / a.nblk) * FD_R;
  const int ntb = a.ntb, K = a.K, k4 = (K + 3) / 4, bstep = ntb * 32;
  double* As = reinterpret_cast<double*>(cgd_raw);
  double* Bs = As + CGD_NST * CGD_KC * FD_R;
  const int bstage = (CGD_KC / 4) * bstep;
  if (tid < FD_R) {
    const int r = r0 + tid;
    s_base[tid] = r < lv.rows ? (long long)lv.cells[r / a.C] * a.C + r % a.C : -1;
  }
  __syncthreads();
  const int nch = (k4 + CGD_KC / 4 - 1) / (CGD_KC / 4);
  const int kk = tid % CGD_KC, m_first = tid / CGD_KC;
  const int a_dst = (kk >> 2) * FD_MT * 32 + (kk & 3);
  const double* W0 = lv.W + (int64_t)nb * k4 * bstep;
  const double* X = lv.X;
  auto load = [&](int c, int st) {
    const int kn = min(CGD_KC / 4, k4 - c * (CGD_KC / 4)), k = c * CGD_KC + kk;
    double* as = As + st * CGD_KC * FD_R + a_dst;
#pragma unroll
    for (int r = 0; r < FD_R * CGD_KC / FD_THREADS; ++r) {
      const int m = m_first + r * (FD_THREADS / CGD_KC);
      const long long b = s_base[m];
      const bool ok = b >= 0 && k < K;
      cp_async_elem(as + (m >> 3) * 32 + (m & 7) * 4, X + (ok ? b * K + k : 0), ok);
    }
    const double* w = W0 + c * bstage + 2 * tid;
    double* bs = Bs + st * bstage + 2 * tid;
    for (int n = kn * ntb * 16 - tid; n > 0; n -= FD_THREADS) {
      cp_async16(bs, w, 16);
      bs += 2 * FD_THREADS;
      w += 2 * FD_THREADS;
    }
  };
  const int wn = warp % NWN, wm = warp / NWN, tn = min(TN, ntb - TN * wn);
  double acc[W::mw][TN][2];
#pragma unroll
  for (int i = 0; i < W::mw; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
#pragma unroll
  for (int s = 0; s < CGD_NST - 1; ++s) {
    if (s < nch) load(s, s);
    cp_async_commit();
  }
  int st = 0, lst = CGD_NST - 1;
  for (int c = 0; c < nch; ++c) {
    cp_async_wait_group<CGD_NST - 2>();
    __syncthreads();
    if (c + CGD_NST - 1 < nch) load(c + CGD_NST - 1, lst);
    cp_async_commit();
    const int kn = min(CGD_KC / 4, k4 - c * (CGD_KC / 4));
    if (tn > 0)
      fd_step<W::mw, TN, W::nwm, W::mw>(As + st * CGD_KC * FD_R + wm * 32 + lane,
                                        Bs + st * bstage + TN * wn * 32 + lane, kn, bstep, tn, acc);
    if (++st == CGD_NST) st = 0;
    if (++lst == CGD_NST) lst = 0;
  }
#pragma unroll
  for (int i = 0; i < W::mw; ++i) {
    const long long b = s_base[(wm + i * W::nwm) * 8 + (lane >> 2)];
    if (b < 0) continue;
    double* o = lv.Out + b * a.ldo;
#pragma unroll
    for (int j = 0; j < TN; ++j)
      if (j < tn) {
        const int m = 8 * (nb * ntb + TN * wn + j) + 2 * (lane & 3);
        if (m < a.ldo) o[m] = lv.alpha * acc[i][j][0];
        if (m + 1 < a.ldo) o[m + 1] = lv.alpha * acc[i][j][1];
      }
  }
}

template <int TN, int NWN>
static int launch_colgemm_f64(const CgArgs& a, int items, cudaStream_t st) {
  const size_t smem = sizeof(double) * CGD_NST * CGD_KC * (FD_R + 8 * (size_t)a.ntb);
  PB_CUDA(cudaFuncSetAttribute(k_colgemm_f64<TN, NWN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)smem));
  k_colgemm_f64<TN, NWN><<<items, FD_THREADS, smem, st>>>(a);
  PB_LAUNCH("colgemm_f64");
  return PBBFMM_OK;
}

// pre (post = false): proxy = VT (Kw o S) of the nonempty source cells;
// post: F = scale Kw o (U pf) of the nonempty target cells.
static int run_colgemm_f64(pbbfmm_tree* t, bool post, int C, cudaStream_t st) {
  const int L = t->p.tree_level, n3 = t->n3, rf = t->ops.rf, rs = t->ops.rs, rsp = cheb_rsp(rs);
  Workspace& ws = t->ws;
  CgArgs a{};
  a.C = C;
  a.M = post ? n3 : rs;
  a.K = post ? rf : n3;
  a.ldo = post ? n3 : rsp;
  cheb_fragment_blocks(a.M, &a.nblk, &a.ntb);
  const int64_t per_op = (int64_t)cheb_rsp(a.K) * a.nblk * a.ntb * 8;
  int64_t items = 0;
  for (int l = L; l >= 2; --l) {
    const int nc = post ? t->lists.ntgt[l] : t->lists.nsrc[l];
    if (nc == 0) continue;
    const int lvl = t->homog ? 0 : l - 2;
    CgLevel& v = a.lv[a.nlev++];
    v.W = (post ? t->d_U : t->d_VT) + lvl * per_op;
    const double* S = ws.S.as<double>() + level_offset(l, (int64_t)C * n3);
    double* F = ws.F.as<double>() + level_offset(l, (int64_t)C * n3);
    double* proxy = ws.proxy.as<double>() + level_offset(l, (int64_t)C * rsp);
    const double* pf = ws.pf.as<double>() + level_offset(l, (int64_t)C * rf);
    v.X = post ? pf : S;
    v.Out = post ? F : proxy;
    v.cells = ws.lists.as<int>() + (post ? t->lists.tgt_off[l] : t->lists.src_off[l]);
    v.rows = nc * C;
    v.item0 = (int)items;
    v.alpha = 1.0;
    if (post) {
      double len = t->p.L;
      for (int i = 0; i < l; ++i) len = 0.5 * len;
      v.alpha = pow(1.0 / len, t->homogen_neg);
    }
    items += (int64_t)((v.rows + FD_R - 1) / FD_R) * a.nblk;
  }
  if (items == 0) return PBBFMM_OK;
  const int n = (int)items;
  if (a.ntb > 12) return launch_colgemm_f64<4, 4>(a, n, st);
  if (a.ntb > 8) return launch_colgemm_f64<3, 4>(a, n, st);
  if (a.ntb > 6) return launch_colgemm_f64<2, 4>(a, n, st);
  if (a.ntb > 4) return launch_colgemm_f64<3, 2>(a, n, st);
  if (a.ntb > 2) return launch_colgemm_f64<2, 2>(a, n, st);
  if (a.ntb == 2) return launch_colgemm_f64<1, 2>(a, n, st);
  return launch_colgemm_f64<1, 1>(a, n, st);
}

// ------------------------------------------------------------------------
// Parts per tile: 1 when the tiles alone give every resident CTA (two per SM)
// four items or more, otherwise enough parts for that, of at least 8 offsets.
static int m2l_cheb_f64_split(int64_t items, int nsm) {
  const int64_t want = 8 * (int64_t)nsm;
  if (items >= want || items == 0) return 1;
  return (int)std::min<int64_t>((want + items - 1) / items, FD_OFFS / 8);
}

template <int KC, int NST, int TN, int NWN>
static int launch_f64(const FdArgs& a, int items, cudaStream_t st) {
  const size_t smem = fd_smem(a.ntb, KC, NST);
  PB_CUDA(cudaFuncSetAttribute(k_m2l_cheb_f64<KC, NST, TN, NWN>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  k_m2l_cheb_f64<KC, NST, TN, NWN><<<items, FD_THREADS, smem, st>>>(a);
  PB_LAUNCH("m2l_cheb_f64");
  return PBBFMM_OK;
}

// Combined operators of the tree's current set (made on first use, kept with it).
static int ensure_kara_ops(pbbfmm_tree* t, int64_t per_op, cudaStream_t st) {
  if (t->d_Ek) return PBBFMM_OK;
  const int nlev = t->ops.nlev;
  if (int rc = dev_alloc((void**)&t->d_Ek, sizeof(double) * nlev * kKaraJ * kKaraD * per_op))
    return rc;
  k_kara_ops<<<dim3((unsigned)std::min<int64_t>((per_op + 255) / 256, 64), kKaraJ * kKaraD,
                    (unsigned)nlev),
               256, 0, st>>>(t->d_E, t->d_offs + 4 * (8 * FD_OFFS + kKaraJ * kKaraD), per_op,
                             t->d_Ek);
  count_launches(1);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {  // (a kernel's first launch may need memory of its own)
    cudaFree(t->d_Ek);
    t->d_Ek = nullptr;
    return cuda_status(e, "kara_ops");
  }
  return PBBFMM_OK;
}

// The parts of the far field and their arrays.  What the combinations need is not
// needed by the direct lists: where it cannot be allocated, less is asked for, in
// the end nothing.
static int plan_m2l_f64(pbbfmm_tree* t, int C, int64_t per_op, ChebPlan* plan, cudaStream_t st) {
  const int L = t->p.tree_level, rf = t->ops.rf, rsp = cheb_rsp(t->ops.rs);
  bool dense[kMaxLevel + 1] = {}, used[kMaxLevel + 1] = {};
  for (int l = 2; l <= L; ++l) {
    used[l] = t->lists.ntgt[l] > 0;
    dense[l] = cheb_kara_level(t, l);
  }
  for (int64_t bound = t->kara_bytes;; bound = kara_less(bound)) {
    *plan = cheb_plan(dense, used, L, C, 8 * rsp, 8 * rf, 0, bound);
    if (plan->y_bytes == 0) return PBBFMM_OK;
    int rc = ensure_kara_ops(t, per_op, st);
    if (!rc) rc = grow(t->ws.kara_x, plan->x_bytes);
    if (!rc) rc = grow(t->ws.kara_y, plan->y_bytes);
    if (rc != PBBFMM_ERR_ALLOC) return rc;
  }
}

static int launch_m2l_f64(pbbfmm_tree* t, int C, const std::vector<ChebPart>& parts, FdArgs a,
                          int64_t per_op, int nsm, cudaStream_t st) {
  const int L = t->p.tree_level, rf = t->ops.rf, rsp = a.rsp;
  Workspace& ws = t->ws;
  int64_t items = 0;
  for (const ChebPart& q : parts) {
    const int l = q.level;
    FdLevel& v = a.lv[a.nlev++];
    v.C = q.nc;
    if (q.nj) {
      const int np = t->lists.ntgt[l - 1];
      v.E = t->d_Ek + (int64_t)(t->homog ? 0 : l - 2) * kKaraJ * kKaraD * per_op;
      v.proxy = ws.kara_x.as<double>() + q.x / 8;
      v.pf = ws.kara_y.as<double>() + q.y / 8;
      v.typed = ws.lists.as<int>() + t->lists.tgt_off[l - 1];
      v.lev = l - 1;
      v.span = (int)cells_at(L - l + 1);
      v.mult = q.nj;
      v.j0 = q.j0;
      v.count[0] = np;
      v.tile0[0] = (int)(((int64_t)np * q.nc + FD_R - 1) / FD_R);
      v.tile0[8] = q.nj * v.tile0[0];
      v.rows = q.nj * np * q.nc;
      items += (int64_t)v.tile0[8] * a.nblk;
      const int ns = t->lists.nsrc[l - 1];
      const int64_t warps = (int64_t)ns * q.nc;
      if (warps > 0) {
        (q.nj == kKaraJ ? k_kara_in<kKaraJ> : k_kara_in<kKaraJ / 3>)
            <<<(unsigned)((warps + 7) / 8), 256, 0, st>>>(
                ws.lists.as<int>() + t->lists.src_off[l - 1], ns, ws.sstart_p, (int)cells_at(L - l),
                ws.proxy.as<double>() + level_offset(l, (int64_t)C * rsp),
                ws.kara_x.as<double>() + q.x / 8, C, q.c0, q.nc, q.j0, rsp);
        PB_LAUNCH("kara_in");
      }
      continue;
    }
    v.E = t->d_E + (int64_t)(t->homog ? 0 : l - 2) * 316 * per_op;
    v.proxy = ws.proxy.as<double>() + level_offset(l, (int64_t)C * rsp);
    v.pf = ws.pf.as<double>() + level_offset(l, (int64_t)C * rf);
    v.typed = ws.lists.as<int>() + t->lists.typ_off[l];
    v.lev = l;
    v.span = (int)cells_at(L - l);
    int tiles = 0;
    for (int y = 0; y < 8; ++y) {
      v.tile0[y] = tiles;
      v.first[y] = t->lists.ntyp[l][y];
      v.count[y] = t->lists.ntyp[l][y + 1] - t->lists.ntyp[l][y];
      tiles += (int)(((int64_t)v.count[y] * C + FD_R - 1) / FD_R);
    }
    v.tile0[8] = tiles;
    v.rows = t->lists.ntyp[l][8] * C;
    items += (int64_t)tiles * a.nblk;
  }
  if (items == 0) return PBBFMM_OK;
  int64_t part = 0, rows = 0;
  // (without the parts where there is no room for them)
  for (int nsplit = m2l_cheb_f64_split(items, nsm);; nsplit = 1) {
    items = part = rows = 0;
    for (int i = 0; i < a.nlev; ++i) {
      FdLevel& v = a.lv[i];
      v.item0 = (int)items;
      // (of the combinations' 26 offsets at least 6 to a part)
      v.nsplit = v.mult ? std::min(nsplit, kKaraD / 6) : nsplit;
      v.row0 = (int)rows;
      items += (int64_t)v.tile0[8] * a.nblk * v.nsplit;
      if (v.nsplit == 1) continue;
      rows += v.rows;
      part += (int64_t)v.nsplit * v.rows * rf;
    }
    const int rc = rows > 0 ? grow(ws.m2l_part, sizeof(double) * part) : PBBFMM_OK;
    if (!rc) break;
    if (rc != PBBFMM_ERR_ALLOC) return rc;
  }
  if (rows > 0) {
    double* p = ws.m2l_part.as<double>();
    for (int i = 0; i < a.nlev; ++i) {
      if (a.lv[i].nsplit == 1) continue;
      a.lv[i].part = p;
      p += (int64_t)a.lv[i].nsplit * a.lv[i].rows * rf;
    }
  }
  // slices of TN column groups so that all 8 warps have work; the deepest
  // staging that leaves two CTAs per SM (227 KB less 1 KB per CTA and the row
  // lists: 16 column groups have room for three stages of 8, not two of 16)
  const int ntb = a.ntb, n = (int)items;
  int rc;
  if (ntb == 16)
    rc = launch_f64<8, 3, 4, 4>(a, n, st);
  else if (ntb > 12)
    rc = launch_f64<16, 2, 4, 4>(a, n, st);
  else if (ntb > 8)
    rc = launch_f64<16, 2, 3, 4>(a, n, st);
  else if (ntb > 6)
    rc = launch_f64<16, 3, 2, 4>(a, n, st);
  else if (ntb > 4)
    rc = launch_f64<16, 3, 3, 2>(a, n, st);
  else if (ntb > 2)
    rc = launch_f64<16, 3, 2, 2>(a, n, st);
  else if (ntb == 2)
    rc = launch_f64<16, 3, 1, 2>(a, n, st);
  else
    rc = launch_f64<16, 3, 1, 1>(a, n, st);
  if (rc) return rc;
  if (rows > 0) {
    k_m2l_parts<<<(unsigned)((rows + 7) / 8), 256, 0, st>>>(a, (int)rows);
    PB_LAUNCH("m2l_parts");
  }
  for (const ChebPart& q : parts)
    if (q.nj && t->lists.ntgt[q.level - 1] > 0)
      if ((rc = launch_kara_out(t, q, ws.kara_y.as<double>() + q.y / 8,
                                ws.pf.as<double>() + level_offset(q.level, (int64_t)C * rf), C, rf,
                                st)))
        return rc;
  return PBBFMM_OK;
}

static int run_m2l_f64(pbbfmm_tree* t, int C, cudaStream_t st) {
  FdArgs a{};
  a.rf = t->ops.rf;
  a.rsp = cheb_rsp(t->ops.rs);
  cheb_fragment_blocks(a.rf, &a.nblk, &a.ntb);
  a.sstart = t->ws.sstart_p;
  a.offs = t->d_offs;
  int nsm = 148;
  PB_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, t->device));
  const int64_t per_op = (int64_t)a.rsp * a.nblk * a.ntb * 8;
  ChebPlan plan;
  if (int rc = plan_m2l_f64(t, C, per_op, &plan, st)) return rc;
  for (const std::vector<ChebPart>& parts : plan.launches)
    if (int rc = launch_m2l_f64(t, C, parts, a, per_op, nsm, st)) return rc;
  return PBBFMM_OK;
}

int run_m2l_cheb_f64(pbbfmm_tree* t, int C, cudaStream_t st) {
  int rc;
  if ((rc = kt_begin(t, KS_M2L_PRE, st))) return rc;
  if ((rc = run_colgemm_f64(t, false, C, st))) return rc;
  if ((rc = kt_end(t, st))) return rc;
  if ((rc = kt_begin(t, KS_M2L, st))) return rc;
  if ((rc = run_m2l_f64(t, C, st))) return rc;
  if ((rc = kt_end(t, st))) return rc;
  if ((rc = kt_begin(t, KS_M2L_POST, st))) return rc;
  if ((rc = run_colgemm_f64(t, true, C, st))) return rc;
  return kt_end(t, st);
}

}  // namespace pbbfmm
