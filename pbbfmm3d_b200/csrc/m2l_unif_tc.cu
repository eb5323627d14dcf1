// Frequency-domain M2L of the uniform path on the tensor cores (mixed
// precision), for levels with at least 16 parents per side and column groups
// of 8.
//
// Reference: FarFieldInteractions / FrequencyProduct, include/compute.hpp:
// 488-544 and 930-943: for each frequency k, each target child t of a parent
// P accumulates E_k[o] x_k(s) over the source children s of P's 27
// neighbour parents whose offset o (in child widths) is far.  Written per
// parent offset D in {-1, 0, 1}^3 this is a block product
//     y_k(P)[t] += sum_s B_{k,D}[t][s] x_k(P + D)[s],
// with B_{k,D} an 8 x 8 complex block that is zero where (t, s) are near
// neighbours.  In real form (x = re + i im) the block is 16 x 16, and the
// whole step is a GEMM whose rows are (parent, column) pairs.
//
// Tiling.  A work item is a frequency slot and a block of 8 x 1 x 16 target
// parents (x0..x0+7, y, z0..z0+15): 8 accumulators of 128 rows (z, column) x
// 32 columns (child and re/im, the products with B hi, then with B lo).  The
// item walks the 10 source planes x0-1..x0+8; of each it takes the three lines
// y-1..y+1 of 18 parents z0-1..z0+16.  A source plane is one pipeline stage:
// the A operand, 3 x 144 rows (z, column) x K = 16 (child, re/im) in F16 hi and
// lo parts.  For (D_y, D_z) the window of 128 rows of line y + D_y shifted by
// D_z parents lines up with the target rows: it is a start address of the
// descriptor.  The operator tiles B stack the three D_x in N (96 rows: D_x x
// (hi, lo) x (child, re/im)), so one MMA serves the three target planes x - D_x
// at once; their TMEM accumulators are adjacent.  Each (D_y, D_z) issues two
// tcgen05.mma kind::f16 (A hi and A lo, K = 16): D = A_hi B + A_lo B =
// (A_hi + A_lo)(B_hi + B_lo), accumulated in float32.
//
// Scaling.  F16 holds 11 significant bits between 2^-14 and 2^16, so both
// operands are scaled by powers of two before the split: the spectra of a
// column by 2^sA with sA from a bound on them over the level (the largest sum
// of a cell's |moments|), the operator tiles of a frequency by 2^sB(slot) from
// their largest entry.  hi = fp16(x 2^s), lo = fp16(x 2^s - hi) keep 22
// significant bits for values down to 2^-17 of the scale's maximum and an
// absolute error below 2^-39 of it for smaller ones.  A TMEM row holds one
// column only (source and target rows share the column), so one factor
// 2^-(sA + sB) per drained row and item undoes the scaling exactly.
//
// The forward transform (k_fft_fwd, SPLIT) writes the spectra already scaled,
// split and padded in the stage's layout (UnifPlanes), so that a stage is 12
// contiguous bulk copies and no thread touches an operand.  M2L of 1M points
// with 8 columns at order 5: 6.1 ms; with float32 spectra loaded and split by 9
// producer warps 19.2 ms: each value was split about four times, and the loads
// and conversions kept the MMA thread waiting for 55 % of its time.
//
// Roles (192 threads): warp 0 issues the copies, one thread of warp 1 the MMAs,
// warps 2-5 drain the accumulators (two TMEM sets, alternating by item), write
// the target spectra and zero the accumulators.  Items go round robin over the
// CTAs with the slot varying slowest, so that the CTAs share one or two slots'
// spectra in L2; the operator tiles are loaded when a CTA's slot changes.
// Source planes without sources around the line and items without targets are
// skipped.  Every wait is bounded; on timeout the kernel sets *err, waits
// (bounded) for its issued copies and MMAs, frees its TMEM and returns.
#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "fmm.cuh"
#include "tcgen05.cuh"
#include "unif_tc.cuh"

namespace pbbfmm {

constexpr int UT_BX = 8;                   // target planes of an item (along x)
constexpr int UT_LINE = 16;                // parents of a target line (along z)
constexpr int UT_ROWS = (UT_LINE + 2) * 8; // A rows of a source line: (z, column)
constexpr int UT_SRC = UT_BX + 2;          // source planes of an item
constexpr int UT_LINEB = UT_ROWS * 16;     // bytes of one part of a source line
constexpr int UT_PART = 3 * UT_LINEB;      // of one part of a stage (three lines)
constexpr int UT_ASTAGE = 4 * UT_PART;     // hi and lo parts of both K halves
constexpr int UT_NST = 6;                  // A stages
constexpr int UT_BROWS = 96;               // B rows of one (D_y, D_z) tile
constexpr int UT_BPLANE = UT_BROWS * 16;
constexpr int UT_BTILE = 2 * UT_BPLANE;
constexpr int UT_BFREQ = 9 * UT_BTILE;     // operator tiles of one frequency (bytes)
constexpr int UT_THREADS = 6 * 32;
constexpr int UT_DRAIN0 = 2 * 32;          // the drain thread that waits and signals
constexpr int UT_TMEM_COLS = 512;          // two sets of UT_BX x 32 columns
constexpr int UT_SMEM = UT_NST * UT_ASTAGE + 2 * UT_BFREQ + 1024;
static_assert(2 * UT_BX * 32 == UT_TMEM_COLS, "two accumulator sets fill the TMEM");
static_assert(UT_SMEM <= 232448 - 1024, "shared memory of one CTA");

// F16 values (uint16 bit patterns) of the operator tiles per (level, frequency).
constexpr int kUnifTcTileHalves = UT_BFREQ / 2;

// Poll limit of the pipeline waits (see g_pipe_wait_iters in m2l_tc.cu).
__device__ long long g_unif_wait_iters = kWaitIters;

// Barrier among the `n` threads of a role group (named barrier `id`).
__device__ __forceinline__ void group_sync(int id, int n) {
  asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(n) : "memory");
}

// OR of `v` over the 128 drain threads (named barrier 2).
__device__ __forceinline__ bool drains_any(bool v) {
  uint32_t r;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.u32 q, %1, 0;\n bar.red.or.pred p, 2, 128, q;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(r)
      : "r"((uint32_t)v)
      : "memory");
  return r != 0;
}

__global__ void k_occupancy(const int* __restrict__ start, int span, int64_t ncells,
                            uint8_t* __restrict__ occ) {
  const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c < ncells) occ[c] = start[(c + 1) * span] > start[c * span] ? 1 : 0;
}

// line[(x S + y) S/16 + zb]: sources in the 3 lines x 18 parents that the item
// line (y, zb) takes of plane x; item[...]: targets in the line of plane x.
__global__ void k_unif_lines(const uint8_t* __restrict__ socc, const uint8_t* __restrict__ tocc,
                             int S, uint8_t* __restrict__ line, uint8_t* __restrict__ item) {
  const int nzb = S / UT_LINE, i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= S * S * nzb) return;
  const int zb = i % nzb, y = i / nzb % S, x = i / nzb / S;
  const uint64_t* s8 = reinterpret_cast<const uint64_t*>(socc);
  const uint64_t* t8 = reinterpret_cast<const uint64_t*>(tocc);
  uint64_t s = 0, t = 0;
  for (int yy = max(y - 1, 0); yy <= min(y + 1, S - 1); ++yy)
    for (int z = max(zb * UT_LINE - 1, 0); z <= min(zb * UT_LINE + UT_LINE, S - 1); ++z)
      s |= s8[morton_encode(x, yy, z)];
  for (int z = zb * UT_LINE; z < (zb + 1) * UT_LINE; ++z) t |= t8[morton_encode(x, y, z)];
  line[i] = s != 0;
  item[i] = t != 0;
}

// Zeros in the padding rows of every part: y = -1, y = S and z = -1, z = S.
__global__ void k_unif_borders(unsigned char* __restrict__ X, int S, int nparts) {
  const int pitch = (S + 2) * 8;            // rows of a padded line
  const int ends = pitch + 8;               // rows before (0, 0) and from (S-1, S) on
  const int per = 2 * ends + (S - 1) * 16;  // padding rows of a part
  for (int part = blockIdx.y; part < nparts; part += gridDim.y) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= per) return;
    int row;
    if (i < ends) {
      row = i;
    } else if (i < 2 * ends) {
      row = (S + 2) * pitch - ends + (i - ends);
    } else {  // z = S of line y and z = -1 of line y + 1
      const int q = i - 2 * ends;
      row = (q / 16 + 1) * pitch + (S + 1) * 8 + q % 16;
    }
    *reinterpret_cast<uint4*>(X + (int64_t)part * UnifPlanes::part_bytes(S) + (int64_t)row * 16) =
        make_uint4(0, 0, 0, 0);
  }
}

struct UnifTcArgs {
  const unsigned char* X;  // UnifPlanes input
  float2* Y;               // UnifPlanes output
  const uint16_t* tiles;   // [nk][kUnifTcTileHalves] operator tiles of this level (F16)
  const int* bexp;         // [nk] exponent sB of each frequency's tiles
  const uint32_t* amax;    // [8] bound on the spectra per column (float bits)
  const uint8_t* tocc;     // [cell] target cell nonempty
  const uint8_t* line;     // k_unif_lines
  const uint8_t* item;
  int S, nk, nblocks;
  int* err;
};

__global__ void __launch_bounds__(UT_THREADS, 1) k_m2l_unif_tc(const UnifTcArgs a) {
  extern __shared__ unsigned char smraw[];
  unsigned char* base = smraw + ((1024 - (smem_u32(smraw) & 1023)) & 1023);
  unsigned char* astage = base;                       // UT_NST x [part][line][row]
  unsigned char* bbuf = astage + UT_NST * UT_ASTAGE;  // 2 x operator tiles
  __shared__ uint64_t s_full[UT_NST], s_empty[UT_NST], s_bfull[2], s_bempty[2], s_accf[2],
      s_acce[2];
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort_flag;
  volatile int* s_abort = &s_abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long long piters = g_unif_wait_iters;
  const int S = a.S, nzb = S / UT_LINE;
  const int nitems = a.nk * a.nblocks;

  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                     smem_u32(&s_tmem)),
                 "r"(UT_TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  if (tid == 0) {
    for (int i = 0; i < UT_NST; ++i) {
      mbar_init(&s_full[i], 1);   // the copies' expect_tx
      mbar_init(&s_empty[i], 1);  // the MMA commit
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_bfull[i], 1);
      mbar_init(&s_bempty[i], 1);
      mbar_init(&s_accf[i], 1);
      mbar_init(&s_acce[i], 1);
    }
    s_abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem;
  // the drain warps zero both accumulator sets before the first MMA
  if (warp >= 2) {
    const uint32_t lb = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
    const float z[16] = {};
    for (int c = 0; c < UT_TMEM_COLS; c += 16) tc_st16(lb + (uint32_t)c, z);
    tc_wait_st();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  // item w = (slot, block), block = (x group, y, z block); every role walks the
  // same items and skips the same planes
  struct Item {
    int slot, x0, y, zb;
  };
  auto item_of = [&](int w) {
    Item t;
    t.slot = w / a.nblocks;
    const int b = w % a.nblocks;
    t.zb = b % nzb;
    t.y = b / nzb % S;
    t.x0 = b / nzb / S * UT_BX;
    return t;
  };
  auto has_targets = [&](const Item& t) {
    int any = 0;
#pragma unroll
    for (int i = 0; i < UT_BX; ++i)
      any |= __ldg(a.item + ((int64_t)(t.x0 + i) * S + t.y) * nzb + t.zb);
    return any != 0;
  };
  // bit i: plane x0 - 1 + i has sources for this line
  auto planes = [&](const Item& t) {
    uint32_t m = 0;
#pragma unroll
    for (int i = 0; i < UT_SRC; ++i) {
      const int x = t.x0 - 1 + i;
      if (x >= 0 && x < S && __ldg(a.line + ((int64_t)x * S + t.y) * nzb + t.zb)) m |= 1u << i;
    }
    return m;
  };

  if (warp == 0) {
    // ------------------------------------------------------------ copies
    if (elect_one()) {
      int li = 0, f = 0, slot = -1;
      bool ok = true;
      const int64_t pitch = (int64_t)(S + 2) * 8 * 16, part = UnifPlanes::part_bytes(S);
      for (int w = blockIdx.x; w < nitems && ok; w += gridDim.x) {
        const Item t = item_of(w);
        if (!has_targets(t)) continue;
        const uint32_t pm = planes(t);
        if (t.slot != slot) {
          slot = t.slot;
          const int fb = f & 1;
          ok = f < 2 || mbar_wait_sleep(&s_bempty[fb], ((f - 2) >> 1) & 1, s_abort, piters);
          if (!ok) break;
          mbar_arrive_expect_tx(&s_bfull[fb], UT_BFREQ);
          bulk_load(bbuf + fb * UT_BFREQ, a.tiles + (int64_t)slot * kUnifTcTileHalves, UT_BFREQ,
                    &s_bfull[fb]);
          ++f;
        }
        const unsigned char* src0 = a.X + (int64_t)slot * UnifPlanes::slot_bytes(S) +
                                    t.y * pitch + (int64_t)t.zb * UT_LINE * 8 * 16;
        for (int i = 0; i < UT_SRC; ++i) {
          if (!((pm >> i) & 1)) continue;
          const int s = li % UT_NST;
          ok = li < UT_NST || mbar_wait_sleep(&s_empty[s], (li / UT_NST - 1) & 1, s_abort, piters);
          if (!ok) break;
          mbar_arrive_expect_tx(&s_full[s], UT_ASTAGE);
          const unsigned char* src = src0 + (int64_t)(t.x0 - 1 + i) * 4 * part;
#pragma unroll
          for (int cp = 0; cp < 4; ++cp)  // part
#pragma unroll
            for (int cy = 0; cy < 3; ++cy)  // line
              bulk_load(astage + s * UT_ASTAGE + cp * UT_PART + cy * UT_LINEB,
                        src + cp * part + cy * pitch, UT_LINEB, &s_full[s]);
          ++li;
        }
      }
      if (!ok) *s_abort = 1;
      // no copy may still be writing when the CTA ends: wait (bounded) for the
      // last load into each stage and buffer
      for (int i = 0; i < UT_NST; ++i) {
        const int uses = li / UT_NST + (i < li % UT_NST ? 1 : 0);
        if (uses > 0 && !mbar_wait(&s_full[i], (uses - 1) & 1, nullptr)) *s_abort = 1;
      }
      for (int i = 0; i < 2; ++i) {
        const int uses = f / 2 + (i < f % 2 ? 1 : 0);
        if (uses > 0 && !mbar_wait(&s_bfull[i], (uses - 1) & 1, nullptr)) *s_abort = 1;
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issue
    if (elect_one()) {
      int li = 0, f = 0, it = 0, slot = -1;
      bool ok = true, bused = false;
      for (int w = blockIdx.x; w < nitems && ok; w += gridDim.x) {
        const Item t = item_of(w);
        if (!has_targets(t)) continue;
        const uint32_t pm = planes(t);
        if (t.slot != slot) {
          if (bused) tc_commit(&s_bempty[(f - 1) & 1]);  // the last slot's tiles are free
          slot = t.slot;
          bused = true;
          ok = mbar_wait_sleep(&s_bfull[f & 1], (f >> 1) & 1, s_abort, piters);
          ++f;
          if (!ok) break;
        }
        const int ab = it & 1;
        if (it >= 2 && !mbar_wait_sleep(&s_acce[ab], ((it - 2) >> 1) & 1, s_abort, piters)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t bb = smem_u32(bbuf + ((f - 1) & 1) * UT_BFREQ);
        const uint32_t dset = tmem + (uint32_t)(ab * UT_BX * 32);
        for (int i = 0; i < UT_SRC; ++i) {
          if (!((pm >> i) & 1)) continue;
          const int s = li % UT_NST;
          if (!mbar_wait_sleep(&s_full[s], (li / UT_NST) & 1, s_abort, piters)) {
            ok = false;
            break;
          }
          tc_fence_after();
          // target planes i - 2 .. i (source plane i - 1) of the 8
          const int lo = max(0, i - 2), hi = min(UT_BX - 1, i);
          const uint32_t idesc = f16_idesc(128, 32 * (hi - lo + 1));
          const uint32_t d = dset + (uint32_t)(32 * lo);
          // descriptors differ only in their start address (16-byte units, no
          // carry: shared memory is below 256 KB)
          const uint64_t a0 = kmajor_desc(smem_u32(astage + s * UT_ASTAGE), UT_PART, 128);
          const uint64_t b0 = kmajor_desc(bb + (uint32_t)((lo - (i - 2)) * 32 * 16), UT_BPLANE, 128);
#pragma unroll
          for (int q = 0; q < 9; ++q) {  // (D_y, D_z)
            const uint64_t ah = a0 + (((q / 3) * UT_LINEB + (q % 3) * 8 * 16) >> 4);
            const uint64_t bd = b0 + ((q * UT_BTILE) >> 4);
            tc_mma_f16(d, ah, bd, idesc, 1u);
            tc_mma_f16(d, ah + ((2 * UT_PART) >> 4), bd, idesc, 1u);
          }
          tc_commit(&s_empty[s]);
          ++li;
        }
        if (!ok) break;
        tc_commit(&s_accf[ab]);
        ++it;
      }
      if (!ok) *s_abort = 1;
      // MMAs complete in order: the last stage commit covers all of them
      if (li > 0 && !mbar_wait(&s_empty[(li - 1) % UT_NST], ((li - 1) / UT_NST) & 1, nullptr))
        *s_abort = 1;
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------ drains
    const int row = 32 * (warp & 3) + lane;  // TMEM lane: (z, column) of the target lines
    const int tz = row >> 3, col = row & 7;
    const uint32_t lb = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
    const float zero[16] = {};
    const float ua = exp2i(-unif_scale_exp(__ldg(a.amax + col)));  // undoes the column's scale
    const uint64_t* t8 = reinterpret_cast<const uint64_t*>(a.tocc);
    const int64_t tstride = (int64_t)S * S * 8;  // outputs between children
    int it = 0;
    for (int w = blockIdx.x; w < nitems; w += gridDim.x) {
      const Item t = item_of(w);
      if (!has_targets(t)) continue;
      const int ab = it & 1;
      const int z = t.zb * UT_LINE + tz;
      const float ub = exp2i(-__ldg(a.bexp + t.slot));
      uint64_t occ[UT_BX];
#pragma unroll
      for (int x = 0; x < UT_BX; ++x) occ[x] = __ldg(t8 + morton_encode(t.x0 + x, t.y, z));
      // one thread waits for the accumulators; the barrier-with-reduction
      // releases the other drain threads (uniformly: the TMEM loads below
      // are warp-collective)
      bool bad = false;
      if (tid == UT_DRAIN0 && !mbar_wait_sleep(&s_accf[ab], (it >> 1) & 1, s_abort, piters))
        bad = true;
      if (drains_any(bad)) {
        *s_abort = 1;
        break;
      }
      tc_fence_after();
      float2* y0 = a.Y + (int64_t)t.slot * UnifPlanes::slot_outputs(S) +
                   UnifPlanes::out_index(S, t.x0, 0, t.y, z, col);
#pragma unroll
      for (int x = 0; x < UT_BX; ++x) {
        const uint32_t ta = lb + (uint32_t)(ab * UT_BX * 32 + 32 * x);
        uint32_t h[16], l[16];
        tc_ld16_wait(ta, h);
        tc_ld16_wait(ta + 16, l);
        tc_st16(ta, zero);
        tc_st16(ta + 16, zero);
#pragma unroll
        for (int c = 0; c < 8; ++c)
          if ((occ[x] >> (8 * c)) & 0xffu)
            y0[(x * 8 + c) * tstride] = make_float2(
                (__uint_as_float(h[2 * c]) + __uint_as_float(l[2 * c])) * ua * ub,
                (__uint_as_float(h[2 * c + 1]) + __uint_as_float(l[2 * c + 1])) * ua * ub);
      }
      tc_wait_st();
      tc_fence_before();
      group_sync(2, 128);  // every drain thread's loads and stores
      if (tid == UT_DRAIN0) mbar_arrive(&s_acce[ab]);
      ++it;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (tid == 0 && *s_abort && a.err) atomicExch(a.err, 1);
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem),
                 "r"(UT_TMEM_COLS)
                 : "memory");
  }
}

// Operator tiles of the tensor-core MAC from the spectra op[lvl][k][343]
// (complex, lex-indexed offsets, inner 27 zero): for each level and frequency
// slot nine tiles (D_y, D_z), each [kcore 2][row 96][8 halves], row = 32 dxi +
// 16 part + 2 t + ri_out (D_x = 1 - dxi; part 0: F16 hi, 1: lo), element
// K = 8 kcore + e = 2 s + ri_in, value the real form of E[o] with
// o = 2 D + bits(s) - bits(t):  (re, re) = a, (im, re) = -b, (re, im) = b,
// (im, im) = a for E = a + i b, zero where o is near; every value of a
// frequency scaled by 2^sB (bexp), sB putting the largest in [2^14, 2^15).
void unif_tc_tiles(int n, const std::vector<double>& op, int nlev, std::vector<uint16_t>* tiles,
                   std::vector<int>* bexp) {
  const int m = 2 * n - 1, nfull = m * m * n, nk = unif_slots(n);
  tiles->assign((size_t)nlev * nk * kUnifTcTileHalves, 0);
  bexp->assign((size_t)nlev * nk, 0);
  parallel_for((int64_t)nlev * nk, [&](int64_t b0, int64_t b1) {
    std::vector<float> val(UT_BFREQ / 4);  // float32 values of the hi slots, tile order
    for (int64_t b = b0; b < b1; ++b) {
      const double* E = &op[(size_t)(b / nk * nfull + unif_slot_freq(n, (int)(b % nk))) * 343 * 2];
      float vmax = 0.f;
      for (int tile = 0; tile < 9; ++tile) {
        const int dyi = tile / 3, dzi = tile % 3;
        for (int row = 0; row < UT_BROWS; ++row) {
          const int dxi = row / 32, part = (row / 16) & 1, t = (row & 15) >> 1, ro = row & 1;
          if (part) continue;
          const int D[3] = {1 - dxi, dyi - 1, dzi - 1};
          for (int kk = 0; kk < 16; ++kk) {
            const int s = kk >> 1, ri = kk & 1;
            int o[3], far = 0;
            for (int d = 0; d < 3; ++d) {
              o[d] = 2 * D[d] + ((s >> (2 - d)) & 1) - ((t >> (2 - d)) & 1);
              far |= o[d] > 1 || o[d] < -1;
            }
            float v = 0.f;
            if (far) {
              const int lex = 49 * (o[0] + 3) + 7 * (o[1] + 3) + (o[2] + 3);
              const double re = E[2 * lex], im = E[2 * lex + 1];
              v = (float)(ri == ro ? re : (ri ? -im : im));
            }
            val[(size_t)(tile * 48 + dxi * 16 + (row & 15)) * 16 + kk] = v;
            vmax = std::max(vmax, std::fabs(v));
          }
        }
      }
      int e = 0;
      if (vmax > 0.f && std::isfinite(vmax)) {
        int k2;
        std::frexp(vmax, &k2);
        e = std::max(-126, std::min(127, 15 - k2));
      }
      (*bexp)[b] = e;
      uint16_t* dst = tiles->data() + (size_t)b * kUnifTcTileHalves;
      for (int tile = 0; tile < 9; ++tile)
        for (int row = 0; row < UT_BROWS; ++row) {
          const int dxi = row / 32, part = (row / 16) & 1;
          for (int kk = 0; kk < 16; ++kk) {
            const float x = std::ldexp(val[(size_t)(tile * 48 + dxi * 16 + (row & 15)) * 16 + kk], e);
            const __half xh = __float2half_rn(x);
            const __half xv = part ? __float2half_rn(x - __half2float(xh)) : xh;
            memcpy(&dst[tile * (UT_BTILE / 2) + (kk >> 3) * (UT_BPLANE / 2) + row * 8 + (kk & 7)],
                   &xv, 2);
          }
        }
    }
  });
}

bool unif_tc_eligible(const pbbfmm_tree* t, int l, int C) {
  return t->use_tc && t->f_unif_tiles && t->f_unif_bexp && (C % 8) == 0 && l >= 5 && l <= 10;
}

// ws.occ: source and target occupancy of the cells, then the line flags of
// k_unif_lines; ws.amax: a level's column bounds.
int run_unif_tc_occupancy(pbbfmm_tree* t, int l, uint8_t** socc, uint8_t** tocc, cudaStream_t st) {
  const int64_t ncells = cells_at(l);
  const int S = 1 << (l - 1), nlines = S * S * (S / UT_LINE);
  Workspace& ws = t->ws;
  if (int rc = grow(ws.occ, 2 * (size_t)ncells + 2 * (size_t)nlines)) return rc;
  if (int rc = grow(ws.amax, 8 * sizeof(uint32_t))) return rc;
  *socc = ws.occ.as<uint8_t>();
  *tocc = *socc + ncells;
  const int span = (int)cells_at(t->p.tree_level - l);
  const unsigned g = (unsigned)((ncells + 255) / 256);
  k_occupancy<<<g, 256, 0, st>>>(ws.sstart_p, span, ncells, *socc);
  k_occupancy<<<g, 256, 0, st>>>(ws.tstart.as<int>(), span, ncells, *tocc);
  k_unif_lines<<<(unsigned)((nlines + 127) / 128), 128, 0, st>>>(*socc, *tocc, S, *tocc + ncells,
                                                               *tocc + ncells + nlines);
  PB_LAUNCH_N("occupancy", 3);
  return PBBFMM_OK;
}

int run_unif_tc_borders(pbbfmm_tree* t, int S, unsigned char* X, cudaStream_t st) {
  const int per = 2 * ((S + 2) * 8 + 8) + (S - 1) * 16, nparts = t->nk * S * 4;
  k_unif_borders<<<dim3((unsigned)((per + 255) / 256), (unsigned)std::min(nparts, 65535)), 256, 0,
                   st>>>(X, S, nparts);
  PB_LAUNCH("unif_borders");
  return PBBFMM_OK;
}

// Level l of the tensor-core MAC, one group of 8 columns: Y = sum_D B X.
int run_m2l_unif_tc_level(pbbfmm_tree* t, int l, int lvl, const unsigned char* X, float2* Y,
                          const uint32_t* amax, const uint8_t* tocc, cudaStream_t st) {
  if (!t->d_tc_err) {
    set_error("tensor-core uniform M2L: the tree has no timeout flag");
    return PBBFMM_ERR_STATE;
  }
  PB_CUDA(cudaFuncSetAttribute(k_m2l_unif_tc, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               UT_SMEM));
  const int S = 1 << (l - 1), nk = t->nk;
  UnifTcArgs a{};
  a.X = X;
  a.Y = Y;
  a.tiles = t->f_unif_tiles + (size_t)lvl * nk * kUnifTcTileHalves;
  a.bexp = t->f_unif_bexp + (size_t)lvl * nk;
  a.amax = amax;
  a.tocc = tocc;
  a.line = tocc + cells_at(l);
  a.item = a.line + (int64_t)S * S * (S / UT_LINE);
  a.S = S;
  a.nk = nk;
  a.nblocks = (S / UT_BX) * S * (S / UT_LINE);
  a.err = t->d_tc_err;
  int nsm = 148;
  PB_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, t->device));
  k_m2l_unif_tc<<<(unsigned)nsm, UT_THREADS, UT_SMEM, st>>>(a);
  PB_LAUNCH("m2l_unif_tc");
  return PBBFMM_OK;
}

int set_unif_tc_wait_limit(long long polls) {
  PB_CUDA(cudaMemcpyToSymbol(g_unif_wait_iters, &polls, sizeof(polls)));
  return PBBFMM_OK;
}

}  // namespace pbbfmm


