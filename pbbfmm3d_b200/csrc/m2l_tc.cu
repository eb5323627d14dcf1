// Chebyshev M2L of the mixed-precision path on the 5th-generation tensor
// cores (tcgen05 with TMEM accumulators), in split precision:
//     D += A_lo B_hi + A_hi B_lo + A_hi B_hi,
// with x = hi + lo, accumulated in float32.  Two operand formats:
//   F16  (default): x scaled by a power of two 2^e (one e per proxy row and
//        one per operator, so that the largest magnitude lies in
//        [2^14, 2^15)), hi = fp16(x 2^e), lo = fp16(x 2^e - hi);
//        kind::f16, K = 16 per instruction.  Elements down to 2^-17 of their
//        row's largest keep 22 significant bits; smaller ones an absolute
//        error below 2^-39 of it.  Each offset's accumulator is unscaled by
//        2^-(e_row + e_op) (exact) when it is drained.
//   TF32: hi = tf32(x), lo = tf32(x - hi); kind::tf32, K = 8 per instruction.
// Either way the dropped A_lo B_lo term and the splitting leave a relative
// error near 2^-21 per product.  F16 moves half the bytes and issues half the
// instructions per useful product.  The float32 accumulation inside the
// tensor pipe loses about one unit in the last place per accumulation step,
// so accumulators are drained into a running sum every few offsets (every
// offset for F16, see `group`), which keeps the result within ~1e-6 of float64.
//
// Same product as k_m2l_cheb (reference: FarFieldInteractions / Moment2Local,
// include/compute.hpp:402-508 and 881-914): for a tile of targets of one
// level that share their child type, D[(target, col)][f] = sum over the 189
// offsets o of sum_s proxy_{target+o}[col][s] E_o[f][s].
//
//   M = 128 rows (target, col) of one child type,  N = rf padded to 16,
//   K = (offsets with a source in the tile) x (rs padded to 32).
//
// Operands are K-major, 128-byte-swizzled tiles (rows of 128 bytes: 32 TF32 or
// 64 F16 values; groups of 8 rows 1024 bytes apart), A filled with cp.async
// (zero-fill for absent sources) and B by TMA, in NST stages.  Every wait is bounded: on timeout the kernel sets
// *err, waits (bounded) for its last MMAs, frees its TMEM and returns.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cstdlib>
#include <mutex>

#include "cheb_kara.cuh"
#include "fmm.cuh"
#include "tcgen05.cuh"

namespace pbbfmm {

constexpr int TC_M = 128;
constexpr int TC_ROWB = 128;       // bytes of K per stage: one 128-byte swizzle row
constexpr int TC_PRODUCERS = 128;  // warps 0-3: operand loads
constexpr int TC_MMA_WARP = 4;     // warp 4: TMEM allocation, MMA issue (one thread)
constexpr int TC_THREADS = 288;    // + warps 5-8: accumulator drains
constexpr int TC_TMEM_COLS = 512;  // columns allocated (accumulators and running sum)
// Poll limit of the M2L kernel's pipeline waits (stage and accumulator
// barriers inside its main loops), per device; kWaitIters unless a test
// lowers it through pbbfmm_debug_set_pipeline_wait_limit to make those waits
// run out.  The waits for committed copies and MMAs before a CTA exits always
// keep the full bound.
__device__ long long g_pipe_wait_iters = kWaitIters;

// One part of the launch (ChebPart): a level's tiles of each child type, or (mult
// > 0, dense levels, cheb_kara.cuh) of each combination of the children, whose rows
// are (parent, combination, column) and whose offsets are 26 parent offsets.
struct TcLevel {
  const int* typed;                // targets by child type; combined: target parents
  const unsigned char *ph, *pl;    // proxy hi / lo, rows of rowb bytes
  const int* pexp;                 // F16: scale exponent of each row
  float* pf;                       // output rows of rf floats
  int lev, span, item0;            // item0: first tile of the level
  int mult;                        // 0: direct; combined: combinations from j0 on (start[1] tiles each)
  int j0, C;                       // C: columns of the rows
  int op0;                         // first operator of the level
  int start[9];                    // first tile of each type; start[8] = total tiles
  int first[8];                    // first list position of each type
  int count[8];                    // targets of each type
};
struct TcArgs {
  TcLevel lv[kChebParts];
  int nlev, rf, NP, rowb, group;
  const int* sstart;
  const int* offs;                 // [8][189], then [27][26] (ox, oy, oz, operator)
  const int *eexp, *kexp;          // F16: scale exponents of the operators / combined ones
  int* err;
};

// Stage layout: A_hi 16 KB | A_lo 16 KB | B_hi NP*128 | B_lo NP*128, each
// part 1024-byte aligned (NP is a multiple of 16).
__host__ __device__ constexpr int tc_stage_bytes(int NP) { return 2 * 16384 + 2 * NP * 128; }
__host__ __device__ constexpr int tc_smem_bytes(int NP, int nst) {
  return nst * tc_stage_bytes(NP) + 1024;
}

// TMEM columns (512 allocated): accumulator b at b * stride.  With the
// running sum in registers (N <= TC_REG_SUM) four accumulators take turns;
// otherwise two, and when a third region fits (N <= 160) a running sum at
// 2 * stride that the drains update inside TMEM, so that pf is written once;
// beyond that drains add into pf.
__host__ __device__ constexpr int tc_acc_stride(int NP) { return NP <= 160 ? (NP + 31) / 32 * 32 : 256; }
__host__ __device__ constexpr bool tc_sum_in_tmem(int NP) { return NP <= 160; }
// Up to this many columns the running sum lives in the drain threads'
// registers (the CTA is alone on its SM, so they cost no occupancy).
constexpr int TC_REG_SUM = 128;

// One CTA per tile of 128 (target, col) rows of one child type (or
// combination); NST stages; the tiles of all levels in one launch (a level
// alone leaves a last wave that is nearly empty, the shallow ones a single one).
// One launch and the combinations, against a launch per level on direct lists:
// M2L of 4M clustered points, order 6: 18.1 -> 15.3 ms; of 250,000 points, r =
// 125, 4 columns, forward and adjoint: 7.7 -> 4.4 ms (and 0.35 ms more for the
// split, which forms the combinations).
//   tm_eh, tm_el : [operator][NP] rows of hi / lo of E_o^T (row f holds
//                  E_o[f][s] over s), zero padded to rowb bytes;
//   tm_kh, tm_kl : the same of the combined operators
//   proxies, exponents and outputs: TcLevel (pexp and the proxy rows are read
//   for nonempty source cells only)
// Warp roles:
//   warps 0-3  producers: each warp gathers its 32 rows of A with cp.async and
//              signals the stage's full barrier when its copies land
//              (cp.async.mbarrier.arrive); one thread of warp 0 also loads B
//              (the operator tile, hi and lo) with two TMA copies;
//   warp 4     allocates TMEM; one thread waits for full stages, issues the
//              MMAs and commits them to the stage's empty barrier;
//   warps 5-8  drain accumulators into the running sum (TMEM lane quadrant
//              warp % 4).
// NACC TMEM accumulators (four with the register running sum, else two) take
// turns, one per group of `group` consecutive offsets, so every float32
// accumulation chain inside the tensor pipe spans at most `group` offsets;
// an accumulator is reused NACC groups later, once drained (the commit that
// releases a group's accumulator to the drains arrives well after its MMAs
// are issued, so two accumulators left the MMA thread waiting for drains).
//   s_full[s]  : 128 producer arrivals, one per thread, when its copies land
//   s_tfull[s] : the operator tile's TMA bytes (thread 0's expect_tx)
//   s_empty[s] : MMAs reading stage s done (tcgen05.commit)
//   s_accf[b]  : MMAs of accumulator b's group done (tcgen05.commit)
//   s_acce[b]  : accumulator b drained (128 drainer arrivals)
template <int NST, bool F16, bool RSUM>
__global__ void __launch_bounds__(TC_THREADS, 1)
    k_m2l_cheb_tc(const __grid_constant__ CUtensorMap tm_eh,
                  const __grid_constant__ CUtensorMap tm_el,
                  const __grid_constant__ CUtensorMap tm_kh,
                  const __grid_constant__ CUtensorMap tm_kl, const __grid_constant__ TcArgs a) {
  extern __shared__ unsigned char smraw[];
  int li = 0;
  for (int i = 1; i < a.nlev; ++i)
    if ((int)blockIdx.x >= a.lv[i].item0) li = i;
  const TcLevel& lv = a.lv[li];
  const int rf = a.rf, NP = a.NP, rowb = a.rowb, C = lv.C, lev = lv.lev, span = lv.span;
  const int group = a.group, mult = max(lv.mult, 1);
  const bool kara = lv.mult > 0;
  const int* __restrict__ sstart = a.sstart;
  const int* __restrict__ typed = lv.typed;
  const unsigned char* __restrict__ Ph = lv.ph;
  const unsigned char* __restrict__ Pl = lv.pl;
  const int* __restrict__ pexp = lv.pexp;
  float* __restrict__ pf = lv.pf;
  int* __restrict__ err = a.err;
  const int tile = (int)blockIdx.x - lv.item0;
  const int bbytes = NP * 128;
  const int stage_bytes = tc_stage_bytes(NP);
  unsigned char* base = smraw + ((1024 - (smem_u32(smraw) & 1023)) & 1023);
  constexpr int NACC = RSUM ? 4 : 2;  // TMEM accumulators (4 x 128 columns at most)
  __shared__ uint64_t s_full[NST], s_tfull[NST], s_empty[NST], s_accf[NACC], s_acce[NACC];
  __shared__ uint32_t s_tmem;
  __shared__ int s_cell[TC_M];     // target cell of each row, or -1
  __shared__ int s_xyz[TC_M];      // target coordinates, x << 20 | y << 10 | z
  __shared__ uint32_t s_valid[6];  // bit o: some target of the tile has a source at offset o
  __shared__ uint32_t s_tmask[TC_M][6];  // per target of the tile: bit o = source at offset o
  __shared__ int4 s_off[189];      // valid offsets: (ox, oy, oz, operator index)
  __shared__ uint8_t s_oidx[189];  // valid offset q: its index o in the type's list
  __shared__ int s_oexp[189];      // F16: valid offset q: its operator's scale exponent
  __shared__ int s_nvalid;
  __shared__ int s_abort_flag;
  volatile int* s_abort = &s_abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long long piters = g_pipe_wait_iters;  // poll limit of the pipeline waits

  // child type (or combination) of this tile
  int type = 0, tstart = 0, tlist = 0, tcount = 0, noff = 189, comb = 0;
  const int* my_offs = a.offs;
  if (kara) {
    type = comb = tile / lv.start[1];
    tstart = type * lv.start[1];
    tcount = lv.count[0];
    noff = kKaraD;
    my_offs += 4 * (8 * 189 + (lv.j0 + type) * kKaraD);
  } else {
    for (int i = 1; i < 8; ++i)
      if (tile >= lv.start[i]) type = i;
    tstart = lv.start[type];
    tlist = lv.first[type];
    tcount = lv.count[type];
    my_offs += type * 189 * 4;
  }
  const int per_tile = TC_M / C;
  const int tfirst = (tile - tstart) * per_tile;
  const int ntile = min(per_tile, tcount - tfirst);
  const int nside = 1 << lev;

  if (tid < TC_M) {
    const int cell = (tid < per_tile * C && tid / C < ntile) ? typed[tlist + tfirst + tid / C] : -1;
    int x = 0, y = 0, z = 0;
    if (cell >= 0) morton_decode((uint32_t)cell, &x, &y, &z);
    s_cell[tid] = cell;
    s_xyz[tid] = (x << 20) | (y << 10) | z;
  }
  if (tid < 6) s_valid[tid] = 0;
  for (int i = tid; i < TC_M * 6; i += TC_THREADS) (&s_tmask[0][0])[i] = 0;
  if (warp == TC_MMA_WARP) {  // 128 lanes x 512 float32 columns
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                     smem_u32(&s_tmem)),
                 "r"(TC_TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  if (tid == 0) {
    for (int i = 0; i < NST; ++i) {
      mbar_init(&s_full[i], TC_PRODUCERS);
      mbar_init(&s_tfull[i], 1);
      mbar_init(&s_empty[i], 1);
    }
    for (int b = 0; b < NACC; ++b) {
      mbar_init(&s_accf[b], 1);
      mbar_init(&s_acce[b], TC_M);
    }
    s_abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  // which (target, offset) pairs of the tile have a source cell: all threads,
  // one pair per item, independent loads
#pragma unroll 4
  for (int i = tid; i < ntile * noff; i += TC_THREADS) {
    const int tg = i / noff, o = i - tg * noff;
    const int xyz = s_xyz[tg * C];
    const int bx = (xyz >> 20) + my_offs[4 * o], by = ((xyz >> 10) & 1023) + my_offs[4 * o + 1],
              bz = (xyz & 1023) + my_offs[4 * o + 2];
    if (bx < 0 || by < 0 || bz < 0 || bx >= nside || by >= nside || bz >= nside) continue;
    const uint32_t bm = morton_encode(bx, by, bz);
    if (sstart[(int64_t)(bm + 1) * span] > sstart[(int64_t)bm * span]) {
      atomicOr(&s_tmask[tg][o >> 5], 1u << (o & 31));
      atomicOr(&s_valid[o >> 5], 1u << (o & 31));
    }
  }
  __syncthreads();
  if (tid == 0) {
    int nv = 0;
    for (int o = 0; o < noff; ++o)
      if ((s_valid[o >> 5] >> (o & 31)) & 1) {
        s_oidx[nv] = (uint8_t)o;
        s_off[nv++] = make_int4(my_offs[4 * o], my_offs[4 * o + 1], my_offs[4 * o + 2],
                                my_offs[4 * o + 3]);
      }
    s_nvalid = nv;
  }
  __syncthreads();
  if constexpr (F16)
    for (int q = tid; q < s_nvalid; q += TC_THREADS)
      s_oexp[q] = (kara ? a.kexp : a.eexp)[lv.op0 + s_off[q].w];
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem;
  const int nvalid = s_nvalid;
  const int kchunks = rowb / TC_ROWB;
  const int niter = nvalid * kchunks;
  const int group_iters = max(group, 1) * kchunks;
  const int ngroups = (niter + group_iters - 1) / group_iters;

  if (warp < TC_PRODUCERS / 32) {
    // ---------------------------------------------------------------- producers
    // Lane l copies 16-byte chunk (l & 7) of rows 4 warp + (l >> 3) + 16 i of
    // A (i < 8) and B (i < NP / 16): four 128-byte rows per warp instruction.
    // Lane l also owns A row 4 warp + (l & 3) + 16 (l >> 2): it finds that
    // row's source once per offset (from the tile's source mask: no global
    // load) and the lanes copying the row fetch the result by shuffle.
    const int own = 4 * warp + (lane & 3) + 16 * (lane >> 2);
    const int ocell = s_cell[own], ocol = own % C, otg = own / C;
    const int ox = s_xyz[own] >> 20, oy = (s_xyz[own] >> 10) & 1023, oz = s_xyz[own] & 1023;
    const int ch = lane & 7, r0 = 4 * warp + (lane >> 3);
    const uint32_t soff0 = sw128_off(r0, ch);  // row r0 + 16 i lies 2048 i bytes further
    int cur_q = -1;
    long long cur_row = -1;  // this lane's own row: source row offset or -1
    int tma_last[NST];       // the TMA thread: last iteration whose TMA went into each stage
#pragma unroll
    for (int i = 0; i < NST; ++i) tma_last[i] = -1;
    for (int j = 0; j < niter; ++j) {
      const int s = j % NST;
      // warp-uniform: the shuffles below are warp-collective
      if (j >= NST &&
          !__all_sync(0xffffffffu, mbar_wait_sleep(&s_empty[s], (j / NST - 1) & 1, s_abort, piters))) {
        *s_abort = 1;
        break;
      }
      const int q = j / kchunks, kc = j - q * kchunks;
      if (q != cur_q) {
        const int o = s_oidx[q];
        cur_row = -1;
        if (ocell >= 0 && ((s_tmask[otg][o >> 5] >> (o & 31)) & 1)) {
          const int4 d = s_off[q];
          cur_row = (((long long)morton_encode(ox + d.x, oy + d.y, oz + d.z) * mult + comb) * C +
                     ocol) * rowb;
        }
        cur_q = q;
      }
      unsigned char* st = base + s * stage_bytes;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const long long rr = __shfl_sync(0xffffffffu, cur_row, (lane >> 3) | (i << 2));
        const bool ok = rr >= 0;
        const int64_t off = ok ? rr + kc * TC_ROWB + 16 * ch : 0;
        cp_async16(st + soff0 + 2048 * i, Ph + off, ok ? 16 : 0);
        cp_async16(st + 16384 + soff0 + 2048 * i, Pl + off, ok ? 16 : 0);
      }
      if (warp == 0 && elect_one()) {
        // the operator tile (NP rows x 128 bytes, hi and lo) by TMA; x in
        // elements: 64 per 128 bytes for F16, 32 for TF32
        const int y = (lv.op0 + s_off[q].w) * NP;
        const int x = kc * (F16 ? 64 : 32);
        mbar_arrive_expect_tx(&s_tfull[s], 2u * NP * 128u);
        tma_load_2d(st + 32768, kara ? &tm_kh : &tm_eh, x, y, &s_tfull[s]);
        tma_load_2d(st + 32768 + bbytes, kara ? &tm_kl : &tm_el, x, y, &s_tfull[s]);
        tma_last[s] = j;
      }
      cp_async_arrive(&s_full[s]);
    }
    cp_async_wait_all();
    // no TMA may still be writing when the CTA ends: wait (bounded) for the
    // last load issued into each stage
    __syncwarp();
    if (warp == 0 && elect_one())
      for (int s2 = 0; s2 < NST; ++s2)
        if (tma_last[s2] >= 0 && !mbar_wait(&s_tfull[s2], (tma_last[s2] / NST) & 1, nullptr))
          *s_abort = 1;
  } else if (warp == TC_MMA_WARP) {
    // ---------------------------------------------------------------- MMA issue
    if (elect_one()) {
      const uint32_t idesc = F16 ? f16_idesc(TC_M, NP) : tf32_idesc(TC_M, NP);
      const int astride = tc_acc_stride(NP);
      int last = -1;  // last iteration whose MMAs were committed
      for (int it = 0; it < niter; ++it) {
        const int s = it % NST;
        const int g = it / group_iters;
        const bool fresh = it == g * group_iters;
        // accumulator g % NACC is free once the drain of group g - NACC is done
        const int ab = g % NACC;
        if (fresh && g >= NACC &&
            !mbar_wait_sleep(&s_acce[ab], ((g - NACC) / NACC) & 1, s_abort, piters)) {
          *s_abort = 1;
          break;
        }
        if (!mbar_wait_sleep(&s_full[s], (it / NST) & 1, s_abort, piters) ||
            !mbar_wait_sleep(&s_tfull[s], (it / NST) & 1, s_abort, piters)) {
          *s_abort = 1;
          break;
        }
        fence_async_smem();  // the producers' copies, seen through the barrier, to the async proxy
        tc_fence_after();
        const uint32_t a_hi = smem_u32(base + s * stage_bytes), a_lo = a_hi + 16384;
        const uint32_t b_hi = a_hi + 32768, b_lo = b_hi + bbytes;
        const uint32_t d = tmem + (uint32_t)(ab * astride);
        // four K steps of 32 bytes (16 F16 or 8 TF32 values) per 128-byte row
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint32_t off = k * 32;
          if constexpr (F16) {
            tc_mma_f16(d, sw128_desc(a_lo + off), sw128_desc(b_hi + off), idesc,
                       (fresh && k == 0) ? 0u : 1u);
            tc_mma_f16(d, sw128_desc(a_hi + off), sw128_desc(b_lo + off), idesc, 1u);
            tc_mma_f16(d, sw128_desc(a_hi + off), sw128_desc(b_hi + off), idesc, 1u);
          } else {
            tc_mma_tf32(d, sw128_desc(a_lo + off), sw128_desc(b_hi + off), idesc,
                        (fresh && k == 0) ? 0u : 1u);
            tc_mma_tf32(d, sw128_desc(a_hi + off), sw128_desc(b_lo + off), idesc, 1u);
            tc_mma_tf32(d, sw128_desc(a_hi + off), sw128_desc(b_hi + off), idesc, 1u);
          }
        }
        tc_commit(&s_empty[s]);
        if (it + 1 == niter || it + 1 == (g + 1) * group_iters) tc_commit(&s_accf[ab]);
        last = it;
      }
      // Before the TMEM is freed: MMAs complete in order, so the last commit
      // covers all of them (waited for even after an abort, still bounded).
      if (last >= 0 && !mbar_wait(&s_empty[last % NST], (last / NST) & 1, nullptr)) *s_abort = 1;
    }
    __syncwarp();
  } else {
    // ---------------------------------------------------------------- drainers
    const int row = 32 * (warp & 3) + lane;  // TMEM lane quadrant of this warp
    const int cell = s_cell[row];
    float* dst = cell >= 0 ? pf + (((int64_t)cell * mult + comb) * C + row % C) * rf : nullptr;
    const uint32_t lane_base = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
    const int astride = tc_acc_stride(NP);
    const bool tsum = tc_sum_in_tmem(NP);
    const uint32_t sum_base = lane_base + (uint32_t)(2 * astride);
    // F16 (one offset per group): the unscaling exponent of this row at offset
    // q is e_op + e_row of its source.  The row's exponent is loaded two
    // offsets ahead, unconditionally (index 0 when the row has no source at q,
    // the flag then marks it unused), so that no instruction waits for the
    // load before the offset's drain.
    const int rcol = row % C;
    const int rx = s_xyz[row] >> 20, ry = (s_xyz[row] >> 10) & 1023, rz = s_xyz[row] & 1023;
    const int rtg = row / C;
    auto has_src = [&](int q) -> bool {
      if (!F16 || q >= nvalid || cell < 0) return false;
      const int oi = s_oidx[q];
      return (s_tmask[rtg][oi >> 5] >> (oi & 31)) & 1;
    };
    auto src_row = [&](int q, bool ok) -> int64_t {
      if (!ok) return 0;
      const int4 o = s_off[q];
      return ((int64_t)morton_encode(rx + o.x, ry + o.y, rz + o.z) * mult + comb) * C + rcol;
    };
    bool v1 = has_src(0), v2 = has_src(1);
    int x1 = F16 ? pexp[src_row(0, v1)] : 0, x2 = F16 && nvalid > 1 ? pexp[src_row(1, v2)] : 0;
    float rsum[RSUM ? TC_REG_SUM : 1];  // running sum (RSUM: NP <= TC_REG_SUM)
#pragma unroll
    for (int i = 0; i < (RSUM ? TC_REG_SUM : 1); ++i) rsum[i] = 0.f;
    for (int g = 0; g < ngroups; ++g) {
      const int b = g % NACC;
      // the unscaling 2^-e, e = e_op + e_row, as two exact powers of two
      // 2^-e1 2^-e2 with e1 in [-126, 126] (a normal number) and the rest in
      // e2 (normal or subnormal): a sum beyond one float's exponent range
      // still scales correctly as long as the result itself is a normal
      // number; rows without a source are zero (any scale)
      const int e = v1 ? s_oexp[g] + min(max(x1, -256), 256) : 0;
      const int e1 = min(max(e, -126), 126), e2 = min(max(e - e1, -126), 149);
      const float sc = __int_as_float((127 - e1) << 23);
      const float sc2 = e2 <= 126 ? __int_as_float((127 - e2) << 23) : __int_as_float(1 << (149 - e2));
      v1 = v2;
      x1 = x2;
      v2 = has_src(g + 2);
      if (F16 && g + 2 < nvalid) x2 = pexp[src_row(g + 2, v2)];
      // warp-uniform: the TMEM loads below are warp-collective
      if (!__all_sync(0xffffffffu, mbar_wait_sleep(&s_accf[b], (g / NACC) & 1, s_abort, piters))) {
        *s_abort = 1;
        break;
      }
      tc_fence_after();
      if constexpr (RSUM) {
        // batches of 16 columns (one wait each) added into the register sum;
        // the accumulator is released once its last batch is in registers
#pragma unroll
        for (int c = 0; c < TC_REG_SUM / 16; ++c) {
          if (c * 16 >= NP) break;
          uint32_t r[16];
          tc_ld16_wait(lane_base + (uint32_t)(b * astride + c * 16), r);
          if ((c + 1) * 16 >= NP) {
            tc_fence_before();
            mbar_arrive(&s_acce[b]);
          }
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float x = __uint_as_float(r[i]);
            rsum[c * 16 + i] = F16 ? fmaf(x * sc, sc2, rsum[c * 16 + i]) : rsum[c * 16 + i] + x;
          }
        }
        continue;
      } else {
      const bool final_group = g + 1 == ngroups;
      float v[16], u[16];
      for (int n0 = 0; n0 < NP; n0 += 16) {
        tc_ld16(lane_base + (uint32_t)(b * astride + n0), v);
        if constexpr (F16) {
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = v[i] * sc * sc2;  // exact unless the result is subnormal
        }
        if (tsum) {
          if (g > 0) {
            tc_ld16(sum_base + (uint32_t)n0, u);
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] += u[i];
          }
          if (!final_group) {
            tc_st16(sum_base + (uint32_t)n0, v);
          } else if (dst) {
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (n0 + i < rf) dst[n0 + i] = v[i];
          }
        } else if (dst) {
#pragma unroll
          for (int i = 0; i < 16; ++i)
            if (n0 + i < rf) dst[n0 + i] = g == 0 ? v[i] : dst[n0 + i] + v[i];
        }
      }
      if (tsum && !final_group) tc_wait_st();
      tc_fence_before();
      mbar_arrive(&s_acce[b]);
      }
    }
    if constexpr (RSUM) {
      if (dst)
#pragma unroll
        for (int i = 0; i < TC_REG_SUM; ++i)
          if (i < rf) dst[i] = rsum[i];
    } else if (ngroups == 0 && dst) {  // no source in any interaction list of the tile
      for (int n = 0; n < rf; ++n) dst[n] = 0.f;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (tid == 0 && *s_abort && err) atomicExch(err, 1);
  if (warp == TC_MMA_WARP) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem),
                 "r"(TC_TMEM_COLS)
                 : "memory");
  }
}

// Split the proxies of the listed source cells into TF32 hi / lo rows of KP
// floats (zero padded from rs): thread per (row, k).  (TF32 operands.)
__global__ void k_split_proxy(const int* __restrict__ cells, int64_t nrows, int C, int rs, int KP,
                              const float* __restrict__ proxy, float* __restrict__ ph,
                              float* __restrict__ pl) {
  const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e >= nrows * KP) return;
  const int64_t r = e / KP;
  const int k = (int)(e - r * KP);
  const int64_t row = (int64_t)cells[r / C] * C + r % C;
  const float v = k < rs ? proxy[row * rs + k] : 0.f;
  const float h = to_tf32(v);
  ph[row * KP + k] = h;
  pl[row * KP + k] = to_tf32(v - h);
}

// F16 operands: split the proxies of the listed source cells into scaled F16
// hi / lo rows of KP values (zero padded from rs) and the row's exponent e,
// chosen so that the row's largest |x| 2^e lies in [2^14, 2^15) (e = 0 for a
// zero row): one warp per row.
__global__ void k_split_proxy_f16(const int* __restrict__ cells, int64_t nrows, int C, int rs,
                                  int KP, const float* __restrict__ proxy, __half* __restrict__ ph,
                                  __half* __restrict__ pl, int* __restrict__ pexp) {
  const int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (r >= nrows) return;  // uniform over the warp
  const int64_t row = (int64_t)cells[r / C] * C + r % C;
  const float* x = proxy + row * rs;
  float m = 0.f;
  for (int k = lane; k < rs; k += 32) m = fmaxf(m, fabsf(x[k]));
#pragma unroll
  for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  const int e = m > 0.f ? 15 - exponent_of(m) : 0;  // m in [2^(k2-1), 2^k2)
  for (int k = lane; k < KP; k += 32) {
    const float v = k < rs ? scale2(x[k], e) : 0.f;
    const __half h = __float2half_rn(v);
    ph[row * KP + k] = h;
    pl[row * KP + k] = __float2half_rn(v - __half2float(h));
  }
  if (lane == 0) pexp[row] = e;
}

// Combined proxies j0 <= j < j0 + nj of columns [c0, c0 + nc) of each listed source
// parent (cheb_kara.cuh), split as above into rows (parent nj + j - j0) nc + column:
// warp per (parent, column), a first pass over K for the rows' magnitudes, a second
// for the split.  NJ = nj (27: j0 is 0), fixed so that the stores need no test of j.
template <int NJ>
__global__ void k_split_kara_f16(const int* __restrict__ parents, int np,
                                 const int* __restrict__ sstart, int span, int C, int c0, int nc,
                                 int j0_, int rs, int KP, const float* __restrict__ proxy,
                                 __half* __restrict__ ph, __half* __restrict__ pl,
                                 int* __restrict__ pexp) {
  const int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= (int64_t)np * nc) return;  // uniform over the warp
  constexpr int nj = NJ;
  const int j0 = NJ == kKaraJ ? 0 : j0_;
  const int64_t p = parents[w / nc];
  const int c = (int)(w % nc);
  const unsigned present = children_present(sstart, p, span);
  auto load = [&](int k, float* v) {
#pragma unroll
    for (int ch = 0; ch < 8; ++ch)
      v[ch] = ((present >> ch) & 1) && k < rs ? proxy[((8 * p + ch) * C + c0 + c) * rs + k] : 0.f;
  };
  auto in = [&](int j) { return (unsigned)(j - j0) < (unsigned)nj; };
  float m[kKaraJ];
#pragma unroll
  for (int j = 0; j < kKaraJ; ++j) m[j] = 0.f;
  for (int k = lane; k < rs; k += 32) {
    float v[8];
    load(k, v);
    kara_combine(v, [&](int j, float x) { m[j] = fmaxf(m[j], fabsf(x)); });
  }
  int e[kKaraJ];
#pragma unroll
  for (int j = 0; j < kKaraJ; ++j) {
#pragma unroll
    for (int o = 16; o; o >>= 1) m[j] = fmaxf(m[j], __shfl_xor_sync(0xffffffffu, m[j], o));
    e[j] = m[j] > 0.f ? 15 - exponent_of(m[j]) : 0;
    if (lane == 0 && in(j)) pexp[(p * nj + j - j0) * nc + c] = e[j];
  }
  for (int k = lane; k < KP; k += 32) {
    float v[8];
    load(k, v);
    kara_combine(v, [&](int j, float x0) {
      if (!in(j)) return;
      const float x = scale2(x0, e[j]);
      const __half h = __float2half_rn(x);
      const int64_t at = ((p * nj + j - j0) * nc + c) * KP + k;
      ph[at] = h;
      pl[at] = __float2half_rn(x - __half2float(h));
    });
  }
}

// Combined operators as the M2L's F16 operands, from the float64 operators in
// fragment order (cheb_fragment_operators: element (f, k) of an operator at
// frag(f, k)): a block per (combination, parent offset) and level.
__global__ void k_kara_ops_f16(const double* __restrict__ E, const int* __restrict__ terms, int rf,
                               int rs, int ntb, int64_t per_blk, int64_t per_op, int NP, int KP,
                               __half* __restrict__ eh, __half* __restrict__ el,
                               int* __restrict__ kexp) {
  const int op = blockIdx.x, lvl = blockIdx.y;
  const double* e = E + (int64_t)lvl * 316 * per_op;
  const int64_t o = (int64_t)lvl * gridDim.x + op;
  auto value = [&](int f, int k) {
    const int64_t i = (f / 8 / ntb) * per_blk + ((int64_t)(k / 4) * ntb + f / 8 % ntb) * 32 +
                      (f % 8) * 4 + k % 4;
    double v = 0.0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int s = terms[op * 8 + q];
      if (s) v += s > 0 ? e[(s - 1) * per_op + i] : -e[(-s - 1) * per_op + i];
    }
    return (float)v;
  };
  __shared__ float sm[32];
  float m = 0.f;
  for (int i = threadIdx.x; i < rf * rs; i += blockDim.x) m = fmaxf(m, fabsf(value(i / rs, i % rs)));
#pragma unroll
  for (int q = 16; q; q >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, q));
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = m;
  __syncthreads();
  for (int q = 0; q < (int)blockDim.x / 32; ++q) m = fmaxf(m, sm[q]);
  const int ex = m > 0.f ? 15 - exponent_of(m) : 0;
  if (threadIdx.x == 0) kexp[o] = ex;
  for (int i = threadIdx.x; i < NP * KP; i += blockDim.x) {
    const int f = i / KP, k = i % KP;
    const float x = f < rf && k < rs ? scale2(value(f, k), ex) : 0.f;
    const __half h = __float2half_rn(x);
    eh[o * NP * KP + i] = h;
    el[o * NP * KP + i] = __float2half_rn(x - __half2float(h));
  }
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (the
// library links no driver library).
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static std::once_flag once;
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  });
  return fn;
}

// Tensor map over an operator half (rows of KP values, nrows rows): boxes of
// NP rows x 128 bytes (32 TF32 or 64 F16 values), 128-byte swizzle (the
// layout the MMA descriptors read).
static int operator_tensor_map(CUtensorMap* m, const void* base, bool f16, int NP, int KP,
                               int64_t nrows) {
  PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
  if (!enc) {
    set_error("cuTensorMapEncodeTiled is not available from the driver");
    return PBBFMM_ERR_CUDA;
  }
  const int esize = f16 ? 2 : 4;
  const cuuint64_t dims[2] = {(cuuint64_t)KP, (cuuint64_t)nrows};
  const cuuint64_t strides[1] = {(cuuint64_t)KP * esize};
  const cuuint32_t box[2] = {(cuuint32_t)(TC_ROWB / esize), (cuuint32_t)NP};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = enc(m, f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32,
                         2, const_cast<void*>(base), dims,
                         strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed for the tensor-core operator tiles");
    return PBBFMM_ERR_CUDA;
  }
  return PBBFMM_OK;
}

// Offsets per TMEM accumulation chain (PBBFMM_TC_GROUP overrides the TF32
// default): one offset when the running sum stays in TMEM (drains then cost
// nothing measurable), four when drains add into pf in global memory.  F16
// operands always drain every offset (each has its own scale).
static int tc_group(int NP, bool f16) {
  if (f16) return 1;
  const char* e = getenv("PBBFMM_TC_GROUP");
  const int g = e ? atoi(e) : (tc_sum_in_tmem(NP) ? 1 : 4);
  return g < 1 ? 1 : (g > 189 ? 189 : g);
}

bool tc_eligible(const pbbfmm_tree* t) {
  return t->p.use_chebyshev && t->use_tc && t->tc.eth && t->tc.eh16 && t->tc.np > 0 &&
         t->tc.np <= kTcMaxN;
}

template <int NST, bool F16, bool RSUM>
static int launch_tc(const TcArgs& a, unsigned tiles, int smem, const CUtensorMap* tm,
                     cudaStream_t st) {
  PB_CUDA(cudaFuncSetAttribute(k_m2l_cheb_tc<NST, F16, RSUM>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  k_m2l_cheb_tc<NST, F16, RSUM><<<tiles, TC_THREADS, smem, st>>>(tm[0], tm[1], tm[2], tm[3], a);
  PB_LAUNCH("m2l_cheb_tc");
  return PBBFMM_OK;
}

// The combined operators of the tree's current set (made on first use): one
// allocation, hi parts, lo parts, exponents, so that they are there as a whole or
// not at all.
static int ensure_kara_tc_ops(pbbfmm_tree* t, cudaStream_t st) {
  TcOps& o = t->tc;
  if (o.kh16) return PBBFMM_OK;
  constexpr int nops = kKaraJ * kKaraD;
  const int nlev = t->ops.nlev, rf = t->ops.rf, rs = t->ops.rs;
  const size_t n = (size_t)nlev * nops * o.np * o.kp16;
  if (int rc = dev_alloc((void**)&o.kh16, 4 * n + sizeof(int) * nlev * nops)) return rc;
  o.kl16 = o.kh16 + n;
  o.kexp = reinterpret_cast<int*>(o.kl16 + n);
  int nblk, ntb;
  cheb_fragment_blocks(rf, &nblk, &ntb);
  const int64_t per_blk = (int64_t)(cheb_rsp(rs) / 4) * ntb * 32;
  k_kara_ops_f16<<<dim3(nops, (unsigned)nlev), 256, 0, st>>>(
      t->d_E, t->d_offs + 4 * (8 * 189 + nops), rf, rs, ntb, per_blk, per_blk * nblk, o.np, o.kp16,
      reinterpret_cast<__half*>(o.kh16), reinterpret_cast<__half*>(o.kl16), o.kexp);
  count_launches(1);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {  // (a kernel's first launch may need memory of its own)
    cudaFree(o.kh16);
    o.kh16 = nullptr;
    return cuda_status(e, "kara_ops_f16");
  }
  return PBBFMM_OK;
}

// The parts of the far field and their arrays (see plan_m2l_f64).  Direct levels
// hold their split proxies together up to the same bound, or one level at a time
// where that is larger.
static int plan_m2l_tc(pbbfmm_tree* t, int C, bool f16, int rowb, ChebPlan* plan, cudaStream_t st) {
  const int L = t->p.tree_level, rf = t->ops.rf, row = 2 * rowb + (f16 ? 4 : 0);
  bool dense[kMaxLevel + 1] = {}, used[kMaxLevel + 1] = {};
  for (int l = 2; l <= L; ++l) {
    used[l] = t->lists.ntgt[l] > 0;
    dense[l] = f16 && cheb_kara_level(t, l);
  }
  for (int64_t bound = t->kara_bytes;; bound = kara_less(bound)) {
    *plan = cheb_plan(dense, used, L, C, row, 4 * rf, row, bound);
    int rc = PBBFMM_OK;
    if (plan->y_bytes > 0) {
      rc = ensure_kara_tc_ops(t, st);
      if (!rc) rc = grow(t->ws.kara_x, plan->x_bytes);
      if (!rc) rc = grow(t->ws.kara_y, plan->y_bytes);
    }
    if (!rc) rc = grow(t->ws.tc_proxy, plan->direct_bytes);
    if (rc != PBBFMM_ERR_ALLOC || bound == 0) return rc;
  }
}

static int launch_m2l_tc(pbbfmm_tree* t, int C, const std::vector<ChebPart>& parts, TcArgs a,
                         bool f16, int KP, const CUtensorMap* tm, cudaStream_t st) {
  const int L = t->p.tree_level, rf = a.rf, rs = t->ops.rs, NP = a.NP, rowb = a.rowb;
  Workspace& ws = t->ws;
  const int* lists = ws.lists.as<int>();
  int rc;
  int64_t tiles = 0;
  if ((rc = kt_begin(t, KS_M2L_SPLIT, st))) return rc;
  for (const ChebPart& q : parts) {
    const int l = q.level, lvl = t->homog ? 0 : l - 2, per_tile = TC_M / q.nc;
    const bool kara = q.nj > 0;
    const int64_t rows = kara ? cells_at(l - 1) * q.nj * q.nc : cells_at(l) * q.nc;
    unsigned char* ph = (kara ? ws.kara_x : ws.tc_proxy).as<unsigned char>() + q.x;
    unsigned char* pl = ph + rows * rowb;
    int* pexp = f16 ? reinterpret_cast<int*>(pl + rows * rowb) : nullptr;
    const float* proxy = ws.proxy.as<float>() + level_offset(l, (int64_t)C * rs);
    const int ns = t->lists.nsrc[kara ? l - 1 : l];
    const int* src = lists + t->lists.src_off[kara ? l - 1 : l];
    const int64_t nrows = (int64_t)ns * q.nc;
    if (ns > 0) {
      if (kara)
        (q.nj == kKaraJ ? k_split_kara_f16<kKaraJ> : k_split_kara_f16<kKaraJ / 3>)
            <<<(unsigned)((nrows * 32 + 255) / 256), 256, 0, st>>>(
                src, ns, ws.sstart_p, (int)cells_at(L - l), C, q.c0, q.nc, q.j0, rs, KP, proxy,
                reinterpret_cast<__half*>(ph), reinterpret_cast<__half*>(pl), pexp);
      else if (f16)
        k_split_proxy_f16<<<(unsigned)((nrows * 32 + 255) / 256), 256, 0, st>>>(
            src, nrows, C, rs, KP, proxy, reinterpret_cast<__half*>(ph),
            reinterpret_cast<__half*>(pl), pexp);
      else
        k_split_proxy<<<(unsigned)((nrows * KP + 255) / 256), 256, 0, st>>>(
            src, nrows, C, rs, KP, proxy, reinterpret_cast<float*>(ph),
            reinterpret_cast<float*>(pl));
      PB_LAUNCH("m2l_split");
    }
    TcLevel& v = a.lv[a.nlev++];
    v.ph = ph;
    v.pl = pl;
    v.pexp = pexp;
    v.item0 = (int)tiles;
    v.C = q.nc;
    v.lev = l;
    v.span = (int)cells_at(L - l);
    v.op0 = lvl * 316;
    v.typed = lists + t->lists.typ_off[l];
    v.pf = ws.pf.as<float>() + level_offset(l, (int64_t)C * rf);
    if (kara) {
      v.mult = q.nj;
      v.j0 = q.j0;
      v.lev = l - 1;
      v.span = (int)cells_at(L - l + 1);
      v.op0 = lvl * kKaraJ * kKaraD;
      v.typed = lists + t->lists.tgt_off[l - 1];
      v.pf = ws.kara_y.as<float>() + q.y / 4;
      v.count[0] = t->lists.ntgt[l - 1];
      v.start[1] = (v.count[0] + per_tile - 1) / per_tile;
      v.start[8] = q.nj * v.start[1];
    } else {
      int n = 0;
      for (int ty = 0; ty < 8; ++ty) {
        v.start[ty] = n;
        v.first[ty] = t->lists.ntyp[l][ty];
        v.count[ty] = t->lists.ntyp[l][ty + 1] - t->lists.ntyp[l][ty];
        n += (v.count[ty] + per_tile - 1) / per_tile;
      }
      v.start[8] = n;
    }
    tiles += v.start[8];
  }
  if ((rc = kt_end(t, st))) return rc;
  if (tiles == 0) return PBBFMM_OK;
  // three stages when they fit in shared memory next to the static arrays
  const int nst = tc_smem_bytes(NP, 3) + 8192 <= 232448 ? 3 : 2;
  const int smem = tc_smem_bytes(NP, nst);
  if ((rc = kt_begin(t, KS_M2L, st))) return rc;
  // register running sum up to TC_REG_SUM columns (three stages always fit there)
  const bool rsum = NP <= TC_REG_SUM && nst == 3;
  const unsigned nt = (unsigned)tiles;
  if (f16)
    rc = rsum ? launch_tc<3, true, true>(a, nt, smem, tm, st)
              : (nst == 3 ? launch_tc<3, true, false>(a, nt, smem, tm, st)
                          : launch_tc<2, true, false>(a, nt, smem, tm, st));
  else
    rc = rsum ? launch_tc<3, false, true>(a, nt, smem, tm, st)
              : (nst == 3 ? launch_tc<3, false, false>(a, nt, smem, tm, st)
                          : launch_tc<2, false, false>(a, nt, smem, tm, st));
  if (rc) return rc;
  for (const ChebPart& q : parts)
    if (q.nj && t->lists.ntgt[q.level - 1] > 0)
      if ((rc = launch_kara_out(t, q, ws.kara_y.as<float>() + q.y / 4,
                                ws.pf.as<float>() + level_offset(q.level, (int64_t)C * rf), C, rf,
                                st)))
        return rc;
  return kt_end(t, st);
}

// The tensor-core M2L: per launch of the plan (one, where the arrays of all levels
// fit its bound) split the proxies, then the MMA kernel.
int run_m2l_cheb_tc(pbbfmm_tree* t, int C, cudaStream_t st) {
  const bool f16 = t->tc_fmt == PBBFMM_TC_F16;
  const int NP = t->tc.np, KP = f16 ? t->tc.kp16 : t->tc.kp, esize = f16 ? 2 : 4;
  if (C > TC_M) {
    set_error("tensor-core M2L takes at most 128 columns per block");
    return PBBFMM_ERR_UNSUPPORTED;
  }
  TcArgs a{};
  a.rf = t->ops.rf;
  a.NP = NP;
  a.rowb = KP * esize;
  a.group = tc_group(NP, f16);
  int rc;
  ChebPlan plan;
  if ((rc = plan_m2l_tc(t, C, f16, a.rowb, &plan, st))) return rc;
  a.sstart = t->ws.sstart_p;
  a.offs = t->d_offs;
  a.eexp = t->tc.eexp;
  a.kexp = t->tc.kexp;
  a.err = t->d_tc_err;
  CUtensorMap tm[4];
  const int64_t nrows = (int64_t)t->ops.nlev * 316 * NP;
  const void* eh = f16 ? (const void*)t->tc.eh16 : (const void*)t->tc.eth;
  const void* el = f16 ? (const void*)t->tc.el16 : (const void*)t->tc.etl;
  if ((rc = operator_tensor_map(&tm[0], eh, f16, NP, KP, nrows))) return rc;
  if ((rc = operator_tensor_map(&tm[1], el, f16, NP, KP, nrows))) return rc;
  tm[2] = tm[0];
  tm[3] = tm[1];
  if (plan.y_bytes > 0) {
    const int64_t krows = (int64_t)t->ops.nlev * kKaraJ * kKaraD * NP;
    if ((rc = operator_tensor_map(&tm[2], t->tc.kh16, true, NP, KP, krows))) return rc;
    if ((rc = operator_tensor_map(&tm[3], t->tc.kl16, true, NP, KP, krows))) return rc;
  }
  for (const std::vector<ChebPart>& parts : plan.launches)
    if ((rc = launch_m2l_tc(t, C, parts, a, f16, KP, tm, st))) return rc;
  return PBBFMM_OK;
}

// ------------------------------------------------------------------------
// M2L pre / post transforms on the tensor cores, same split as the F16 M2L:
//   Out[row_n][m] = alpha oscale[m] sum_k W[m][k] bscale[k] X[row_n][k],  m < M,
// for the columns n < ncols, row_n = cells[n / C] * C + n % C (reference:
// UpwardPass tail, include/compute.hpp:373-396, and the Moment2Local
// post-transform, include/compute.hpp:881-914).  One CTA of 128 threads per
// 128 columns n = 128 blockIdx.x + t:
//   A = row t of X (times bscale), scaled by its own power of two and split
//       into F16 hi / lo, written to shared memory (SW128 K-major) one K chunk
//       of 64 at a time by warp t / 32, lanes over K, 8 rows in flight;
//   B = W (mp rows, pre-split with one exponent per level), by TMA;
//   D[n][m] (128 lanes x mp columns, TMEM) accumulates three products per
//       K step; thread t drains lane t, unscales and writes row_n of Out.
// Bound: latency of the row loads (few CTAs per SM, one stage).  A row per
// thread, read with a stride of K floats between lanes, moved a 32-byte sector
// for every 16 bytes used and wrote the outputs one scattered float per lane;
// with lanes over K and outputs through shared memory, order 5 with 4 columns
// (K = 125, not a multiple of 4; 250,000 points, forward and adjoint) pre + post
// 1.33 -> 0.89 ms, order 6 with 1 column (4M points) 2.51 -> 2.12 ms, all of it
// in the post-transform.
// Chunks run one after another (one stage); two CTAs share an SM (one when
// mp > 256: then each product is two MMAs of N = mp / 2 and the CTA holds all
// 512 TMEM columns).  When
// mp <= 128 each chunk's accumulator is drained into a register sum (the
// tensor pipe's float32 accumulation loses about one ulp per step, so chains
// stay 12 steps long); otherwise the chunks accumulate in TMEM.
constexpr int CG_TC_THREADS = 128;

// A of rows that fit one chunk (K <= 64), the warp's 32 rows: lr lanes per row (two
// values each), so that a load covers 32 / lr rows; a row's values stay in
// registers between its maximum and the split.  With all lanes along K, as for
// longer rows, most of them idle and the rows are read twice: 120,000 points, 16
// columns, pre + post at orders 2, 3, 4: 0.62, 0.68, 0.83 ms, so 0.36, 0.46, 0.66 ms
// (a row per thread: 0.35, 0.53, 0.75 ms).
template <bool BSCALE>
__device__ __forceinline__ void colgemm_rows_short(int K, const float* __restrict__ X,
                                                   const float* __restrict__ bscale,
                                                   const int64_t* s_row, int* s_exp,
                                                   unsigned char* a_hi, unsigned char* a_lo) {
  const int lane = threadIdx.x & 31, w0 = threadIdx.x & ~31;
  const int lr = K <= 16 ? 8 : K <= 32 ? 16 : 32, rows = 32 / lr, l = lane & (lr - 1), k = 2 * l;
  const bool k0 = k < K, k1 = k + 1 < K;
  const float b0 = BSCALE && k0 ? bscale[k] : 1.f, b1 = BSCALE && k1 ? bscale[k + 1] : 1.f;
  for (int r0 = w0 + lane / lr; r0 < w0 + 32; r0 += 8 * rows) {
    float x[8][2];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int64_t r = s_row[r0 + i * rows];
      x[i][0] = r >= 0 && k0 ? X[r * K + k] : 0.f;
      x[i][1] = r >= 0 && k1 ? X[r * K + k + 1] : 0.f;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float v0 = BSCALE ? x[i][0] * b0 : x[i][0], v1 = BSCALE ? x[i][1] * b1 : x[i][1];
      float mx = fmaxf(fabsf(v0), fabsf(v1));
      for (int o = lr >> 1; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      const int e = mx > 0.f ? 15 - exponent_of(mx) : 0, r = r0 + i * rows;
      if (l == 0) s_exp[r] = e;
      const float u0 = scale2(v0, e), u1 = scale2(v1, e);
      const __half2 vh = __floats2half2_rn(u0, u1);
      const float2 vf = __half22float2(vh);
      const uint32_t off = sw128_off(r, l >> 2) + (l & 3) * 4;
      *reinterpret_cast<__half2*>(a_hi + off) = vh;
      *reinterpret_cast<__half2*>(a_lo + off) = __floats2half2_rn(u0 - vf.x, u1 - vf.y);
    }
  }
  for (int ch = lr / 4; ch < 8; ++ch) {  // past the lanes' values: zeros
    const uint32_t off = sw128_off(threadIdx.x, ch);
    *reinterpret_cast<uint4*>(a_hi + off) = make_uint4(0, 0, 0, 0);
    *reinterpret_cast<uint4*>(a_lo + off) = make_uint4(0, 0, 0, 0);
  }
}

template <bool BSCALE, bool OSCALE>
__global__ void __launch_bounds__(CG_TC_THREADS, 1)
    k_colgemm_tc(int M, int mp, int K, int kp, const __grid_constant__ CUtensorMap tm_wh,
                 const __grid_constant__ CUtensorMap tm_wl, int wrow0, int wexp,
                 const int* __restrict__ cells, int ncols, int C, const float* __restrict__ X,
                 const float* __restrict__ bscale, float* __restrict__ Out,
                 const float* __restrict__ oscale, float alpha, int* __restrict__ err) {
  extern __shared__ unsigned char smraw[];
  unsigned char* base = smraw + ((1024 - (smem_u32(smraw) & 1023)) & 1023);
  const int nh = mp > 256 ? 2 : 1;             // MMAs (and TMA boxes) per product
  const int hn = mp / nh;                      // their N (a multiple of 16)
  const uint32_t tcols = mp > 256 ? 512 : 256;  // TMEM columns
  unsigned char* a_hi = base;
  unsigned char* a_lo = base + 16384;
  unsigned char* b_hi = base + 32768;
  unsigned char* b_lo = b_hi + mp * 128;
  __shared__ uint64_t s_tma, s_mma;
  __shared__ uint32_t s_tmem;
  __shared__ int s_fail;
  const int tid = threadIdx.x, warp = tid >> 5;
  const int n = blockIdx.x * CG_TC_THREADS + tid;
  const bool valid = n < ncols;
  const int64_t row = valid ? (int64_t)cells[n / C] * C + n % C : 0;
  __shared__ int64_t s_row[CG_TC_THREADS];  // row_n, or -1 past the end
  __shared__ int s_exp[CG_TC_THREADS];      // its exponent: max |bscale x| 2^e in [2^14, 2^15)
  const int lane = tid & 31;
  s_row[tid] = valid ? row : -1;
  __syncwarp();
  const bool one = K <= 64;  // one chunk holds the rows: read once, below
  for (int r0 = 32 * warp; !one && r0 < 32 * warp + 32; r0 += 8) {
    float mx[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) mx[i] = 0.f;
    for (int k = lane; k < K; k += 32) {
      const float b = BSCALE ? bscale[k] : 1.f;
      float x[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = s_row[r0 + i] >= 0 ? X[s_row[r0 + i] * K + k] : 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) mx[i] = fmaxf(mx[i], fabsf(BSCALE ? x[i] * b : x[i]));
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
#pragma unroll
      for (int o = 16; o; o >>= 1) mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], o));
      if (lane == 0) s_exp[r0 + i] = mx[i] > 0.f ? 15 - exponent_of(mx[i]) : 0;
    }
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                     smem_u32(&s_tmem)),
                 "r"(tcols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  if (tid == 0) {
    mbar_init(&s_tma, 1);
    mbar_init(&s_mma, 1);
    s_fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem;
  const uint32_t idesc = f16_idesc(TC_M, hn);
  const int nchunks = kp / 64;
  const bool rdrain = mp <= 128;  // uniform
  const uint32_t lane_base = tmem + ((uint32_t)(32 * warp) << 16);
  float racc[128];  // register sum of the drained chunks (rdrain)
#pragma unroll
  for (int i = 0; i < 128; ++i) racc[i] = 0.f;
  int last_tma = -1;  // thread 0: the last chunk whose TMA was issued
  for (int c = 0; c < nchunks; ++c) {
    // A chunk: 64 values of each row (zero past K), scaled and split; lane k / 2
    // of a row's warp takes values k and k + 1
    if (one) colgemm_rows_short<BSCALE>(K, X, bscale, s_row, s_exp, a_hi, a_lo);
    for (int r0 = 32 * warp; !one && r0 < 32 * warp + 32; r0 += 8) {
      const int k = c * 64 + 2 * lane;
      const bool k0 = k < K, k1 = k + 1 < K;
      float x[8][2];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int64_t r = s_row[r0 + i];
        x[i][0] = r >= 0 && k0 ? X[r * K + k] : 0.f;
        x[i][1] = r >= 0 && k1 ? X[r * K + k + 1] : 0.f;
      }
      const float b0 = BSCALE && k0 ? bscale[k] : 1.f, b1 = BSCALE && k1 ? bscale[k + 1] : 1.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int er = s_exp[r0 + i];  // uniform over the warp
        float v0 = BSCALE ? x[i][0] * b0 : x[i][0], v1 = BSCALE ? x[i][1] * b1 : x[i][1];
        if (er >= -126 && er <= 127) {
          const float f = exp2i(er);
          v0 *= f, v1 *= f;
        } else {
          v0 = scale2(v0, er), v1 = scale2(v1, er);
        }
        const __half2 vh = __floats2half2_rn(v0, v1);
        const float2 vf = __half22float2(vh);
        const uint32_t off = sw128_off(r0 + i, lane >> 2) + (lane & 3) * 4;
        *reinterpret_cast<__half2*>(a_hi + off) = vh;
        *reinterpret_cast<__half2*>(a_lo + off) = __floats2half2_rn(v0 - vf.x, v1 - vf.y);
      }
    }
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");  // to the tensor pipe
    if (tid == 0) {
      mbar_arrive_expect_tx(&s_tma, 2u * (uint32_t)mp * 128u);
      for (int h = 0; h < nh; ++h) {  // boxes of hn rows
        tma_load_2d(b_hi + h * hn * 128, &tm_wh, c * 64, wrow0 + h * hn, &s_tma);
        tma_load_2d(b_lo + h * hn * 128, &tm_wl, c * 64, wrow0 + h * hn, &s_tma);
      }
      last_tma = c;
    }
    __syncthreads();
    if (tid == 0) {
      if (mbar_wait(&s_tma, c & 1, nullptr)) {
        tc_fence_after();
        const uint32_t ah = smem_u32(a_hi), al = smem_u32(a_lo);
        const uint32_t bh = smem_u32(b_hi), bl = smem_u32(b_lo);
        for (int h = 0; h < nh; ++h) {  // D columns [h hn, (h + 1) hn)
          const uint32_t d = tmem + (uint32_t)(h * hn), bo = (uint32_t)(h * hn * 128);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const uint32_t off = k * 32;
            tc_mma_f16(d, sw128_desc(al + off), sw128_desc(bh + bo + off), idesc,
                       ((c > 0 && !rdrain) || k > 0) ? 1u : 0u);
            tc_mma_f16(d, sw128_desc(ah + off), sw128_desc(bl + bo + off), idesc, 1u);
            tc_mma_f16(d, sw128_desc(ah + off), sw128_desc(bh + bo + off), idesc, 1u);
          }
        }
        tc_commit(&s_mma);
      } else {
        s_fail = 1;
        mbar_arrive(&s_mma);  // release the others; the result is not used
      }
    }
    // the chunk's MMAs (or the failure) before its shared memory is rewritten
    if (!mbar_wait(&s_mma, c & 1, nullptr)) s_fail = 1;
    __syncthreads();
    if (s_fail) break;
    if (rdrain) {
      // all lanes (warp-collective loads); done before the next chunk's MMAs
      // are issued (the barrier at the top of the next chunk orders them)
      tc_fence_after();
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        if (q * 16 >= mp) break;
        uint32_t r[16];
        tc_ld16_wait(lane_base + (uint32_t)(q * 16), r);
#pragma unroll
        for (int i = 0; i < 16; ++i) racc[q * 16 + i] += __uint_as_float(r[i]);
      }
      tc_fence_before();
    }
  }
  if (s_fail) {
    // no copy or MMA may still be running when the CTA ends: wait (bounded)
    // once more for the last chunk's
    if (tid == 0 && last_tma >= 0) {
      mbar_wait(&s_tma, last_tma & 1, nullptr);
      mbar_wait(&s_mma, last_tma & 1, nullptr);
    }
    if (tid == 0 && err) atomicExch(err, 1);
  } else {
    // every lane of the warp takes part in the (warp-collective) TMEM loads;
    // only valid rows are written
    tc_fence_after();
    // the unscaling 2^-(e + wexp) as two exact power-of-two factors applied
    // one after the other (never multiplied together, which could leave the
    // float range although the result lies inside it), then alpha
    const int kt = -(s_exp[tid] + wexp), k1 = min(max(kt, -126), 127), k2 = min(max(kt - k1, -149), 127);
    const float sc = exp2i(k1), sc2 = exp2i(k2);
    float* so = reinterpret_cast<float*>(base);  // [128 rows][129] (the tiles are done with)
    for (int m0 = 0; m0 < mp; m0 += 128) {  // uniform
      __syncthreads();
      if (rdrain) {
#pragma unroll
        for (int m = 0; m < 128; ++m)
          if (m < mp) so[tid * 129 + m] = racc[m] * sc * sc2 * alpha;
      } else {
        for (int q = 0; q < min(128, mp - m0); q += 16) {
          uint32_t r[16];
          tc_ld16_wait(lane_base + (uint32_t)(m0 + q), r);
#pragma unroll
          for (int i = 0; i < 16; ++i)
            so[tid * 129 + q + i] = __uint_as_float(r[i]) * sc * sc2 * alpha;
        }
      }
      __syncthreads();
      for (int r = warp; r < CG_TC_THREADS; r += CG_TC_THREADS / 32) {
        if (s_row[r] < 0) continue;
        float* o = Out + s_row[r] * M + m0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int m = lane + 32 * q;
          if (m0 + m < M) o[m] = OSCALE ? so[r * 129 + m] * oscale[m0 + m] : so[r * 129 + m];
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem),
                 "r"(tcols)
                 : "memory");
  }
}

// Tensor cores when the output width fits two MMAs (mp <= 512) and no TMEM
// accumulation chain is longer than two K chunks (24 steps): either the
// chunks are drained into registers (mp <= 128) or there are at most two
// (K <= 128).  Longer chains would add ~1e-6 of accumulation error.
bool colgemm_tc_eligible(const pbbfmm_tree* t, bool post) {
  if (!t->p.use_chebyshev || !t->use_tc || t->ops.nlev > 32) return false;
  const TcOps& o = t->tc;
  const int mp = post ? o.u_mp : o.vt_mp, kp = post ? o.u_kp : o.vt_kp;
  if (!(post ? o.uh : o.vth) || mp > 512) return false;
  return mp <= 128 || kp <= 128;
}

int run_colgemm_tc(pbbfmm_tree* t, bool post, int lvl, const int* cells, int ncols, int C,
                   const float* X, float* Out, float alpha, cudaStream_t st) {
  if (ncols <= 0) return PBBFMM_OK;
  const TcOps& o = t->tc;
  const int M = post ? t->n3 : t->ops.rs, K = post ? t->ops.rf : t->n3;
  const int mp = post ? o.u_mp : o.vt_mp, kp = post ? o.u_kp : o.vt_kp;
  const uint16_t* wh = post ? o.uh : o.vth;
  const uint16_t* wl = post ? o.ul : o.vtl;
  const int wexp = post ? o.u_exp[lvl] : o.vt_exp[lvl];
  CUtensorMap tm_h, tm_l;
  const int64_t nrows = (int64_t)t->ops.nlev * mp;
  const int hn = mp > 256 ? mp / 2 : mp;  // rows per TMA box
  if (int rc = operator_tensor_map(&tm_h, wh, true, hn, kp, nrows)) return rc;
  if (int rc = operator_tensor_map(&tm_l, wl, true, hn, kp, nrows)) return rc;
  // at least 78 KB (114 KB when a CTA takes all 512 TMEM columns), so that
  // the CTAs sharing an SM always find their TMEM columns free and no
  // allocation waits for another CTA
  const int smem = std::max(32768 + 2 * mp * 128 + 1024, (mp > 256 ? 114 : 78) * 1024);
  const unsigned grid = (unsigned)((ncols + CG_TC_THREADS - 1) / CG_TC_THREADS);
  const float* Kw = t->f_Kw;
  if (post) {
    PB_CUDA(cudaFuncSetAttribute(k_colgemm_tc<false, true>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    k_colgemm_tc<false, true><<<grid, CG_TC_THREADS, smem, st>>>(
        M, mp, K, kp, tm_h, tm_l, lvl * mp, wexp, cells, ncols, C, X, nullptr, Out, Kw, alpha,
        t->d_tc_err);
  } else {
    PB_CUDA(cudaFuncSetAttribute(k_colgemm_tc<true, false>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    k_colgemm_tc<true, false><<<grid, CG_TC_THREADS, smem, st>>>(
        M, mp, K, kp, tm_h, tm_l, lvl * mp, wexp, cells, ncols, C, X, Kw, Out, nullptr, alpha,
        t->d_tc_err);
  }
  PB_LAUNCH(post ? "m2l_post_tc" : "m2l_pre_tc");
  return PBBFMM_OK;
}


}  // namespace pbbfmm

extern "C" int pbbfmm_debug_set_pipeline_wait_limit(int device, long long polls) {
  using namespace pbbfmm;
  int cur = 0;
  PB_CUDA(cudaGetDevice(&cur));
  if (device >= 0 && device != cur) PB_CUDA(cudaSetDevice(device));
  const long long v = polls > 0 ? polls : kWaitIters;
  const cudaError_t e = cudaMemcpyToSymbol(g_pipe_wait_iters, &v, sizeof(v));
  const int rc = e == cudaSuccess ? set_unif_tc_wait_limit(v) : PBBFMM_OK;
  if (device >= 0 && device != cur) cudaSetDevice(cur);
  if (e != cudaSuccess) return cuda_status(e, "set pipeline wait limit");
  return rc;
}
