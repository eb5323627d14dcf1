// Layouts and entry points shared by the uniform path's transforms
// (m2l_unif.cu) and its tensor-core MAC (m2l_unif_tc.cu).
#pragma once
#include "fmm.cuh"
#include "tcgen05.cuh"

namespace pbbfmm {

// Spectra of one level (S parents per side) and one group of 8 columns, as the
// tensor-core MAC reads and writes them.
//   in : [slot][x][part][y + 1][z + 1][column] rows of 16 bytes (4 children x
//        (re, im) F16), parts hi of children 0-3, hi of 4-7, lo of 0-3, lo of
//        4-7; y and z padded by one parent of zeros on either side, so that
//        every line of 18 parents is one contiguous copy;
//   out: [slot][x][child][y][z][column] float2.
struct UnifPlanes {
  static __host__ __device__ constexpr int64_t part_bytes(int S) {
    return (int64_t)(S + 2) * (S + 2) * 8 * 16;
  }
  static __host__ __device__ constexpr int64_t slot_bytes(int S) { return S * 4 * part_bytes(S); }
  static __host__ __device__ constexpr int64_t lo_off(int S) { return 2 * part_bytes(S); }
  static __host__ __device__ constexpr int64_t row_byte(int S, int x, int part, int y, int z, int c) {
    return ((int64_t)x * 4 + part) * part_bytes(S) +
           (((int64_t)(y + 1) * (S + 2) + z + 1) * 8 + c) * 16;
  }
  static __host__ __device__ constexpr int64_t slot_outputs(int S) { return (int64_t)S * S * S * 64; }
  static __host__ __device__ constexpr int64_t out_index(int S, int x, int t, int y, int z, int c) {
    return ((((int64_t)x * 8 + t) * S + y) * S + z) * 8 + c;
  }
};

// 2^s puts a magnitude with these float bits into [2^14, 2^15): s, clamped to
// the float exponent range (0 for 0 and for infinities and NaNs).
__device__ __forceinline__ int unif_scale_exp(uint32_t mbits) {
  if (mbits == 0u || (mbits & 0x7f800000u) == 0x7f800000u) return 0;
  return max(-126, min(127, 15 - exponent_of(__uint_as_float(mbits))));
}

template <typename T>
struct FftFwdArgs {
  const T* S;           // moments of the level, [cell][C][n^3]
  cplx_t<T>* X;         // spectra
  int64_t slot_stride;  // values (SPLIT: bytes) between frequency slots
  int64_t lo_off;       // SPLIT: bytes from the hi to the lo part
  int C, c0;
  const int* cells;     // nonempty source cells
  int64_t nunits;       // their (cell, column) pairs
  int side;             // SPLIT: parents per side
  const uint8_t* occ;   // SPLIT: cell has sources
  const uint32_t* amax; // SPLIT: bounds per column of the group
};
template <typename T>
struct FftInvArgs {
  const cplx_t<T>* Y;
  T* F;                 // locals of the level
  int64_t slot_stride;
  int C, c0;
  const int* cells;     // nonempty target cells
  int64_t nunits;
  int side;
  const uint8_t* occ;   // SPLIT: cell has targets
  T scale, invP;
};

// cell occupancy of a level, for sources and targets, and of the MAC's lines
int run_unif_tc_occupancy(pbbfmm_tree* t, int l, uint8_t** socc, uint8_t** tocc, cudaStream_t st);
// zeros in the padding of the spectra
int run_unif_tc_borders(pbbfmm_tree* t, int S, unsigned char* X, cudaStream_t st);
int run_m2l_unif_tc_level(pbbfmm_tree* t, int l, int lvl, const unsigned char* X, float2* Y,
                          const uint32_t* amax, const uint8_t* tocc, cudaStream_t st);

}  // namespace pbbfmm
