// The on-chip CG solves (lpm_pcg.cu): arguments and launch limits.
#pragma once

#include "lpm_internal.cuh"

namespace lpm {

constexpr int kPcgMaxBlocks = 160;  // blocks of a solve, at most one per SM (GB300: 152)
constexpr int kPcgMaxSlices = 32;   // 32-row slices of a block (a lane each in its sums)

// Threads per block, one block per SM, the message warp included: registers
// for an operator group in flight beside the one in use (2-D: 80, 3-D: 128).
// The wide form has a warp more for 2-D blocks of 24 slices (72 registers).
template <int DIM>
constexpr int kPcgThreads = DIM == 3 ? 512 : 768;
template <int DIM>
constexpr int kPcgWideThreads = DIM == 3 ? 512 : 800;

// Shared memory of one resident group of a slice: 32 rows x four blocks of
// DIM*DIM FP32 values and their 16-bit positions.
template <int DIM>
constexpr int kPcgUnit = 32 * (DIM * DIM * 16 + 8);

// First slice of block b of G: whole slices, spread evenly.
__host__ __device__ __forceinline__ int plan_slice(int b, int G, int nslice) {
  return (int)((long long)b * nslice / G);
}

struct PcgMixedArgs {
  const int64_t* sell_ptr;
  const int *ucnt, *uown, *ulist, *scol;
  const unsigned short* lidx;
  const float *A32, *S32, *invd;
  const double *A64, *b;
  float *r, *rlo, *x, *xlo, *zp;
  double *x64, *xs;  // xs: the solution a reliable update multiplies
  unsigned long long* words;
  CgScalars* cg;
  // coarse correction: coarse DOFs and the most of a block; the entries
  // (block, aggregate) by block (cblk_*: first, place in aggregate order,
  // aggregate) and by aggregate (cagg_ptr); per row its aggregate among its
  // block's; the records of y and e
  int nc, cmaxrows, cmaxagg, centries;
  const int *cblk_ptr, *cblk_pos, *cblk_agg, *cagg_ptr;
  const unsigned* crow;
  const float* coff;
  const unsigned char* cfixed;
  const double* cAinv;
  float* crec;
  int64_t nslots;
  int n, nslice, umax, gs, gx, maxS, T;
  int off_p, off_list, off_part, off_row, off_coarse, off_op;  // byte offsets of the dynamic shared memory's parts
};

}  // namespace lpm
