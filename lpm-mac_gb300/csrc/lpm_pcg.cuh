// The on-chip CG solves (lpm_pcg.cu): arguments and launch limits.
#pragma once

#include "lpm_device.cuh"
#include "lpm_internal.cuh"

namespace lpm {

constexpr int kPcgMaxBlocks = 160;  // blocks of a solve, at most one per SM (GB300: 152)
constexpr int kPcgMaxSlices = 32;   // 32-row slices of a block (a lane each in its sums)

// Most threads per block, the message warp included (of an SM to itself; small
// systems take less, shape_on_plan): registers
// for an operator group in flight beside the one in use (2-D: 80, 3-D: 128).
// The wide form has a warp more for 2-D blocks of 24 slices (72 registers),
// the narrow one 128 registers in 2-D too: at 80 the message warp keeps part of
// its records in local memory, on the path from one iteration to the next (us
// per iteration of the mixed solve, 768 and 512 threads: plates of 3.6k rows
// 7.7 and 6.75, 28k 8.8 and 7.9, 60k 11.6 and 10.6).  It stands back where its
// fifteen compute warps leave a slice one and the others leave it two (45k
// rows: 9.6 and 9.9).
template <int DIM>
constexpr int kPcgThreads = DIM == 3 ? 512 : 768;
template <int DIM>
constexpr int kPcgWideThreads = DIM == 3 ? 512 : 800;
constexpr int kPcgNarrowThreads = 512;

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

// Shared memory of one resident group of a slice in the FP64 solve.
template <int DIM>
constexpr int kPcgUnit64 = 32 * (DIM * DIM * 32 + 8);
// Compute warps of an FP64 block of S slices, a multiple of four: of 4, 8 and
// 12, eight were best for plates of one to four slices a block (10.7 us of
// an iteration at 2,581 rows; 10.9 and 11.0), twelve for cubes (29.5 at 26^3
// against 30.5 and 40.6).
constexpr int kPcg64Slices = 12;
__host__ __device__ __forceinline__ int fp64_warps(int dim, int S) {
  return dim == 3 ? kPcg64Slices : S <= 8 ? 8 : kPcg64Slices;
}
// Most slices of a block whose launch leaves room for a second block on its SM
// (shape_on_plan, shape64).
constexpr int kSharingSlices = 2;
// Threads per block of the FP64 solve, at most, the message warp included
// (128 registers).
constexpr int kPcg64Threads = 512;

struct PcgFp64Args {
  const int64_t* sell_ptr;
  const int *ucnt, *uown, *ulist;
  const unsigned short* lidx;
  const double *A, *invd;
  double *x, *r;
  float* zp;
  unsigned long long* words;
  CgScalars* cg;
  int64_t nslots;
  int n, nslice, umax, maxS, W;
  int R, gx, tails;  // groups of a warp kept on chip, one more of the first gx; tail blocks of a slice kept
  int off_p, off_list, off_part, off_row, off_tail, off_op;
};

// Bytes per row of the two copies of z: a record each in the mixed solve, two
// records in the FP64 one.
constexpr size_t kZBytes = 32, kZBytes64 = 64;

// Polls of a record before a wait gives up: about 0.15 us each.
constexpr long long kPollLimit = 1LL << 22;

// ---------------------------------------------------------------- messages
// Blocks talk through 16-byte records, written and read whole (the 128-bit
// accesses of the memory model), that carry their own tag: a reader polls the
// record itself, so no fence and no separate flag stands between the data and
// its use.
struct Rec {
  unsigned x, y, z, w;
};
__device__ __forceinline__ void st_rec(void* a, unsigned x, unsigned y, unsigned z, unsigned w) {
  asm volatile(
      "{.reg .b128 v; .reg .b64 l, h; mov.b64 l, {%1, %2}; mov.b64 h, {%3, %4}; mov.b128 v, {l, h}; "
      "st.relaxed.gpu.global.b128 [%0], v;}" ::"l"(a),
      "r"(x), "r"(y), "r"(z), "r"(w)
      : "memory");
}
__device__ __forceinline__ Rec ld_rec(const void* a) {
  Rec r;
  asm volatile(
      "{.reg .b128 v; .reg .b64 l, h; ld.relaxed.gpu.global.b128 v, [%4]; mov.b128 {l, h}, v; mov.b64 {%0, %1}, l; "
      "mov.b64 {%2, %3}, h;}"
      : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
      : "l"(a)
      : "memory");
  return r;
}

// Records of the grid sums (a.words): arrivals of the two sums of an
// iteration and of the reliable update's, each twice (by parity), then the
// replies.
enum : int { kArrAlpha = 0, kArrBeta = 2, kArrUpdate = 4, kReplies = 8 };  // sets of kPcgMaxBlocks records
constexpr int kReplyCopies = 4;  // copies of a reply, read by every fourth block

__device__ __forceinline__ Rec* arrivals(Rec* words, int set, unsigned parity) {
  return words + (size_t)(set + (int)parity) * kPcgMaxBlocks;
}
__device__ __forceinline__ Rec* reply(Rec* words, unsigned epoch, int copy) {
  return words + (size_t)kReplies * kPcgMaxBlocks + ((epoch & 1) * kReplyCopies + copy) * 8;  // 128 bytes apart
}

// Bytes of the grid sums' records.
constexpr size_t kWordBytes = 16 * ((size_t)kReplies * kPcgMaxBlocks + 2 * kReplyCopies * 8);

// One record per lane and stride of 32 blocks, polled until match() accepts
// it; bounded.
template <typename F>
__device__ __forceinline__ bool gather_records(const Rec* set, int G, Rec (&r)[kPcgMaxBlocks / 32], F match) {
  const int lane = threadIdx.x & 31;
  for (long long polls = 0; polls < kPollLimit; ++polls) {
#pragma unroll
    for (int q = 0; q < kPcgMaxBlocks / 32; ++q)
      if (lane + 32 * q < G) r[q] = ld_rec(set + lane + 32 * q);
    bool all = true;
#pragma unroll
    for (int q = 0; q < kPcgMaxBlocks / 32; ++q)
      if (lane + 32 * q < G) all = all && match(r[q]);
    if (__all_sync(0xffffffffu, all)) return true;
  }
  return false;
}

template <typename F>
__device__ __forceinline__ bool poll_record(const Rec* a, Rec& r, F match) {
  for (long long polls = 0; polls < kPollLimit; ++polls) {
    r = ld_rec(a);
    if (match(r)) return true;
  }
  return false;
}

__device__ __forceinline__ unsigned comp_u16(const ushort4& v, int t) {
  return t == 0 ? v.x : t == 1 ? v.y : t == 2 ? v.z : v.w;
}
__device__ __forceinline__ float comp_f(const float4& v, int t) {
  return t == 0 ? v.x : t == 1 ? v.y : t == 2 ? v.z : v.w;
}

// Groups of a slice in the order the solve takes them: the tail of at most
// three single blocks first (as a group padded with zeros, when the slice
// has one), then the groups of four.
struct SliceGroups {
  int64_t base;  // first slot of the slice
  int g4;        // blocks in groups of four
  int tail;      // blocks after them
  int count;     // groups, the tail included
};
__device__ __forceinline__ SliceGroups slice_groups(const int64_t* __restrict__ sell_ptr, int slice) {
  const int64_t b = sell_ptr[slice];
  const int w = (int)((sell_ptr[slice + 1] - b) / kSlice);
  const int g4 = w / kVec * kVec;
  return SliceGroups{b, g4, w - g4, g4 / kVec + (w > g4 ? 1 : 0)};
}

// A compute thread's place: its slice among the block's, its share of the
// slice's groups, its row.  A block with fewer slices than the widest leaves
// its last warps without a share.  The block's last warp computes nothing: it
// carries the messages, in a loop of its own.
struct Place {
  int s0, S, ls, t, row;
  bool act, mine, owner;  // has a share; owns the slice's rows; owns a row
};
__device__ __forceinline__ Place place_of(const PcgMixedArgs& a) {
  Place p;
  p.s0 = plan_slice(blockIdx.x, gridDim.x, a.nslice);
  p.S = plan_slice(blockIdx.x + 1, gridDim.x, a.nslice) - p.s0;
  const int warp = threadIdx.x >> 5;
  p.ls = warp % p.S;
  p.t = warp / p.S;
  p.row = (p.s0 + p.ls) * kSlice + (int)(threadIdx.x & 31);
  p.act = p.t < a.T;
  p.mine = p.t == 0;
  p.owner = p.mine && p.row < a.n;
  return p;
}

// Barrier of the compute warps alone.
__device__ __forceinline__ void compute_sync(int threads) { asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory"); }

}  // namespace lpm
