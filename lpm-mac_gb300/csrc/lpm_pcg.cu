// The CG solves of systems with at most one row per resident thread, as one
// cooperative kernel whose working set stays on the SMs.
//
// What bounds a solve of this size is neither HBM nor the FP32 pipe but
// latency: of the chain "column index, partner value, next group" in each
// row, and of the grid barriers between the phases of an iteration.  So
//   - block b owns whole 32-row slices of the operator for the whole solve,
//     and T of its warps share a slice, each taking every T-th group of four
//     blocks of the slice's rows (a small system then still fills its SMs);
//   - the operator's groups live in shared memory from the first iteration
//     on, as many as fit (all of a 21^3 cube or a 28k-particle plate); the
//     rest streams from L2;
//   - the direction p at every column the block needs (its own rows and
//     their halo, at most a few thousand) is staged into shared memory once
//     per iteration, so that a block's value is fetched by its 16-bit
//     position there;
//   - the row's residual, a double-float pair, and its product stay in the
//     registers of the warp that owns its slice (x, a pair too, is updated in
//     global memory while the sums travel);
//   - two grid barriers per iteration instead of three: the new direction
//     p = zc z + beta p is formed by every block from the z and the old p of
//     the columns it stages, not written by the owner and read back;
//   - block 0 gathers the blocks' partial sums, decides (alpha; beta and
//     what follows) and replies; sums, replies and z travel as 16-byte
//     records that carry their own tag, so no fence stands in the loop.
// The recurrence, the reliable updates and the stopping rule are those of
// k_mx_update, k_mx_residual, k_mx_replace and k_mx_pupdate (lpm_cg.cu).
//
// Measured on GB300, us per iteration of the mixed solve, here against the
// better of the graph and the persistent loop of lpm_cg.cu: hexagonal plates
// of 1,661 rows 6.7 (16.1), 28,126 rows 7.8 (18.2), 80,401 rows 12.6 (21.9)
// and 112,658 rows 15.9 (24.7); simple cubes of 21^3 9.9 (25.5), 31^3 17 (30)
// and 41^3 41 (50); a BCC polycrystal of 27,287 rows 12.8 (27).  Of an
// iteration of the 28k plate (16.5k cycles) the product takes 4.0k, the two
// sums about 4k each (two trips of some 550 to 900 cycles through L2, the
// fold, the division), the rest is the block's own reductions and barriers.
// What was tried for the sums, in cycles per grid-wide sum over 152 blocks:
// atomic counter and fold 5,900, every block polling every block's word 5,400
// to 10,700 (the polls get in the words' way), by clusters 4,100 to 7,200,
// gathered and answered by one block 3,100.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <vector>

#include "lpm_coarse.cuh"
#include "lpm_device.cuh"
#include "lpm_df.cuh"
#include "lpm_pcg.cuh"

namespace lpm {
namespace {

constexpr int kPlanThreads = 256;
// ------------------------------------------------------------------ plan
// Columns of the block's slices as a bitmap over all particles, in shared
// memory (at most 24 slices of 160 blocks, 122,880 particles: 15 KB), and for each
// word the number of columns below it.
__device__ void plan_bitmap(int n, int s0, int s1, const int64_t* __restrict__ sell_ptr,
                            const int* __restrict__ scol, const int* __restrict__ rowlen, unsigned* bits) {
  const int words = (n + 31) / 32;
  for (int w = threadIdx.x; w < words; w += blockDim.x) bits[w] = 0u;
  __syncthreads();
  const int r0 = s0 * kSlice, r1 = min(n, s1 * kSlice);
  for (int j = r0 + (int)threadIdx.x; j < r1; j += blockDim.x) {
    atomicOr(&bits[j / 32], 1u << (j % 32));
    const SellRow sr = sell_row(sell_ptr, j);
    const int len = rowlen[j];
    for (int k = 0; k < len; ++k) {
      const int c = scol[sell_slot(sr, k)];
      atomicOr(&bits[c / 32], 1u << (c % 32));
    }
  }
  __syncthreads();
}

// Exclusive prefix sum of the words' bit counts; returns the total.
__device__ int plan_prefix(int n, const unsigned* bits, int* before) {
  __shared__ int part[kPlanThreads];
  const int words = (n + 31) / 32, per = (words + (int)blockDim.x - 1) / (int)blockDim.x;
  const int w0 = threadIdx.x * per, w1 = min(words, w0 + per);
  int s = 0;
  for (int w = w0; w < w1; ++w) s += __popc(bits[w]);
  part[threadIdx.x] = s;
  __syncthreads();
  for (int o = 1; o < (int)blockDim.x; o <<= 1) {
    const int v = (int)threadIdx.x >= o ? part[threadIdx.x - o] : 0;
    __syncthreads();
    part[threadIdx.x] += v;
    __syncthreads();
  }
  int at = part[threadIdx.x] - s;
  for (int w = w0; w < w1; ++w) {
    before[w] = at;
    at += __popc(bits[w]);
  }
  const int total = part[blockDim.x - 1];
  __syncthreads();
  return total;
}

__global__ void __launch_bounds__(kPlanThreads) k_plan_count(int n, int nslice, const int64_t* __restrict__ sell_ptr,
                                                             const int* __restrict__ scol,
                                                             const int* __restrict__ rowlen, int* __restrict__ ucnt) {
  extern __shared__ unsigned bits[];
  const int s0 = plan_slice(blockIdx.x, gridDim.x, nslice), s1 = plan_slice(blockIdx.x + 1, gridDim.x, nslice);
  plan_bitmap(n, s0, s1, sell_ptr, scol, rowlen, bits);
  int s = 0;
  for (int w = threadIdx.x; w < (n + 31) / 32; w += blockDim.x) s += __popc(bits[w]);
  atomicAdd(&ucnt[blockIdx.x], s);
}

// The block's columns in ascending order, the position of its first row
// among them, and each slot's position (the row's own for slots past its end,
// whose operator values are zero).
__global__ void __launch_bounds__(kPlanThreads) k_plan_fill(int n, int nslice, const int64_t* __restrict__ sell_ptr,
                                                            const int* __restrict__ scol,
                                                            const int* __restrict__ rowlen, int umax,
                                                            int* __restrict__ ulist, int* __restrict__ uown,
                                                            unsigned short* __restrict__ lidx) {
  extern __shared__ unsigned bits[];
  const int words = (n + 31) / 32;
  int* before = (int*)(bits + words);
  const int s0 = plan_slice(blockIdx.x, gridDim.x, nslice), s1 = plan_slice(blockIdx.x + 1, gridDim.x, nslice);
  plan_bitmap(n, s0, s1, sell_ptr, scol, rowlen, bits);
  plan_prefix(n, bits, before);
  for (int w = threadIdx.x; w < words; w += blockDim.x) {
    unsigned m = bits[w];
    int at = before[w];
    while (m) {
      const int c = w * 32 + __ffs(m) - 1;
      ulist[(int64_t)blockIdx.x * umax + at++] = c;
      m &= m - 1;
    }
  }
  const int r0 = s0 * kSlice, r1 = min(n, s1 * kSlice);
  auto position = [&](int c) { return before[c / 32] + __popc(bits[c / 32] & ((1u << (c % 32)) - 1u)); };
  if (threadIdx.x == 0) uown[blockIdx.x] = position(r0);
  for (int j = r0 + (int)threadIdx.x; j < r1; j += blockDim.x) {
    const SellRow sr = sell_row(sell_ptr, j);
    const int len = rowlen[j], w = (int)((sell_ptr[j / kSlice + 1] - sell_ptr[j / kSlice]) / kSlice);
    const int own = position(j);
    for (int k = 0; k < w; ++k) {
      const int64_t s = sell_slot(sr, k);
      lidx[s] = (unsigned short)(k < len ? position(scol[s]) : own);
    }
  }
}

// Sums of pairs over the warp, in every lane.
template <int K>
__device__ __forceinline__ void warp_df_sum(float (&s)[K], float (&c)[K]) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const float so = __shfl_xor_sync(0xffffffffu, s[k], o), co = __shfl_xor_sync(0xffffffffu, c[k], o);
      df_add(s[k], c[k], so, co);
    }
}
__device__ __forceinline__ void warp_df_sum(float& s, float& c) {
  float a[1] = {s}, b[1] = {c};
  warp_df_sum<1>(a, b);
  s = a[0];
  c = b[0];
}

// --------------------------------------------------------- mixed precision
constexpr double kRuDelta2 = 0.1 * 0.1;  // reliable-update trigger on |r|^2 (kDelta of lpm_cg.cu squared)

// One block of a row (element e from at(e)) times the staged difference p - pi,
// compensated.
template <int DIM, typename F>
__device__ __forceinline__ void block_acc(F at, const float* p, const float (&pi)[DIM], float (&s)[DIM],
                                          float (&c)[DIM]) {
  float pc[DIM];
  if constexpr (DIM == 2) {
    const float2 v = *reinterpret_cast<const float2*>(p);
    pc[0] = v.x - pi[0];
    pc[1] = v.y - pi[1];
  } else {
#pragma unroll
    for (int k = 0; k < DIM; ++k) pc[k] = p[k] - pi[k];
  }
#pragma unroll
  for (int r = 0; r < DIM; ++r)
#pragma unroll
    for (int k = 0; k < DIM; ++k) dot2_acc(s[r], c[r], at(r * DIM + k), pc[k]);
}

template <int DIM, bool KEEP>
__device__ __forceinline__ void load_group(const PcgMixedArgs& a, const SliceGroups& sg, int pos, int lane,
                                           float4 (&v)[DIM * DIM], ushort4& l, unsigned own) {
  const int g = sg.tail ? pos - 1 : pos;
  if (g < 0) {
    const int64_t s = sg.base + (int64_t)sg.g4 * kSlice + lane;
    l = make_ushort4((unsigned short)own, (unsigned short)own, (unsigned short)own, (unsigned short)own);
#pragma unroll
    for (int e = 0; e < DIM * DIM; ++e) v[e] = make_float4(0.f, 0.f, 0.f, 0.f);
    // (at least one tail block here)
    l.x = a.lidx[s];
#pragma unroll
    for (int e = 0; e < DIM * DIM; ++e) v[e].x = a.A32[e * a.nslots + s];
    if (sg.tail > 1) {
      l.y = a.lidx[s + kSlice];
#pragma unroll
      for (int e = 0; e < DIM * DIM; ++e) v[e].y = a.A32[e * a.nslots + s + kSlice];
    }
    if (sg.tail > 2) {
      l.z = a.lidx[s + 2 * kSlice];
#pragma unroll
      for (int e = 0; e < DIM * DIM; ++e) v[e].z = a.A32[e * a.nslots + s + 2 * kSlice];
    }
    return;
  }
  const int64_t s = sg.base + (int64_t)g * (kSlice * kVec) + lane * kVec;
  l = __ldg(reinterpret_cast<const ushort4*>(a.lidx + s));
#pragma unroll
  for (int e = 0; e < DIM * DIM; ++e) {
    const float4* q = reinterpret_cast<const float4*>(a.A32 + e * a.nslots + s);
    v[e] = KEEP ? __ldg(q) : __ldcs(q);
  }
}

// The scalars of a solve.  Block 0 keeps them and decides; the others hold
// what its replies carry.  r.z, alpha and beta are FP32 pairs, as the sums
// they come from: an FP64 addition takes 65 cycles here and a division 400,
// every one of them on the path from one iteration to the next.
struct SolveState {
  float zh, zl;        // r.z
  float th, tl;        // threshold on |r|^2
  float rmax2;         // largest |r|^2 since the last reliable update
  float rrh, rrl;      // |r|^2
  float ah, al, bh, bl, zc;
  int done, ru, fail;
  long long it, maxit, ru_count;
};

struct PcgShared {
  SolveState st;
  float red[2][2][kPcgMaxSlices];
  double dred[2][kPcgMaxSlices];
  float ye[2][32];  // coarse correction: each warp's part of y.e
  int cdof0, cdof1, cagg0, cagg1, cent0, cent1;  // the block's coarse DOFs, aggregates and entries
  unsigned zn;  // publications of z
  int ubase[kPcgMaxSlices + 1];
};

// The kernel's shared memory: PcgShared, then the parts at a.off_*.  Every
// function takes it from here, so that the accesses stay shared-memory ones.
extern __shared__ __align__(16) unsigned char dyn[];
__device__ __forceinline__ PcgShared& block_state() { return *reinterpret_cast<PcgShared*>(dyn); }
__device__ __forceinline__ float* staged_p(const PcgMixedArgs& a) { return reinterpret_cast<float*>(dyn + a.off_p); }

// (qh, ql) = (ah, al) / (bh, bl): quotient digits of FP32 from the reciprocal,
// each with its remainder by FMA (long division); about 2^-46.  A divisor below
// 2.9e-39 has no FP32 reciprocal: the quotient is not finite, the solve ends as
// broken down (done = 3) and runs again in FP64.  r.z and p.q go with the inverse of
// the stiffness, so that is where a solve of constants past 1e15 at a tolerance
// of 1e-13, or 1e21 at 1e-10, ends.  Scaled into range here such solves went on
// with rows' products of few or no digits, and some never converged.
__device__ __forceinline__ void df_div(float ah, float al, float bh, float bl, float& qh, float& ql) {
  const float rc = __frcp_rn(bh);
  const float q1 = __fmul_rn(ah, rc);
  const float r1 = __fadd_rn(fmaf(-q1, bh, ah), fmaf(-q1, bl, al));
  float q2 = __fmul_rn(r1, rc);
  q2 = fmaf(fmaf(-q2, bh, r1), rc, q2);
  two_sum(q1, q2, qh, ql);
}

template <int DIM>
__device__ __forceinline__ void publish_z(const PcgMixedArgs& a, unsigned zn, int row, const float (&z)[DIM]) {
  st_rec(reinterpret_cast<Rec*>(a.zp) + (size_t)(zn & 1) * a.n + row, __float_as_uint(z[0]), __float_as_uint(z[1]),
         DIM == 3 ? __float_as_uint(z[DIM - 1]) : 0u, zn);
}

// The message warp's part of a grid sum of the reliable update: K <= 2 FP64
// values per block from sh.dred, the blocks' writes before it visible after
// it when `publish` is set (the fences).  In block 0 decide(), given the
// totals, updates the state and take({}, true) makes the reply's payload;
// take(reply, false) applies it in the other blocks.
template <int K, typename D, typename T>
__device__ __forceinline__ void update_sum(Rec* words, unsigned epoch, bool publish, PcgShared& sh, int S, D decide,
                                           T take, bool coarse = false) {
  SolveState& st = sh.st;
  const int G = gridDim.x, lane = threadIdx.x & 31;
  auto tagged = [&](const Rec& r) { return r.z == epoch; };
  auto fold = [](double s) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
  };
  if (publish) __threadfence();
#pragma unroll
  for (int k = 0; k < K; ++k) {
    double v = fold(lane < S ? sh.dred[k][lane] : 0.0);
    if (coarse && k == 0)
      v += fold(lane < (int)(blockDim.x >> 5) - 1 ? (double)sh.ye[0][lane] + (double)sh.ye[1][lane] : 0.0);
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    if (lane == 0)
      st_rec(arrivals(words, kArrUpdate + 2 * k, epoch & 1) + blockIdx.x, (unsigned)b, (unsigned)(b >> 32), epoch, 0u);
  }
  if (blockIdx.x == 0) {
    double tot[K];
    bool ok = true;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      Rec r[kPcgMaxBlocks / 32];
      ok = ok && gather_records(arrivals(words, kArrUpdate + 2 * k, epoch & 1), G, r, tagged);
      double s = 0.0;
#pragma unroll
      for (int q = 0; q < kPcgMaxBlocks / 32; ++q)
        if (lane + 32 * q < G) s += __longlong_as_double((long long)(((unsigned long long)r[q].y << 32) | r[q].x));
      tot[k] = fold(s);
    }
    if (publish) __threadfence();
    if (!ok) {
      if (lane == 0) st.fail = 1;
      return;
    }
    if (lane == 0) decide(tot);
    __syncwarp();
    if (publish) __threadfence();
    const Rec p = take(Rec{}, true);
    if (lane < kReplyCopies) st_rec(reply(words, epoch, lane), p.x, p.y, epoch, p.w);
  } else if (lane == 0) {
    Rec r;
    if (!poll_record(reply(words, epoch, blockIdx.x % kReplyCopies), r, tagged))
      st.fail = 1;
    else
      take(r, false);
    if (publish) __threadfence();
  }
}

// The warp's FP64 sums into sh.dred for the message warp.
template <int K>
__device__ __forceinline__ void warp_to_shared(PcgShared& sh, int ls, double (&v)[K]) {
  warp_sum<K>(v);
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int k = 0; k < K; ++k) sh.dred[k][ls] = v[k];
}

// ---- coarse correction  z = D^-1 r + P A_c^-1 P^T r  (lpm_coarse.cu) ----
// Three exchanges between the blocks, in records tagged like z: each block's
// part of y = P^T r for the aggregates its rows touch; y, each aggregate's
// parts summed by the block that has it (every block reading every part took
// 10k cycles, the reads in each other's way); and e = A_c^-1 y, of which each
// block works out a few entries (its rows of A_c^-1 stay in shared memory).
// r.z comes as r.D^-1 r + y.e, so that no third sum over the rows is needed;
// the e a block's rows need travel while block 0 forms beta.  Bound by those
// trips through L2, one after the other: us per iteration here against
// k_mx_persistent, whose grid barriers they replace, 61x121 plate (363 coarse
// DOFs) 19 (43), 201x401 plate 25 (43), 21^3 cube 25 (65), 41^3 cube 63 (87).
struct CoarseRow {
  float d[3];         // offset from the aggregate's centroid
  unsigned agg_mask;  // aggregate among the block's (low 16 bits), eliminated DOFs (bits 16..)
};
template <int DIM>
struct CoarseView {
  CoarseRow* row;     // [rows]
  float* r;           // [DIM][rows]: r's high words
  double* y;          // [nc]
  double* inv;        // the block's rows of A_c^-1
  float* e;           // the block's entries' e
  int *pos, *agg;     // the block's entries: place among all by aggregate, aggregate
  int rows;
};
template <int DIM>
__device__ __forceinline__ CoarseView<DIM> coarse_view(const PcgMixedArgs& a) {
  CoarseView<DIM> v;
  v.rows = a.maxS * kSlice;
  v.row = reinterpret_cast<CoarseRow*>(dyn + a.off_coarse);
  v.r = reinterpret_cast<float*>(v.row + v.rows);
  v.y = reinterpret_cast<double*>(v.r + DIM * v.rows);
  v.inv = v.y + a.nc;
  v.e = reinterpret_cast<float*>(v.inv + (size_t)a.cmaxrows * a.nc);
  v.pos = reinterpret_cast<int*>(v.e + a.cmaxagg * kModes<DIM>);
  v.agg = v.pos + a.cmaxagg;
  return v;
}
// The records of publication zn: parts of y by entry, y, e.
template <int DIM>
__device__ __forceinline__ Rec* coarse_records(const PcgMixedArgs& a, unsigned zn) {
  return reinterpret_cast<Rec*>(a.crec) + (size_t)(zn & 1) * ((size_t)a.centries * kModes<DIM> + 2 * (size_t)a.nc);
}

// From the rows' r (in v.r, a barrier of the compute warps before) to this
// block's e, published, and its part of y.e in sh.ye.
template <int DIM>
__device__ __forceinline__ void coarse_solve(const PcgMixedArgs& a, PcgShared& sh, unsigned zn, int S) {
  constexpr int NM = kModes<DIM>;
  const CoarseView<DIM> v = coarse_view<DIM>(a);
  const int nth = blockDim.x - 32, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = nth >> 5;
  Rec* parts = coarse_records<DIM>(a, zn);
  Rec* yrec = parts + (size_t)a.centries * NM;
  Rec* erec = yrec + a.nc;
  auto tagged = [&](const Rec& r) { return r.w == zn; };
  const int na = sh.cent1 - sh.cent0;
  for (int k = warp; k < na; k += nw) {
    float sm[NM], cm[NM];
#pragma unroll
    for (int m = 0; m < NM; ++m) sm[m] = cm[m] = 0.f;
    for (int s = 0; s < S; ++s) {
      const int q = s * kSlice + lane;
      const CoarseRow cr = v.row[q];
      if ((int)(cr.agg_mask & 0xffffu) != k) continue;
#pragma unroll
      for (int c = 0; c < DIM; ++c) {
        if (cr.agg_mask >> (16 + c) & 1u) continue;
        float w[NM];
        mode_row<DIM, float>(c, cr.d[0], cr.d[1], cr.d[2], w);
        const float rc = v.r[c * v.rows + q];
#pragma unroll
        for (int m = 0; m < NM; ++m)
          if (m == c || m >= DIM) dot2_acc(sm[m], cm[m], w[m], rc);
      }
    }
    warp_df_sum<NM>(sm, cm);
    float sl = sm[0], cl = cm[0];
#pragma unroll
    for (int m = 1; m < NM; ++m)
      if (lane == m) {
        sl = sm[m];
        cl = cm[m];
      }
    if (lane < NM) st_rec(parts + (size_t)v.pos[k] * NM + lane, __float_as_uint(sl), __float_as_uint(cl), 0u, zn);
  }
  // the block's aggregates: their parts in block order, a warp per DOF and a
  // lane per part (an aggregate of more than 32 parts in rounds)
  for (int c = sh.cagg0 * NM + warp; c < sh.cagg1 * NM; c += nw) {
    const int ag = c / NM, m = c % NM;
    float sv = 0.f, cv = 0.f;
    for (int q = a.cagg_ptr[ag] + lane; q < a.cagg_ptr[ag + 1]; q += 32) {
      Rec r;
      if (!poll_record(parts + (size_t)q * NM + m, r, tagged)) sh.st.fail = 1;
      df_add(sv, cv, __uint_as_float(r.x), __uint_as_float(r.y));
    }
    warp_df_sum(sv, cv);
    if (lane == 0) st_rec(yrec + c, __float_as_uint(sv), __float_as_uint(cv), 0u, zn);
  }
  for (int c = threadIdx.x; c < a.nc; c += nth) {
    Rec r;
    if (!poll_record(yrec + c, r, tagged)) sh.st.fail = 1;
    v.y[c] = (double)__uint_as_float(r.x) + (double)__uint_as_float(r.y);
  }
  compute_sync(nth);
  float ys = 0.f, yc = 0.f;
  for (int c = sh.cdof0 + warp; c < sh.cdof1; c += nw) {
    const double* row = v.inv + (size_t)(c - sh.cdof0) * a.nc;
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    int k = lane;
    for (; k + 96 < a.nc; k += 128) {
      s0 = fma(row[k], v.y[k], s0);
      s1 = fma(row[k + 32], v.y[k + 32], s1);
      s2 = fma(row[k + 64], v.y[k + 64], s2);
      s3 = fma(row[k + 96], v.y[k + 96], s3);
    }
    for (; k < a.nc; k += 32) s0 = fma(row[k], v.y[k], s0);
    double s[1] = {(s0 + s1) + (s2 + s3)};
    warp_sum<1>(s);
    if (lane == 0) {
      const float e = (float)s[0];
      st_rec(erec + c, __float_as_uint(e), 0u, 0u, zn);
      float ph, pl;
      df_split(v.y[c] * (double)e, ph, pl);
      df_add(ys, yc, ph, pl);
    }
  }
  if (lane == 0) {
    sh.ye[0][warp] = ys;
    sh.ye[1][warp] = yc;
  }
}

// The e of the block's aggregates, then z of this thread's row (owner).
template <int DIM>
__device__ __forceinline__ void coarse_row_z(const PcgMixedArgs& a, PcgShared& sh, unsigned zn, const Place& pl,
                                         float (&z)[DIM]) {
  constexpr int NM = kModes<DIM>, E = DIM * DIM;
  const CoarseView<DIM> v = coarse_view<DIM>(a);
  const int nth = blockDim.x - 32, lane = threadIdx.x & 31;
  const Rec* erec = coarse_records<DIM>(a, zn) + (size_t)a.centries * NM + a.nc;
  const int n = (sh.cent1 - sh.cent0) * NM;
  for (int q = threadIdx.x; q < n; q += nth) {
    Rec r;
    if (!poll_record(erec + v.agg[q / NM] * NM + q % NM, r, [&](const Rec& x) { return x.w == zn; })) sh.st.fail = 1;
    v.e[q] = __uint_as_float(r.x);
  }
  compute_sync(nth);
  if (pl.owner) {
    const int q = pl.ls * kSlice + lane;
    const CoarseRow cr = v.row[q];
    const float* rowc = reinterpret_cast<const float*>(dyn + a.off_row) + q;
    const float* e = v.e + (cr.agg_mask & 0xffffu) * NM;
#pragma unroll
    for (int k = 0; k < DIM; ++k) {
      float zi = rowc[(E + k) * v.rows] * v.r[k * v.rows + q];
      if (!(cr.agg_mask >> (16 + k) & 1u)) {
        float w[NM];
        mode_row<DIM, float>(k, cr.d[0], cr.d[1], cr.d[2], w);
#pragma unroll
        for (int m = 0; m < NM; ++m) zi = fmaf(w[m], e[m], zi);
      }
      z[k] = zi;
    }
    publish_z<DIM>(a, zn, pl.row, z);
  }
}

// Reliable update, compute warps: the solution x64 + x of every row
// published, then r64 = s b - A64 (x64 + x) and |r64|^2; unless that ends the
// solve, x64 += x, x = 0, r = r64 as a pair, z published, and r.z and r.p
// give beta and the direction coefficient that restores r.p = 0
// (k_mx_replace).  The message warp's side is update_messages.  (All three
// sums in one exchange measured slower: 8.5 us against 7.7 per iteration of
// a 41x41 plate.)
template <int DIM, bool COARSE>
__device__ __noinline__ void reliable_update(const PcgMixedArgs& a) {
  PcgShared& sh = block_state();
  SolveState& st = sh.st;
  const Place pl = place_of(a);
  const int lane = threadIdx.x & 31, nth = blockDim.x - 32;
  const int64_t i0 = (int64_t)pl.row * DIM;
  if (pl.owner)
#pragma unroll
    for (int k = 0; k < DIM; ++k)
      a.xs[i0 + k] = a.x64[i0 + k] + ((double)a.x[i0 + k] + (double)a.xlo[i0 + k]);
  if (pl.mine && lane == 0) sh.dred[0][pl.ls] = 0.0;
  __syncthreads();  // the solution published
  __syncthreads();
  if (st.fail) return;
  double y[DIM];
#pragma unroll
  for (int k = 0; k < DIM; ++k) y[k] = 0.0;
  if (pl.act && pl.row < a.n) {
    const SliceGroups sg = slice_groups(a.sell_ptr, pl.s0 + pl.ls);
#pragma unroll 1
    for (int g = pl.t; g < sg.g4 / kVec; g += a.T) {
      const int64_t s = sg.base + (int64_t)g * (kSlice * kVec) + lane * kVec;
      const int4 c4 = __ldg(reinterpret_cast<const int4*>(a.scol + s));
      const int cc[kVec] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
      for (int k = 0; k < DIM; ++k) {
        double pc[kVec];
#pragma unroll
        for (int q = 0; q < kVec; ++q) pc[q] = __ldcg(&a.xs[(int64_t)cc[q] * DIM + k]);
#pragma unroll
        for (int r = 0; r < DIM; ++r) {
          const double* v = a.A64 + (r * DIM + k) * a.nslots + s;
          const double2 lo = __ldcs(reinterpret_cast<const double2*>(v));
          const double2 hi = __ldcs(reinterpret_cast<const double2*>(v + 2));
          y[r] = fma(lo.x, pc[0], y[r]);
          y[r] = fma(lo.y, pc[1], y[r]);
          y[r] = fma(hi.x, pc[2], y[r]);
          y[r] = fma(hi.y, pc[3], y[r]);
        }
      }
    }
#pragma unroll 1
    for (int k = pl.t; k < sg.tail; k += a.T) {
      const int64_t s = sg.base + (int64_t)(sg.g4 + k) * kSlice + lane;
      const int64_t c = (int64_t)__ldg(&a.scol[s]) * DIM;
#pragma unroll
      for (int r = 0; r < DIM; ++r)
#pragma unroll
        for (int q = 0; q < DIM; ++q)
          y[r] = fma(__ldcs(a.A64 + (r * DIM + q) * a.nslots + s), __ldcg(&a.xs[c + q]), y[r]);
    }
  }
  if (a.T > 1) {
    double* pd = reinterpret_cast<double*>(dyn + a.off_part);
    if (pl.act && pl.t > 0)
#pragma unroll
      for (int k = 0; k < DIM; ++k) pd[(((pl.t - 1) * pl.S + pl.ls) * DIM + k) * 32 + lane] = y[k];
    compute_sync(nth);
    if (pl.owner)
      for (int w = 0; w + 1 < a.T; ++w)
#pragma unroll
        for (int k = 0; k < DIM; ++k) y[k] += pd[((w * pl.S + pl.ls) * DIM + k) * 32 + lane];
  }
  if (pl.mine) {
    double acc[1] = {0.0};
    if (pl.owner) {
      const double sc = a.cg->bscale;
#pragma unroll
      for (int k = 0; k < DIM; ++k) {
        y[k] = a.b[i0 + k] * sc - y[k];
        acc[0] += y[k] * y[k];
      }
    }
    warp_to_shared<1>(sh, pl.ls, acc);
  }
  __syncthreads();  // |r64|^2
  __syncthreads();
  if (st.fail || st.done) return;
  if (pl.mine) {
    double v[2] = {0.0, 0.0};
    if (pl.owner) {
      const unsigned own = (unsigned)(a.uown[blockIdx.x] + pl.ls * kSlice + lane);
      const float* ps = staged_p(a);
      float z[DIM];
#pragma unroll
      for (int k = 0; k < DIM; ++k) {
        a.x64[i0 + k] = a.xs[i0 + k];
        a.x[i0 + k] = 0.f;
        a.xlo[i0 + k] = 0.f;
        float rh, rl;
        df_split(y[k], rh, rl);
        a.r[i0 + k] = rh;
        a.rlo[i0 + k] = rl;
        z[k] = a.invd[i0 + k] * rh;
        v[0] += y[k] * (double)z[k];
        v[1] += y[k] * (double)ps[own * DIM + k];
        if (COARSE) coarse_view<DIM>(a).r[k * a.maxS * kSlice + pl.ls * kSlice + lane] = rh;
      }
      if (!COARSE) publish_z<DIM>(a, sh.zn + 1, pl.row, z);
    }
    warp_to_shared<2>(sh, pl.ls, v);
  }
  if (COARSE) {
    compute_sync(nth);
    coarse_solve<DIM>(a, sh, sh.zn + 1, pl.S);
  }
  __syncthreads();  // r.z, r.p
  if (COARSE) {
    float z[DIM];
    coarse_row_z<DIM>(a, sh, sh.zn + 1, pl, z);
    compute_sync(nth);
  }
  if (threadIdx.x == 0) sh.zn += 1;
  __syncthreads();
}

// Reliable update, message warp.
template <bool COARSE>
__device__ __noinline__ void update_messages(Rec* words, double threshold, unsigned epoch, int S) {
  PcgShared& sh = block_state();
  SolveState& st = sh.st;
  __syncthreads();
  update_sum<1>(words, ++epoch, true, sh, S, [](const double (&)[1]) {}, [](const Rec&, bool) { return Rec{}; });
  __syncthreads();
  if (st.fail) return;
  __syncthreads();
  update_sum<1>(
      words, ++epoch, false, sh, S,
      [&](const double (&tot)[1]) {
        df_split(tot[0], st.rrh, st.rrl);
        st.ru_count += 1;
        if (!isfinite(tot[0]))
          st.done = 3;
        else if (tot[0] < threshold)
          st.done = 1;
      },
      [&](const Rec& r, bool make) {
        if (make) return Rec{0u, 0u, 0u, (unsigned)(st.done != 0)};
        st.done = (int)r.w;
        return Rec{};
      });
  __syncthreads();
  if (st.fail || st.done) return;
  __syncthreads();
  update_sum<2>(
      words, ++epoch, false, sh, S,
      [&](const double (&tot)[2]) {
        const double beta = tot[0] / ((double)st.zh + (double)st.zl);
        df_split(tot[0], st.zh, st.zl);
        const double gamma = tot[0] != 0.0 ? tot[1] / tot[0] : 0.0;
        df_split(beta, st.bh, st.bl);
        st.zc = (float)(1.0 - beta * gamma);
        st.rmax2 = st.rrh;
        st.ru = 0;
      },
      [&](const Rec& r, bool make) {
        if (make) return Rec{__float_as_uint(st.bh), __float_as_uint(st.bl), 0u, __float_as_uint(st.zc)};
        st.bh = __uint_as_float(r.x);
        st.bl = __uint_as_float(r.y);
        st.zc = __uint_as_float(r.w);
        st.ru = 0;
        return Rec{};
      },
      COARSE);
  __syncthreads();
}

// The message warp's part of an iteration's first sum: p.q to block 0, alpha
// back.
__device__ __forceinline__ void alpha_sum(Rec* words, PcgShared& sh, unsigned m, unsigned epoch, int S) {
  SolveState& st = sh.st;
  const int lane = threadIdx.x & 31;
  float s = lane < S ? sh.red[0][0][lane] : 0.f, c = lane < S ? sh.red[0][1][lane] : 0.f;
  warp_df_sum(s, c);
  Rec* set = arrivals(words, kArrAlpha, m & 1);
  if (lane == 0) st_rec(set + blockIdx.x, __float_as_uint(s), __float_as_uint(c), 0u, m + 1);
  if (blockIdx.x == 0) {
    Rec r[kPcgMaxBlocks / 32];
    if (!gather_records(set, gridDim.x, r, [&](const Rec& q) { return q.w == m + 1; })) {
      st.fail = 1;
      return;
    }
    s = c = 0.f;
#pragma unroll
    for (int q = 0; q < kPcgMaxBlocks / 32; ++q)
      if (lane + 32 * q < (int)gridDim.x) df_add(s, c, __uint_as_float(r[q].x), __uint_as_float(r[q].y));
    warp_df_sum(s, c);
    float ah, al;
    df_div(st.zh, st.zl, s, c, ah, al);
    if (lane < kReplyCopies)
      st_rec(reply(words, epoch, lane), __float_as_uint(ah), __float_as_uint(al), epoch, 0u);
    if (lane == 0) {
      st.ah = ah;
      st.al = al;
    }
  } else if (lane == 0) {
    Rec r;
    if (!poll_record(reply(words, epoch, blockIdx.x % kReplyCopies), r, [&](const Rec& q) { return q.z == epoch; }))
      st.fail = 1;
    st.ah = __uint_as_float(r.x);
    st.al = __uint_as_float(r.y);
  }
}

// The second sum: |r|^2 and r.z to block 0, which forms beta and decides what
// the solve does next.  |r|^2 is not negative, so its sign bit is the
// arrival's tag (each copy is used every other iteration: one bit tells the
// new record from the old).  FIRST: before the first iteration of a solve with
// the coarse correction, the r.z of its first direction.
template <bool COARSE, bool FIRST = false>
__device__ __forceinline__ void beta_sum(Rec* words, PcgShared& sh, unsigned m, unsigned epoch, int S) {
  SolveState& st = sh.st;
  const int lane = threadIdx.x & 31;
  float s0 = lane < S ? sh.red[0][0][lane] : 0.f, c0 = lane < S ? sh.red[0][1][lane] : 0.f;
  float s1 = lane < S ? sh.red[1][0][lane] : 0.f, c1 = lane < S ? sh.red[1][1][lane] : 0.f;
  if (COARSE && lane < (int)(blockDim.x >> 5) - 1) df_add(s1, c1, sh.ye[0][lane], sh.ye[1][lane]);
  warp_df_sum(s0, c0);
  warp_df_sum(s1, c1);
  Rec* set = arrivals(words, kArrBeta, m & 1);
  const unsigned tag = ((m >> 1) & 1u) ^ 1u;
  if (lane == 0)
    st_rec(set + blockIdx.x, (__float_as_uint(s0) & 0x7fffffffu) | (tag << 31), __float_as_uint(c0),
           __float_as_uint(s1), __float_as_uint(c1));
  if (blockIdx.x == 0) {
    Rec r[kPcgMaxBlocks / 32];
    if (!gather_records(set, gridDim.x, r, [&](const Rec& q) { return (q.x >> 31) == tag; })) {
      st.fail = 1;
      return;
    }
    s0 = c0 = s1 = c1 = 0.f;
#pragma unroll
    for (int q = 0; q < kPcgMaxBlocks / 32; ++q)
      if (lane + 32 * q < (int)gridDim.x) {
        df_add(s0, c0, __uint_as_float(r[q].x & 0x7fffffffu), __uint_as_float(r[q].y));
        df_add(s1, c1, __uint_as_float(r[q].z), __uint_as_float(r[q].w));
      }
    warp_df_sum(s0, c0);
    warp_df_sum(s1, c1);
    // every lane decides alike; lane 0 keeps the state
    float rr, rrl, rz, rzl, bh = 0.f, bl = 0.f;
    two_sum(s0, c0, rr, rrl);
    two_sum(s1, c1, rz, rzl);
    const long long it = st.it + (FIRST ? 0 : 1);
    int done = 0, ru = 0;
    if (!isfinite(rr) || !isfinite(rz)) {
      done = 3;
    } else if (!FIRST) {
      ru = rr < st.th || (rr == st.th && rrl < st.tl) || rr < (float)kRuDelta2 * st.rmax2;
      if (!ru) df_div(rz, rzl, st.zh, st.zl, bh, bl);
      if (it >= st.maxit) done = 2;
    }
    if (lane < kReplyCopies)
      st_rec(reply(words, epoch, lane), __float_as_uint(bh), __float_as_uint(bl), epoch,
             (unsigned)(done != 0) | (unsigned)ru << 1);
    __syncwarp();
    if (lane == 0) {
      st.it = it;
      st.rrh = rr;
      st.rrl = rrl;
      st.done = done;
      st.ru = ru;
      if (!ru && done != 3) {
        st.rmax2 = fmaxf(st.rmax2, rr);
        st.zh = rz;
        st.zl = rzl;
        st.bh = bh;
        st.bl = bl;
        st.zc = 1.f;
      }
    }
  } else if (lane == 0) {
    Rec r;
    if (!poll_record(reply(words, epoch, blockIdx.x % kReplyCopies), r, [&](const Rec& q) { return q.z == epoch; }))
      st.fail = 1;
    st.bh = __uint_as_float(r.x);
    st.bl = __uint_as_float(r.y);
    st.zc = 1.f;
    st.done = (int)(r.w & 1u);
    st.ru = (int)(r.w >> 1 & 1u);
  }
}

// The message warp's loop.
template <bool COARSE>
__device__ __noinline__ void messages(Rec* words, CgScalars* cg, int S) {
  PcgShared& sh = block_state();
  SolveState& st = sh.st;
  const int lane = threadIdx.x & 31;
  unsigned epoch = 0, mb = 0;  // replies, second sums
  if (COARSE) {
    __syncthreads();
    beta_sum<true, true>(words, sh, mb++, ++epoch, S);
    __syncthreads();
  }
#pragma unroll 1
  for (unsigned m = 0; !(COARSE && (st.fail || st.done)); ++m) {
    __syncthreads();
    alpha_sum(words, sh, m, ++epoch, S);
    __syncthreads();
    if (st.fail) break;
    __syncthreads();
    beta_sum<COARSE>(words, sh, mb++, ++epoch, S);
    __syncthreads();
    if (st.fail || st.done) break;
    if (st.ru) {
      update_messages<COARSE>(words, cg->threshold, epoch, S);
      epoch += 3;
      if (st.fail || st.done) break;
    }
  }
  if (lane == 0 && st.fail) atomicExch(&cg->pfault, 1);
  if (blockIdx.x == 0 && lane == 0 && !st.fail) {
    cg->done = st.done;
    cg->rr = (double)st.rrh + (double)st.rrl;
    cg->it = st.it;
    cg->abs_new = (double)st.zh + (double)st.zl;
    cg->rmax = sqrt((double)st.rmax2);
    cg->ru = st.ru;
    cg->ru_count = st.ru_count;
    cg->graph_passes = st.it;
  }
}

// The compute warps' iterations up to the next reliable update or the end.
// (The reliable update and the messages are out of line: they keep no
// registers from it.)
template <int DIM, bool KEEP, bool COARSE>
__device__ __forceinline__ void iterate(const PcgMixedArgs& a) {
  PcgShared& sh = block_state();
  constexpr int E = DIM * DIM;
  constexpr int kAhead = 4;  // columns of a thread fetched ahead
  constexpr int kBlk = kPcgUnit<DIM> / kVec;
  SolveState& st = sh.st;
  const Place pl = place_of(a);
  const int S = pl.S, ls = pl.ls, t = pl.t, lane = threadIdx.x & 31;
  const bool act = pl.act, mine = pl.mine, owner = pl.owner;
  const int U = a.ucnt[blockIdx.x];
  const int nth = blockDim.x - 32;  // compute threads
  float* ps = staged_p(a);
  const int* ul = reinterpret_cast<const int*>(dyn + a.off_list);
  float* part = reinterpret_cast<float*>(dyn + a.off_part);
  const float* rowc = reinterpret_cast<const float*>(dyn + a.off_row) + ls * kSlice + lane;
  const int rstride = a.maxS * kSlice;
  const unsigned own = pl.row < a.n ? (unsigned)(a.uown[blockIdx.x] + ls * kSlice + lane) : 0u;
  const SliceGroups sg = slice_groups(a.sell_ptr, pl.s0 + ls);
  const int res = min(sg.count, a.gs + (ls < a.gx ? 1 : 0));  // groups kept in shared memory
  const unsigned char* unit = dyn + a.off_op + (size_t)sh.ubase[ls] * kPcgUnit<DIM>;
  unsigned zn = sh.zn;
  float rh[DIM], rl[DIM];
#pragma unroll
  for (int k = 0; k < DIM; ++k) {
    rh[k] = owner ? a.r[(int64_t)pl.row * DIM + k] : 0.f;
    rl[k] = owner ? a.rlo[(int64_t)pl.row * DIM + k] : 0.f;
  }
  // the first kAhead of this thread's columns, asked for once while the sums
  // travel (asking on and on would crowd out their records) and then, where
  // the record had not come, when they are back
  float zq[kAhead][DIM];
  unsigned need = 0;
  auto ask = [&]() {
    const Rec* zb = reinterpret_cast<const Rec*>(a.zp) + (size_t)(zn & 1) * a.n;
#pragma unroll
    for (int q = 0; q < kAhead; ++q)
      if (need >> q & 1u) {
        const Rec r = ld_rec(zb + ul[threadIdx.x + q * nth]);
        zq[q][0] = __uint_as_float(r.x);
        zq[q][1] = __uint_as_float(r.y);
        if (DIM == 3) zq[q][DIM - 1] = __uint_as_float(r.z);
        if (r.w == zn) need &= ~(1u << q);
      }
  };
  auto ask_first = [&]() {
    need = 0;
#pragma unroll
    for (int q = 0; q < kAhead; ++q)
      if ((int)threadIdx.x + q * nth < U) need |= 1u << q;
    ask();
  };
  ask_first();
  for (;;) {
    // p = zc z + beta p at the block's columns
    {
      for (long long polls = 0; need; ++polls) {
        ask();
        if (polls > kPollLimit) {
          st.fail = 1;
          break;
        }
      }
      const float bh = st.bh, bl = st.bl, zc = st.zc;
#pragma unroll
      for (int q = 0; q < kAhead; ++q) {
        const int u = threadIdx.x + q * nth;
        if (u < U)
#pragma unroll
          for (int k = 0; k < DIM; ++k) {
            const float p = ps[u * DIM + k];
            ps[u * DIM + k] = fmaf(bh, p, fmaf(bl, p, __fmul_rn(zc, zq[q][k])));
          }
      }
      const Rec* zb = reinterpret_cast<const Rec*>(a.zp) + (size_t)(zn & 1) * a.n;
#pragma unroll 1
      for (int u = threadIdx.x + kAhead * nth; u < U; u += nth) {
        Rec r;
        if (!poll_record(zb + ul[u], r, [&](const Rec& q) { return q.w == zn; })) st.fail = 1;
        const float z[3] = {__uint_as_float(r.x), __uint_as_float(r.y), __uint_as_float(r.z)};
#pragma unroll
        for (int k = 0; k < DIM; ++k) {
          const float p = ps[u * DIM + k];
          ps[u * DIM + k] = fmaf(bh, p, fmaf(bl, p, __fmul_rn(zc, z[k])));
        }
      }
    }
    compute_sync(nth);
    // q = A p in difference form (double-float), this warp's share of its slice's groups
    float qh[DIM], ql[DIM];
#pragma unroll
    for (int k = 0; k < DIM; ++k) qh[k] = ql[k] = 0.f;
    if (act) {
      float pi[DIM];
#pragma unroll
      for (int k = 0; k < DIM; ++k) pi[k] = ps[own * DIM + k];
      // the first streamed group is on its way while the resident ones are multiplied
      float4 an[E];
      ushort4 ln;
      int kn = res + ((t - res) % a.T + a.T) % a.T;  // first position >= res of this warp's share
      if (kn < sg.count) load_group<DIM, KEEP>(a, sg, kn, lane, an, ln, own);
#pragma unroll 1
      for (int k = t; k < res; k += a.T) {
#pragma unroll
        for (int q = 0; q < kVec; ++q) {
          const float* b = reinterpret_cast<const float*>(unit + (size_t)k * kPcgUnit<DIM> + q * kBlk);
          const unsigned l = reinterpret_cast<const unsigned short*>(b + E * 32)[lane];
          block_acc<DIM>([&](int e) { return b[e * 32 + lane]; }, ps + l * DIM, pi, qh, ql);
        }
      }
#pragma unroll 1
      while (kn < sg.count) {
        kn += a.T;
#pragma unroll
        for (int q = 0; q < kVec; ++q)
          block_acc<DIM>([&](int e) { return comp_f(an[e], q); }, ps + comp_u16(ln, q) * DIM, pi, qh, ql);
        if (kn < sg.count) load_group<DIM, KEEP>(a, sg, kn, lane, an, ln, own);
      }
    }
    // the block row sum's term, by the slice's last share
    if (act && t == a.T - 1 && pl.row < a.n)
#pragma unroll
      for (int r = 0; r < DIM; ++r)
#pragma unroll
        for (int k = 0; k < DIM; ++k) dot2_acc(qh[r], ql[r], rowc[(r * DIM + k) * rstride], ps[own * DIM + k]);
    if (a.T > 1) {
      if (act && t > 0)
#pragma unroll
        for (int k = 0; k < DIM; ++k) {
          part[((t - 1) * S + ls) * 64 * DIM + k * 64 + lane] = qh[k];
          part[((t - 1) * S + ls) * 64 * DIM + k * 64 + 32 + lane] = ql[k];
        }
      compute_sync(nth);
      if (mine)
#pragma unroll 4
        for (int w = 0; w + 1 < a.T; ++w)
#pragma unroll
          for (int k = 0; k < DIM; ++k)
            df_add(qh[k], ql[k], part[(w * S + ls) * 64 * DIM + k * 64 + lane],
                   part[(w * S + ls) * 64 * DIM + k * 64 + 32 + lane]);
    }
    // the pair normalised, p.q
    if (mine) {
      float sp = 0.f, cp = 0.f;
      if (owner) {
#pragma unroll
        for (int r = 0; r < DIM; ++r) {
          float y, yl;
          two_sum(qh[r], ql[r], y, yl);
          qh[r] = y;
          ql[r] = yl;
          dot2_acc(sp, cp, ps[own * DIM + r], y);
          cp = fmaf(ps[own * DIM + r], yl, cp);
        }
      }
      warp_df_sum(sp, cp);
      if (lane == 0) {
        sh.red[0][0][ls] = sp;
        sh.red[0][1][ls] = cp;
      }
    }
    __syncthreads();  // p.q
    __syncthreads();
    if (st.fail) break;
    // r -= alpha q, z = M r published, |r|^2 and r.z
    ++zn;
    if (mine) {
      const float ah = st.ah, al = st.al;
      float sb[2] = {0.f, 0.f}, cb[2] = {0.f, 0.f};
      if (owner) {
        float z[DIM];
#pragma unroll
        for (int k = 0; k < DIM; ++k) {
          df_madd(rh[k], rl[k], -ah, -al, qh[k], ql[k]);
          z[k] = rowc[(E + k) * rstride] * rh[k];
          if (COARSE) coarse_view<DIM>(a).r[k * rstride + ls * kSlice + lane] = rh[k];
        }
        if (!COARSE) publish_z<DIM>(a, zn, pl.row, z);
#pragma unroll
        for (int k = 0; k < DIM; ++k) {
          dot2_acc(sb[0], cb[0], rh[k], rh[k]);
          cb[0] = fmaf(2.f * rh[k], rl[k], cb[0]);
          dot2_acc(sb[1], cb[1], rh[k], z[k]);
          cb[1] = fmaf(rl[k], z[k], cb[1]);
        }
      }
      warp_df_sum(sb[0], cb[0]);
      warp_df_sum(sb[1], cb[1]);
      if (lane == 0)
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          sh.red[k][0][ls] = sb[k];
          sh.red[k][1][ls] = cb[k];
        }
    }
    if (COARSE) {
      compute_sync(nth);
      coarse_solve<DIM>(a, sh, zn, S);
    }
    __syncthreads();  // |r|^2, r.z
    if (COARSE) {
      float z[DIM];
      coarse_row_z<DIM>(a, sh, zn, pl, z);
    }
    // while the sums travel: x += alpha p, and the z of the block's columns
    if (owner) {
      const float ah = st.ah, al = st.al;
      const int64_t i0 = (int64_t)pl.row * DIM;
#pragma unroll
      for (int k = 0; k < DIM; ++k) {
        float xh = a.x[i0 + k], xl = a.xlo[i0 + k];
        df_madd(xh, xl, ah, al, ps[own * DIM + k], 0.f);
        a.x[i0 + k] = xh;
        a.xlo[i0 + k] = xl;
      }
    }
    ask_first();
    __syncthreads();
    if (st.fail || st.done) break;
    if (st.ru) break;
  }
  // a reliable update works on r in global memory
  if (owner && st.ru) {
    const int64_t i0 = (int64_t)pl.row * DIM;
#pragma unroll
    for (int k = 0; k < DIM; ++k) {
      a.r[i0 + k] = rh[k];
      a.rlo[i0 + k] = rl[k];
    }
  }
  if (threadIdx.x == 0) sh.zn = zn;
}

template <int DIM, bool KEEP, int BOUND, bool COARSE>
__global__ void __launch_bounds__(BOUND, 1) k_pcg_mixed(const __grid_constant__ PcgMixedArgs a) {
  constexpr int E = DIM * DIM;
  PcgShared& sh = block_state();
  SolveState& st = sh.st;
  const Place pl = place_of(a);
  const int S = pl.S, ls = pl.ls, t = pl.t, lane = threadIdx.x & 31;
  const int U = a.ucnt[blockIdx.x];
  const int nth = blockDim.x - 32;  // compute threads
  float* ps = staged_p(a);
  const int* ul = reinterpret_cast<const int*>(dyn + a.off_list);
  // the row's constants, [E + DIM][rows of the block]: block row sum, diagonal
  float* rowc = reinterpret_cast<float*>(dyn + a.off_row) + ls * kSlice + lane;
  const int rstride = a.maxS * kSlice;
  const bool comm = (int)threadIdx.x >= nth;
  const bool act = !comm && pl.act, mine = !comm && pl.mine, owner = !comm && pl.owner;
  const unsigned own = pl.row < a.n ? (unsigned)(a.uown[blockIdx.x] + ls * kSlice + lane) : 0u;
  const SliceGroups sg = slice_groups(a.sell_ptr, pl.s0 + ls);
  const int res = min(sg.count, a.gs + (ls < a.gx ? 1 : 0));  // groups kept in shared memory
  if (threadIdx.x == 0) {
    int at = 0;
    for (int k = 0; k < S; ++k) {
      sh.ubase[k] = at;
      at += min(slice_groups(a.sell_ptr, pl.s0 + k).count, a.gs + (k < a.gx ? 1 : 0));
    }
    const CgScalars* c = a.cg;
    df_split(c->abs_new, st.zh, st.zl);
    df_split(c->threshold, st.th, st.tl);
    st.rmax2 = (float)(c->rmax * c->rmax);
    st.rrh = st.rrl = 0.f;
    st.it = c->it;
    st.maxit = c->maxit;
    st.ru_count = c->ru_count;
    st.done = c->done;
    st.ru = st.fail = 0;
    st.ah = st.al = st.bh = st.bl = 0.f;
    st.zc = 1.f;
    sh.zn = 1;
    if (COARSE) {
      constexpr int NM = kModes<DIM>;
      sh.cdof0 = plan_slice(blockIdx.x, gridDim.x, a.nc);
      sh.cdof1 = plan_slice(blockIdx.x + 1, gridDim.x, a.nc);
      sh.cagg0 = plan_slice(blockIdx.x, gridDim.x, a.nc / NM);
      sh.cagg1 = plan_slice(blockIdx.x + 1, gridDim.x, a.nc / NM);
      sh.cent0 = a.cblk_ptr[blockIdx.x];
      sh.cent1 = a.cblk_ptr[blockIdx.x + 1];
    }
  }
  for (int u = threadIdx.x; u < U; u += blockDim.x) {
    const_cast<int*>(ul)[u] = a.ulist[(int64_t)blockIdx.x * a.umax + u];
#pragma unroll
    for (int k = 0; k < DIM; ++k) ps[u * DIM + k] = 0.f;
  }
  __syncthreads();
  if (st.done) return;  // the same in every block
  if (comm) {
    messages<COARSE>(reinterpret_cast<Rec*>(a.words), a.cg, S);
    return;
  }
  // the resident groups, block by block: the E elements and then the
  // position of each of the 32 rows
  constexpr int kBlk = kPcgUnit<DIM> / kVec;
  unsigned char* unit = dyn + a.off_op + (size_t)sh.ubase[ls] * kPcgUnit<DIM>;
  if (act)
    for (int k = t; k < res; k += a.T) {
      float4 v[E];
      ushort4 l;
      load_group<DIM, KEEP>(a, sg, k, lane, v, l, own);
#pragma unroll
      for (int q = 0; q < kVec; ++q) {
        float* b = reinterpret_cast<float*>(unit + (size_t)k * kPcgUnit<DIM> + q * kBlk);
#pragma unroll
        for (int e = 0; e < E; ++e) b[e * 32 + lane] = comp_f(v[e], q);
        reinterpret_cast<unsigned short*>(b + E * 32)[lane] = (unsigned short)comp_u16(l, q);
      }
    }
  if (owner) {
    const int64_t i0 = (int64_t)pl.row * DIM;
    float z[DIM];
#pragma unroll
    for (int k = 0; k < DIM; ++k) {
      const float iv = a.invd[i0 + k];
      rowc[(E + k) * rstride] = iv;
      z[k] = iv * a.r[i0 + k];
    }
#pragma unroll
    for (int e = 0; e < E; ++e) rowc[e * rstride] = a.S32[(int64_t)pl.row * E + e];
    // z of every row, tagged with the number of its publication, in two
    // copies by that number's parity: a block can be one publication ahead of
    // a slow reader, never two (a reader's next arrival comes after its reads)
    if (!COARSE) publish_z<DIM>(a, 1, pl.row, z);
  }
  if (COARSE) {
    // the rows' places in the aggregates, the block's rows of A_c^-1, and the
    // coarse-corrected z of the initial residual
    const CoarseView<DIM> v = coarse_view<DIM>(a);
    if (mine) {
      CoarseRow cr{{0.f, 0.f, 0.f}, 0xffffu};
      if (owner) {
        cr.agg_mask = a.crow[pl.row];
#pragma unroll
        for (int k = 0; k < 3; ++k) cr.d[k] = a.coff[3 * (int64_t)pl.row + k];
#pragma unroll
        for (int k = 0; k < DIM; ++k) {
          if (a.cfixed && a.cfixed[(int64_t)pl.row * DIM + k]) cr.agg_mask |= 1u << (16 + k);
          v.r[k * v.rows + ls * kSlice + lane] = a.r[(int64_t)pl.row * DIM + k];
        }
      }
      v.row[ls * kSlice + lane] = cr;
    }
    for (int e = threadIdx.x; e < (sh.cdof1 - sh.cdof0) * a.nc; e += nth)
      v.inv[e] = a.cAinv[(int64_t)sh.cdof0 * a.nc + e];
    for (int e = threadIdx.x; e < sh.cent1 - sh.cent0; e += nth) {
      v.pos[e] = a.cblk_pos[sh.cent0 + e];
      v.agg[e] = a.cblk_agg[sh.cent0 + e];
    }
    float s0 = 0.f, c0 = 0.f, s1 = 0.f, c1 = 0.f;
    if (owner)
#pragma unroll
      for (int k = 0; k < DIM; ++k) {
        const int64_t i = (int64_t)pl.row * DIM + k;
        const float rh = a.r[i], z = rowc[(E + k) * rstride] * rh;
        dot2_acc(s0, c0, rh, rh);
        dot2_acc(s1, c1, rh, z);
        c1 = fmaf(a.rlo[i], z, c1);
      }
    if (mine) {
      warp_df_sum(s0, c0);
      warp_df_sum(s1, c1);
      if (lane == 0) {
        sh.red[0][0][ls] = s0;
        sh.red[0][1][ls] = c0;
        sh.red[1][0][ls] = s1;
        sh.red[1][1][ls] = c1;
      }
    }
    compute_sync(nth);
    coarse_solve<DIM>(a, sh, 1, S);
    __syncthreads();
    float z[DIM];
    coarse_row_z<DIM>(a, sh, 1, pl, z);
    __syncthreads();
    if (st.fail || st.done) return;
  }
  compute_sync(nth);
  for (;;) {
    iterate<DIM, KEEP, COARSE>(a);
    if (st.fail || st.done) break;
    reliable_update<DIM, COARSE>(a);
    if (st.fail || st.done) break;
  }
}

}  // namespace

// No memory for the plan: the other loops need none of it.
static int pcg_no_memory(lpm_handle* h) {
  cudaGetLastError();
  h->err.clear();
  return 0;
}

// The column plan of the handle's pattern, once, for a solve of at most `slices`
// to a block: 1 if it can run on the plan, 0 if not (more slices, or no
// cooperative launch), or an error.
int pcg_plan(lpm_handle* h, int slices) {
  PcgPlan& pl = h->pcg;
  if (pl.state) return pl.state > 0 && pl.S <= slices;
  if (!sm_count(h)) return 0;
  const int G = std::min(std::min(h->sms, kPcgMaxBlocks), h->nslice);
  const int S = (h->nslice + G - 1) / G;
  if (S > slices) return 0;
  pl.state = -1;
  Dev& d = h->d;
  int coop = 0, smem = 0, sm_smem = 0, reserved = 0;
  if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, h->device) != cudaSuccess || !coop) return 0;
  if (cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, h->device) != cudaSuccess ||
      cudaDeviceGetAttribute(&sm_smem, cudaDevAttrMaxSharedMemoryPerMultiprocessor, h->device) != cudaSuccess ||
      cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, h->device) != cudaSuccess)
    return 0;
  const int words = (h->n + 31) / 32;
  if ((size_t)words * 8 + sizeof(int) * kPlanThreads > 48 * 1024) return 0;  // (k_plan_fill's)
  d.pl_ucnt = (int*)dev_alloc(h, sizeof(int) * G);
  d.pl_uown = (int*)dev_alloc(h, sizeof(int) * G);
  if (!d.pl_ucnt || !d.pl_uown) return pcg_no_memory(h);
  LPM_CUDA(h, cudaMemsetAsync(d.pl_ucnt, 0, sizeof(int) * G, h->stream));
  k_plan_count<<<G, kPlanThreads, (size_t)words * 4, h->stream>>>(h->n, h->nslice, d.sell_ptr, d.scol, d.rowlen,
                                                                  d.pl_ucnt);
  LPM_LAUNCHED(h, "k_plan_count");
  std::vector<int> cnt((size_t)G);
  LPM_CUDA(h, cudaMemcpyAsync(cnt.data(), d.pl_ucnt, sizeof(int) * G, cudaMemcpyDeviceToHost, h->stream));
  LPM_CUDA(h, cudaStreamSynchronize(h->stream));
  const int umax = *std::max_element(cnt.begin(), cnt.end());
  if (umax > 65535) return 0;
  d.pl_ulist = (int*)dev_alloc(h, sizeof(int) * (size_t)G * umax);
  d.pl_lidx = (unsigned short*)dev_alloc(h, sizeof(unsigned short) * (size_t)std::max<int64_t>(h->nslots, 1));
  d.pl_words = (unsigned long long*)dev_alloc(h, kWordBytes);
  d.pl_zp = (float*)dev_alloc(h, kZBytes64 * (size_t)h->n);
  if (!d.pl_ulist || !d.pl_lidx || !d.pl_words || !d.pl_zp) return pcg_no_memory(h);
  // slots of the rows past the last particle stay at position 0
  LPM_CUDA(h, cudaMemsetAsync(d.pl_lidx, 0, sizeof(unsigned short) * (size_t)std::max<int64_t>(h->nslots, 1),
                              h->stream));
  k_plan_fill<<<G, kPlanThreads, (size_t)words * 8, h->stream>>>(h->n, h->nslice, d.sell_ptr, d.scol, d.rowlen, umax,
                                                                 d.pl_ulist, d.pl_uown, d.pl_lidx);
  LPM_LAUNCHED(h, "k_plan_fill");
  pl.G = G;
  pl.S = S;
  pl.umax = umax;
  pl.smem = smem;
  pl.half = sm_smem / 2 - reserved;
  pl.state = 1;
  return 1;
}

namespace {

size_t align16(size_t b) { return (b + 15) / 16 * 16; }

// Launch shape of a solve on the plan, worked out once per handle: the
// staged vector, its columns, the row data, then as many operator groups per
// slice as fit, gs of every slice and one more of a block's first gx.
// `unit` is a group's bytes, `threads` the most per block, `vec` the bytes of
// a staged entry, `part` of a row's partial sums of one share, `rowc` of a
// row's constants, `coarse` of the coarse correction.
// maxw compute warps and smem bytes at most; `share`: only if all groups fit, in
// blocks of which an SM holds two.
bool shape_with(const lpm_handle* h, const void* fn, int maxw, int smem, bool share, size_t unit, size_t vec,
                size_t part, size_t rowc, size_t coarse, PcgShape* sh) {
  const PcgPlan& pl = h->pcg;
  if (pl.S > maxw) return false;
  auto groups = [&](int s) {
    const int w = (int)((h->sell_host[(size_t)s + 1] - h->sell_host[(size_t)s]) / kSlice);
    return (w + kVec - 1) / kVec;
  };
  int gmax = 0;  // most groups in a slice
  for (int s = 0; s < h->nslice; ++s) gmax = std::max(gmax, groups(s));
  sh->T = std::max(1, std::min(maxw / pl.S, gmax));
  sh->off_p = (int)align16(sizeof(PcgShared));
  sh->off_list = sh->off_p + (int)align16(vec * pl.umax);
  sh->off_part = sh->off_list + (int)align16(sizeof(int) * pl.umax);
  sh->off_row = sh->off_part + (int)align16(part * (size_t)(sh->T - 1) * pl.S * 32);
  sh->off_coarse = sh->off_row + (int)align16(rowc * (size_t)pl.S * 32);
  sh->off_op = sh->off_coarse + (int)align16(coarse);
  const long long room = (long long)smem - sh->off_op;
  if (room < 0) return false;
  size_t units = 0;
  sh->gs = sh->gx = 0;
  for (int g = 0; g < gmax; ++g)
    for (int x = 1; x <= pl.S; ++x) {
      size_t most = 0;  // in the fullest block
      for (int b = 0; b < pl.G; ++b) {
        size_t u = 0;
        const int s0 = plan_slice(b, pl.G, h->nslice), s1 = plan_slice(b + 1, pl.G, h->nslice);
        for (int s = s0; s < s1; ++s) u += (size_t)std::min(g + (s - s0 < x ? 1 : 0), groups(s));
        most = std::max(most, u);
      }
      if ((long long)(most * unit) > room) {
        g = gmax;
        break;
      }
      sh->gs = g;
      sh->gx = x;
      units = most;
    }
  if (share && sh->gs + (sh->gx == pl.S ? 1 : 0) < gmax) return false;
  sh->bytes = (size_t)sh->off_op + units * unit;
  // (warps without a share still take their part in the coarse correction)
  sh->threads = (share && coarse ? maxw + 1 : pl.S * sh->T + 1) * 32;
  int per_sm = 0;
  // (the attribute belongs to the kernel, not to the handle: always the most)
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, pl.smem) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, sh->threads, sh->bytes) != cudaSuccess ||
      per_sm < (share ? 2 : 1)) {
    cudaGetLastError();
    return false;
  }
  return true;
}

// Once per handle.  Blocks of up to two slices take seven compute warps at most
// and half an SM, where their groups fit it, so that the solves of several small
// systems, from several threads, run beside each other; with fifteen warps they
// took turns.  us per iteration alone, with fifteen warps and with seven: a 41x41
// plate 7.1 and 7.2, 61x121 7.1 and 6.9, a 12^3 cube 9.7 and 9.6; of four handles
// solved at once (over all their iterations) 3.5 and 1.9, 7.0 and 3.7, 4.7 and 2.8.
// (With k_mx_persistent, whose blocks are smaller still, 4.2, 4.3 and 7.6.)
constexpr int kSharingWarps = 7;

bool shape_on_plan(const lpm_handle* h, const void* fn, int threads, size_t unit, size_t vec, size_t part,
                   size_t rowc, size_t coarse, PcgShape* sh) {
  const PcgPlan& pl = h->pcg;
  return (pl.S <= kSharingSlices &&
          shape_with(h, fn, kSharingWarps, pl.half, true, unit, vec, part, rowc, coarse, sh)) ||
         shape_with(h, fn, threads / 32 - 1, pl.smem, false, unit, vec, part, rowc, coarse, sh);
}

template <int DIM, bool COARSE>
int run_mixed_dim(lpm_handle* h, bool keep) {
  Dev& d = h->d;
  PcgPlan& pl = h->pcg;
  using Fn = void (*)(PcgMixedArgs);
  constexpr int kBound = kPcgThreads<DIM>, kWide = kPcgWideThreads<DIM>, kNarrow = kPcgNarrowThreads;
  const bool wide = (pl.S + 1) * 32 > kBound;
  // the narrow form, unless it has a warp for each slice where the other has two
  const int share = (kNarrow / 32 - 1) / pl.S;
  const bool narrow = DIM == 2 && share > 0 && (share > 1 || (kBound / 32 - 1) / pl.S == 1);
  const Fn fn = narrow ? k_pcg_mixed<DIM, true, kNarrow, COARSE>
                : wide ? (keep ? k_pcg_mixed<DIM, true, kWide, COARSE> : k_pcg_mixed<DIM, false, kWide, COARSE>)
                       : (keep ? k_pcg_mixed<DIM, true, kBound, COARSE> : k_pcg_mixed<DIM, false, kBound, COARSE>);
  PcgShape& sh = COARSE ? pl.mixed_coarse : pl.mixed;
  const int cmaxrows = COARSE ? (h->cnc + pl.G - 1) / pl.G : 0;
  if (!sh.state) {
    const size_t rows = (size_t)pl.S * kSlice;
    const size_t coarse = COARSE ? rows * (sizeof(CoarseRow) + sizeof(float) * DIM) +
                                       sizeof(double) * (size_t)(1 + cmaxrows) * h->cnc +
                                       (sizeof(float) * kModes<DIM> + 2 * sizeof(int)) * (size_t)pl.cmaxagg
                                 : 0;
    sh.state = shape_on_plan(h, (const void*)fn, narrow ? kNarrow : wide ? kWide : kBound, kPcgUnit<DIM>, sizeof(float) * DIM,
                             sizeof(double) * DIM, sizeof(float) * (DIM * DIM + DIM), coarse, &sh)
                   ? 1
                   : -1;
  }
  if (sh.state < 0) return 0;
  PcgMixedArgs a{};
  a.sell_ptr = d.sell_ptr;
  a.ucnt = d.pl_ucnt;
  a.uown = d.pl_uown;
  a.ulist = d.pl_ulist;
  a.lidx = d.pl_lidx;
  a.scol = d.scol;
  a.A32 = d.A32;
  a.S32 = d.S32;
  a.A64 = d.A64;
  a.b = d.rhs;
  a.invd = d.invd32;
  a.r = d.r32;
  a.rlo = d.r32lo;
  a.x = d.x32;
  a.xlo = d.x32lo;
  a.x64 = d.x64;
  a.xs = d.p64;
  a.zp = d.pl_zp;
  a.words = d.pl_words;
  a.cg = d.cg;
  a.nslots = h->nslots;
  a.n = h->n;
  a.nslice = h->nslice;
  a.umax = pl.umax;
  a.maxS = pl.S;
  a.gs = sh.gs;
  a.gx = sh.gx;
  a.T = sh.T;
  a.off_p = sh.off_p;
  a.off_list = sh.off_list;
  a.off_part = sh.off_part;
  a.off_row = sh.off_row;
  a.off_coarse = sh.off_coarse;
  a.off_op = sh.off_op;
  if (COARSE) {
    a.nc = h->cnc;
    a.cmaxrows = cmaxrows;
    a.cmaxagg = pl.cmaxagg;
    a.centries = pl.centries;
    a.cblk_ptr = d.pc_blk_ptr;
    a.cblk_pos = d.pc_blk_pos;
    a.cblk_agg = d.pc_blk_agg;
    a.cagg_ptr = d.pc_agg_ptr;
    a.crow = d.pc_row;
    a.coff = d.coff;
    a.cfixed = h->last_bc == LPM_BC_ELIMINATE ? d.fixed : nullptr;
    a.cAinv = d.cAinv;
    a.crec = d.pc_rec;
    LPM_CUDA(h, cudaMemsetAsync(d.pc_rec, 0, 16 * 2 * ((size_t)pl.centries * kModes<DIM> + 2 * (size_t)h->cnc),
                                h->stream));
  }
  // the records' tags, which start at 1
  LPM_CUDA(h, cudaMemsetAsync(d.pl_words, 0, kWordBytes, h->stream));
  LPM_CUDA(h, cudaMemsetAsync(d.pl_zp, 0, kZBytes * (size_t)h->n, h->stream));
  void* args[] = {&a};
  LPM_CUDA(h, cudaLaunchCooperativeKernel((const void*)fn, dim3(pl.G), dim3(sh.threads), args, sh.bytes, h->stream));
  LPM_LAUNCHED(h, "k_pcg_mixed");
  return 1;
}

// Most slices of a block in the mixed solve: one to a compute warp.
int mixed_slices(const lpm_handle* h) { return (h->dim == 3 ? kPcgWideThreads<3> : kPcgWideThreads<2>) / 32 - 1; }

}  // namespace

// The aggregates each block's rows touch (coarse_setup, when the plan is
// usable): entries (block, aggregate) in two orders, by block and by
// aggregate, and each row's aggregate among its block's.
int pcg_coarse_plan(lpm_handle* h, const std::vector<int>& agg, int nagg) {
  const int st = pcg_plan(h, mixed_slices(h));
  if (st <= 0) return st < 0 ? st : LPM_OK;
  Dev& d = h->d;
  PcgPlan& pl = h->pcg;
  pl.mixed_coarse = PcgShape{};
  std::vector<int> ptr(1, 0), blk_agg, seen((size_t)nagg, -1);
  std::vector<unsigned> row((size_t)h->n);
  pl.cmaxagg = 0;
  for (int b = 0; b < pl.G; ++b) {
    const int i0 = plan_slice(b, pl.G, h->nslice) * kSlice;
    const int i1 = std::min(h->n, plan_slice(b + 1, pl.G, h->nslice) * kSlice);
    const int at = (int)blk_agg.size();
    for (int i = i0; i < i1; ++i) {
      const int ag = agg[(size_t)i];
      if (seen[(size_t)ag] < at) {
        seen[(size_t)ag] = (int)blk_agg.size();
        blk_agg.push_back(ag);
      }
      row[(size_t)i] = (unsigned)(seen[(size_t)ag] - at);
    }
    ptr.push_back((int)blk_agg.size());
    pl.cmaxagg = std::max(pl.cmaxagg, (int)blk_agg.size() - at);
  }
  pl.centries = (int)blk_agg.size();
  std::vector<int> agg_ptr((size_t)nagg + 1, 0), pos(blk_agg.size());
  for (int ag : blk_agg) agg_ptr[(size_t)ag + 1]++;
  for (int a = 0; a < nagg; ++a) agg_ptr[(size_t)a + 1] += agg_ptr[(size_t)a];
  std::vector<int> fill(agg_ptr.begin(), agg_ptr.end() - 1);
  for (size_t e = 0; e < blk_agg.size(); ++e) pos[e] = fill[(size_t)blk_agg[e]]++;
  const int nm = h->dim == 3 ? kModes<3> : kModes<2>;
  auto up = [&](auto** dst, const auto& v) {
    using V = std::remove_reference_t<decltype(**dst)>;
    *dst = (V*)dev_alloc(h, sizeof(V) * std::max<size_t>(v.size(), 1));
    return *dst && (v.empty() || cudaMemcpyAsync(*dst, v.data(), sizeof(V) * v.size(), cudaMemcpyHostToDevice,
                                                 h->stream) == cudaSuccess);
  };
  d.pc_rec = (float*)dev_alloc(h, 16 * 2 * ((size_t)pl.centries * nm + 2 * (size_t)nagg * nm));
  if (!d.pc_rec || !up(&d.pc_blk_ptr, ptr) || !up(&d.pc_blk_pos, pos) || !up(&d.pc_blk_agg, blk_agg) ||
      !up(&d.pc_agg_ptr, agg_ptr) || !up(&d.pc_row, row)) {
    pl.mixed_coarse.state = -1;
    pcg_no_memory(h);
  }
  LPM_CUDA(h, cudaStreamSynchronize(h->stream));  // the host arrays go out of scope
  return LPM_OK;
}

int pcg_run_mixed(lpm_handle* h, bool keep, bool coarse) {
  const int st = pcg_plan(h, mixed_slices(h));
  if (st <= 0) return st;
  if (coarse) return h->dim == 3 ? run_mixed_dim<3, true>(h, keep) : run_mixed_dim<2, true>(h, keep);
  return h->dim == 3 ? run_mixed_dim<3, false>(h, keep) : run_mixed_dim<2, false>(h, keep);
}

}  // namespace lpm
