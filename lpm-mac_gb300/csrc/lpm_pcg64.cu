// The FP64 CG solve of systems with at most one row per resident thread, as
// one cooperative kernel whose working set stays on the SMs: the recurrence
// of k_cg_spmv, k_cg_update and k_cg_pupdate (lpm_cg.cu; Eigen's), on the
// layout of the mixed solve (lpm_pcg.cu) - operator groups in shared memory,
// the direction staged there once per iteration, the sums and z as tagged
// records through block 0, a warp of its own for them.
//
// A small system is bound by latency, and more of it than in the mixed solve:
// an FP64 addition or FMA takes 65 cycles here and a division 420, so a
// shuffle tree over a warp is 470.  A large one is bound by the FP64 pipe, one
// per scheduler, which takes a warp's instruction in 64 cycles: the work has
// to be even over the four schedulers of an SM, which whole slices per warp
// are not (17 warps leave one scheduler with five).  So the groups of four
// blocks are split over the warps regardless of the slices.
//
// Measured on GB300, us per iteration, here against k_cg_persistent: plates
// of 1,661 rows 8.8 (16.2) and 40,301 rows 20.7 (26.8), simple cubes of 21^3
// 20 (45) and 31^3 45 (67).  With more than twelve slices to a block it is
// even or behind - 80,401 rows in 2-D 34.2 (34.9), in 3-D 102 (98): every
// block forms p at all its columns, and what p and the partial sums take of
// the shared memory leaves the operator to HBM - and k_cg_persistent stays.
#include <algorithm>
#include <cmath>

#include "lpm_device.cuh"
#include "lpm_pcg.cuh"

namespace lpm {
namespace {

struct State64 {
  double rz, rr, threshold, alpha, beta;
  long long it, maxit, passes;
  int done, fail;
};
struct Shared64 {
  State64 st;
  double red[2][kPcgMaxSlices];
  int64_t slot[kPcgMaxSlices];    // first slot of each slice
  int gbase[kPcgMaxSlices + 1];   // groups of four before each slice
};
extern __shared__ __align__(16) unsigned char dyn64[];
__device__ __forceinline__ Shared64& state64() { return *reinterpret_cast<Shared64*>(dyn64); }

__device__ __forceinline__ unsigned lo32(double v) { return (unsigned)__double_as_longlong(v); }
__device__ __forceinline__ unsigned hi32(double v) { return (unsigned)((unsigned long long)__double_as_longlong(v) >> 32); }
__device__ __forceinline__ double pair64(unsigned lo, unsigned hi) {
  return __longlong_as_double((long long)(((unsigned long long)hi << 32) | lo));
}

// z of a row as two records, each with its tag.
template <int DIM>
__device__ __forceinline__ void publish_z64(const PcgFp64Args& a, unsigned zn, int row, const double (&z)[DIM]) {
  Rec* q = reinterpret_cast<Rec*>(a.zp) + ((size_t)(zn & 1) * a.n + row) * 2;
  const double z2 = DIM == 3 ? z[DIM - 1] : 0.0;
  st_rec(q, lo32(z[0]), hi32(z[0]), lo32(z[1]), zn);
  st_rec(q + 1, hi32(z[1]), lo32(z2), hi32(z2), zn);
}
template <int DIM>
__device__ __forceinline__ bool load_z64(const Rec* q, unsigned zn, double (&z)[DIM]) {
  const Rec r = ld_rec(q), s = ld_rec(q + 1);
  z[0] = pair64(r.x, r.y);
  z[1] = pair64(r.z, s.x);
  if (DIM == 3) z[DIM - 1] = pair64(s.y, s.z);
  return r.w == zn && s.w == zn;
}

// One block of a row (element e from at(e)) times the staged p.
template <int DIM, typename F>
__device__ __forceinline__ void block_fma(F at, const double* p, double (&y)[DIM]) {
  double pc[DIM];
  if constexpr (DIM == 2) {
    const double2 v = *reinterpret_cast<const double2*>(p);
    pc[0] = v.x;
    pc[1] = v.y;
  } else {
#pragma unroll
    for (int k = 0; k < DIM; ++k) pc[k] = p[k];
  }
#pragma unroll
  for (int k = 0; k < DIM; ++k)
#pragma unroll
    for (int r = 0; r < DIM; ++r) y[r] = fma(at(r * DIM + k), pc[k], y[r]);
}

// Row r of a group's four blocks: for each column k the four blocks' elements,
// 32 bytes of a lane, and the columns' positions.
template <int DIM>
struct Chunk {
  double2 lo[DIM], hi[DIM];
  ushort4 l;
};
// s: the lane's first slot of the group.
template <int DIM, bool KEEP>
__device__ __forceinline__ void load_chunk(const PcgFp64Args& a, int64_t s, int r, Chunk<DIM>& c) {
  // (worked out afresh: kept in registers through the solve, the planes'
  // addresses would push others out to memory)
  int64_t ns = a.nslots;
  asm volatile("" : "+l"(ns));
  c.l = __ldg(reinterpret_cast<const ushort4*>(a.lidx + s));
  const double* at = a.A + s + r * DIM * ns;
#pragma unroll
  for (int k = 0; k < DIM; ++k, at += ns) {
    const double2* q = reinterpret_cast<const double2*>(at);
    c.lo[k] = KEEP ? __ldg(q) : __ldcs(q);
    c.hi[k] = KEEP ? __ldg(q + 1) : __ldcs(q + 1);
  }
}
template <int DIM>
__device__ __forceinline__ double chunk_fma(const Chunk<DIM>& c, const double* ps, double y) {
#pragma unroll
  for (int q = 0; q < kVec; ++q) {
    const double* p = ps + comp_u16(c.l, q) * DIM;
#pragma unroll
    for (int k = 0; k < DIM; ++k)
      y = fma(q == 0 ? c.lo[k].x : q == 1 ? c.lo[k].y : q == 2 ? c.hi[k].x : c.hi[k].y, p[k], y);
  }
  return y;
}

// Sum of the block's S values (lane s has slice s's), in every lane.
__device__ __forceinline__ double fold_slices(double v, int width) {
  for (int o = width >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// Sum of the blocks' values: `at` gives record q's.
template <typename F>
__device__ __forceinline__ double fold_blocks(F at) {
  static_assert(kPcgMaxBlocks == 160, "five records a lane");
  const int lane = threadIdx.x & 31, G = gridDim.x;
  double v[5];
#pragma unroll
  for (int q = 0; q < 5; ++q) v[q] = lane + 32 * q < G ? at(q) : 0.0;
  double s = v[0];
  if (G > 32) s = ((v[0] + v[1]) + (v[2] + v[3])) + v[4];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// The message warp's part of an iteration's first sum: p.q to block 0, alpha
// back.
__device__ __forceinline__ void alpha64(Rec* words, Shared64& sh, unsigned m, unsigned epoch, int S, int width) {
  State64& st = sh.st;
  const int lane = threadIdx.x & 31;
  const double s = fold_slices(lane < S ? sh.red[0][lane] : 0.0, width);
  Rec* set = arrivals(words, kArrAlpha, m & 1);
  if (lane == 0) st_rec(set + blockIdx.x, lo32(s), hi32(s), 0u, m + 1);
  if (blockIdx.x == 0) {
    Rec r[kPcgMaxBlocks / 32];
    if (!gather_records(set, gridDim.x, r, [&](const Rec& q) { return q.w == m + 1; })) {
      st.fail = 1;
      return;
    }
    const double alpha = st.rz / fold_blocks([&](int q) { return pair64(r[q].x, r[q].y); });
    if (lane < kReplyCopies) st_rec(reply(words, epoch, lane), lo32(alpha), hi32(alpha), epoch, 0u);
    if (lane == 0) st.alpha = alpha;
  } else if (lane == 0) {
    Rec r;
    if (!poll_record(reply(words, epoch, blockIdx.x % kReplyCopies), r, [&](const Rec& q) { return q.z == epoch; }))
      st.fail = 1;
    st.alpha = pair64(r.x, r.y);
  }
}

// The second sum: |r|^2 (its sign bit the arrival's tag, as in the mixed
// solve) and r.z to block 0, which decides: beta back, or the end.
__device__ __forceinline__ void beta64(Rec* words, Shared64& sh, unsigned m, unsigned epoch, int S, int width) {
  State64& st = sh.st;
  const int lane = threadIdx.x & 31;
  const double s0 = fold_slices(lane < S ? sh.red[0][lane] : 0.0, width);
  const double s1 = fold_slices(lane < S ? sh.red[1][lane] : 0.0, width);
  Rec* set = arrivals(words, kArrBeta, m & 1);
  const unsigned tag = ((m >> 1) & 1u) ^ 1u;
  if (lane == 0)
    st_rec(set + blockIdx.x, lo32(s1), hi32(s1), lo32(s0), (hi32(s0) & 0x7fffffffu) | (tag << 31));
  if (blockIdx.x == 0) {
    Rec r[kPcgMaxBlocks / 32];
    if (!gather_records(set, gridDim.x, r, [&](const Rec& q) { return (q.w >> 31) == tag; })) {
      st.fail = 1;
      return;
    }
    const double rr = fold_blocks([&](int q) { return pair64(r[q].z, r[q].w & 0x7fffffffu); });
    const double rz = fold_blocks([&](int q) { return pair64(r[q].x, r[q].y); });
    // every lane decides alike; lane 0 keeps the state
    int done = 0;
    double beta = st.beta;
    long long it = st.it;
    if (!isfinite(rr) || !isfinite(rz)) {
      done = 3;
    } else if (rr < st.threshold) {
      done = 1;
    } else {
      beta = rz / st.rz;
      if (++it >= st.maxit) done = 2;
    }
    if (lane < kReplyCopies) st_rec(reply(words, epoch, lane), lo32(beta), hi32(beta), epoch, (unsigned)(done != 0));
    __syncwarp();
    if (lane == 0) {
      st.rr = rr;
      st.it = it;
      st.done = done;
      st.beta = beta;
      if (done == 0) st.passes += 1;
      if (done == 0 || done == 2) st.rz = rz;
    }
  } else if (lane == 0) {
    Rec r;
    if (!poll_record(reply(words, epoch, blockIdx.x % kReplyCopies), r, [&](const Rec& q) { return q.z == epoch; }))
      st.fail = 1;
    st.beta = pair64(r.x, r.y);
    st.done = (int)r.w;
  }
}

// The message warp's loop.
__device__ __noinline__ void messages64(Rec* words, CgScalars* cg, int S) {
  Shared64& sh = state64();
  State64& st = sh.st;
  const int lane = threadIdx.x & 31;
  int width = 1;
  while (width < S) width *= 2;
  unsigned epoch = 0;
#pragma unroll 1
  for (unsigned m = 0;; ++m) {
    __syncthreads();
    alpha64(words, sh, m, ++epoch, S, width);
    __syncthreads();
    if (st.fail) break;
    __syncthreads();
    beta64(words, sh, m, ++epoch, S, width);
    __syncthreads();
    if (st.fail || st.done) break;
  }
  if (lane == 0 && st.fail) atomicExch(&cg->pfault, 1);
  if (blockIdx.x == 0 && lane == 0 && !st.fail) {
    cg->done = st.done;
    cg->rr = st.rr;
    cg->it = st.it;
    cg->abs_new = st.rz;
    cg->alpha = st.alpha;
    cg->beta = st.beta;
    cg->graph_passes = st.passes;
  }
}

// Block b's slices take W compute warps and the message warp.  Warp w < S owns
// the rows of the block's slice w (r, x, z, the tail blocks of the product);
// the groups of four of all its slices, one after the other, are split evenly
// over the W warps, each keeping the first of its own in shared memory.  Warp
// w's part of slice s goes through place w + s of the partial sums (along the
// split one of the two grows from each part to the next).
template <int DIM, bool KEEP>
__global__ void __launch_bounds__(kPcg64Threads, 1) k_pcg_fp64(const __grid_constant__ PcgFp64Args a) {
  constexpr int E = DIM * DIM;
  constexpr int kAhead = 4;  // columns of a thread fetched ahead
  constexpr int NB = DIM == 2 ? 2 : 1;  // chunks in flight
  constexpr int kBlk = kPcgUnit64<DIM> / kVec;
  Shared64& sh = state64();
  State64& st = sh.st;
  const int s0 = plan_slice(blockIdx.x, gridDim.x, a.nslice);
  const int S = plan_slice(blockIdx.x + 1, gridDim.x, a.nslice) - s0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = a.W;
  const int U = a.ucnt[blockIdx.x];
  const int nth = W * 32;  // compute threads
  double* ps = reinterpret_cast<double*>(dyn64 + a.off_p);
  int* ul = reinterpret_cast<int*>(dyn64 + a.off_list);
  double* part = reinterpret_cast<double*>(dyn64 + a.off_part) + lane;
  double* rowc = reinterpret_cast<double*>(dyn64 + a.off_row) + threadIdx.x;  // [DIM][rows]: the diagonal
  const int rstride = a.maxS * kSlice;
  const int row = s0 * kSlice + (int)threadIdx.x;
  const bool mine = warp < S, owner = mine && row < a.n;
  const unsigned own = owner ? (unsigned)(a.uown[blockIdx.x] + (int)threadIdx.x) : 0u;
  if (threadIdx.x == 0) {
    sh.gbase[0] = 0;
    for (int k = 0; k < S; ++k) {
      const int64_t b = a.sell_ptr[s0 + k];
      sh.slot[k] = b;
      sh.gbase[k + 1] = sh.gbase[k] + (int)((a.sell_ptr[s0 + k + 1] - b) / (kSlice * kVec));
    }
    const CgScalars* c = a.cg;
    st.rz = c->abs_new;
    st.threshold = c->threshold;
    st.alpha = c->alpha;
    st.beta = 0.0;
    st.rr = c->rr;
    st.it = c->it;
    st.maxit = c->maxit;
    st.passes = 0;
    st.done = c->done;
    st.fail = 0;
  }
  for (int u = threadIdx.x; u < U; u += blockDim.x) {
    ul[u] = a.ulist[(int64_t)blockIdx.x * a.umax + u];
#pragma unroll
    for (int k = 0; k < DIM; ++k) ps[u * DIM + k] = 0.0;
  }
  __syncthreads();
  if (st.done) return;  // the same in every block
  if (warp == W) {
    messages64(reinterpret_cast<Rec*>(a.words), a.cg, S);
    return;
  }
  // this warp's groups, those kept on chip up to gr; the slice of the first
  // and the slot of the first streamed one
  const int G = sh.gbase[S], g0 = warp * G / W, g1 = (warp + 1) * G / W;
  const int gr = min(g1, g0 + a.R + (warp < a.gx ? 1 : 0));
  int sfirst = 0;
  while (sfirst + 1 < S && sh.gbase[sfirst + 1] <= g0) ++sfirst;
  auto slot_of = [&](int s, int g) { return sh.slot[s] + (int64_t)(g - sh.gbase[s]) * (kSlice * kVec) + lane * kVec; };
  unsigned char* unit = dyn64 + a.off_op + (size_t)(warp * a.R + min(warp, a.gx)) * kPcgUnit64<DIM>;
  int64_t streamed = 0;
  {
    int s = sfirst;
    for (int g = g0; g < g1 && g <= gr; ++g) {
      while (g >= sh.gbase[s + 1]) ++s;
      if (g == gr) {
        streamed = slot_of(s, g);
        break;
      }
      // block by block: the E elements, then the position of each of the 32 rows
#pragma unroll 1
      for (int e = 0; e < DIM; ++e) {
        Chunk<DIM> c;
        load_chunk<DIM, KEEP>(a, slot_of(s, g), e, c);
#pragma unroll
        for (int q = 0; q < kVec; ++q) {
          double* b = reinterpret_cast<double*>(unit + (size_t)(g - g0) * kPcgUnit64<DIM> + q * kBlk);
#pragma unroll
          for (int j = 0; j < DIM; ++j)
            b[(e * DIM + j) * 32 + lane] = q == 0 ? c.lo[j].x : q == 1 ? c.lo[j].y : q == 2 ? c.hi[j].x : c.hi[j].y;
          reinterpret_cast<unsigned short*>(b + E * 32)[lane] = (unsigned short)comp_u16(c.l, q);
        }
      }
    }
  }
  // the tail blocks of the warp's slice (slot of the first)
  int tail = 0;
  int64_t tslot = 0;
  unsigned char* tunit = dyn64 + a.off_tail + (size_t)(mine ? warp : 0) * a.tails * kBlk;
  if (mine) {
    const int groups = sh.gbase[warp + 1] - sh.gbase[warp];
    tslot = sh.slot[warp] + (int64_t)groups * (kSlice * kVec) + lane;
    tail = (int)((a.sell_ptr[s0 + warp + 1] - sh.slot[warp]) / kSlice) - groups * kVec;
    if (a.tails)
      for (int k = 0; k < tail; ++k) {
        double* b = reinterpret_cast<double*>(tunit + k * kBlk);
        for (int e = 0; e < E; ++e) b[e * 32 + lane] = a.A[e * a.nslots + tslot + k * kSlice];
        reinterpret_cast<unsigned short*>(b + E * 32)[lane] = a.lidx[tslot + k * kSlice];
      }
  }
  // the warps with a part of this warp's slice (one with no group has none)
  unsigned parts = 0;
  if (mine && sh.gbase[warp + 1] > sh.gbase[warp])
    for (int w = ((sh.gbase[warp] + 1) * W - 1) / G; w <= (sh.gbase[warp + 1] * W - 1) / G; ++w)
      if (w * G / W < (w + 1) * G / W) parts |= 1u << w;
  const int64_t i0 = (int64_t)row * DIM;
  double r[DIM];
#pragma unroll
  for (int k = 0; k < DIM; ++k) r[k] = owner ? a.r[i0 + k] : 0.0;
  unsigned zn = 1;
  if (owner) {
    double z[DIM];
#pragma unroll
    for (int k = 0; k < DIM; ++k) {
      const double iv = a.invd[i0 + k];
      rowc[k * rstride] = iv;
      z[k] = iv * r[k];
    }
    publish_z64<DIM>(a, zn, row, z);
  }
  compute_sync(nth);
  // the first kAhead of this thread's columns, asked for once while the sums
  // travel and then, where a record had not come, when they are back
  double zq[kAhead][DIM];
  unsigned need = 0;
  auto zbase = [&]() { return reinterpret_cast<const Rec*>(a.zp) + (size_t)(zn & 1) * a.n * 2; };
  auto ask = [&]() {
    const Rec* zb = zbase();
#pragma unroll
    for (int q = 0; q < kAhead; ++q)
      if (need >> q & 1u)
        if (load_z64<DIM>(zb + 2 * (size_t)ul[threadIdx.x + q * nth], zn, zq[q])) need &= ~(1u << q);
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
    // p = z + beta p at the block's columns
    {
      for (long long polls = 0; need; ++polls) {
        ask();
        if (polls > kPollLimit) {
          st.fail = 1;
          break;
        }
      }
      const double beta = st.beta;
#pragma unroll
      for (int q = 0; q < kAhead; ++q) {
        const int u = threadIdx.x + q * nth;
        if (u < U)
#pragma unroll
          for (int k = 0; k < DIM; ++k) ps[u * DIM + k] = fma(beta, ps[u * DIM + k], zq[q][k]);
      }
      const Rec* zb = zbase();
#pragma unroll 1
      for (int u = threadIdx.x + kAhead * nth; u < U; u += nth) {
        double z[DIM];
        long long polls = 0;
        while (!load_z64<DIM>(zb + 2 * (size_t)ul[u], zn, z))
          if (++polls > kPollLimit) {
            st.fail = 1;
            break;
          }
#pragma unroll
        for (int k = 0; k < DIM; ++k) ps[u * DIM + k] = fma(beta, ps[u * DIM + k], z[k]);
      }
    }
    compute_sync(nth);
    // q = A p: this warp's groups
    {
      double y[DIM];
#pragma unroll
      for (int k = 0; k < DIM; ++k) y[k] = 0.0;
      int s = sfirst, gend = sh.gbase[s + 1], g = g0;
      int64_t slot = streamed;
      // the first streamed chunk is on its way while the resident groups are
      // multiplied; after that one is loaded while the other warps of the
      // scheduler multiply theirs
      Chunk<DIM> c[NB];
      if (gr < g1)
#pragma unroll
        for (int i = 0; i < NB; ++i) load_chunk<DIM, KEEP>(a, slot, i, c[i]);
      auto next_slice = [&]() {
#pragma unroll
        for (int k = 0; k < DIM; ++k) {
          part[((warp + s) * DIM + k) * 32] = y[k];
          y[k] = 0.0;
        }
        while (g >= sh.gbase[s + 1]) ++s;
        gend = sh.gbase[s + 1];
      };
#pragma unroll 1
      for (; g < gr; ++g) {
        if (g == gend) next_slice();
#pragma unroll
        for (int q = 0; q < kVec; ++q) {
          const double* b = reinterpret_cast<const double*>(unit + (size_t)(g - g0) * kPcgUnit64<DIM> + q * kBlk);
          const unsigned l = reinterpret_cast<const unsigned short*>(b + E * 32)[lane];
          block_fma<DIM>([&](int e) { return b[e * 32 + lane]; }, ps + l * DIM, y);
        }
      }
#pragma unroll 1
      for (; g < g1; ++g) {
        if (g == gend) next_slice();
        const int64_t here = slot;
        if (g + 1 < g1) {
          slot += kSlice * kVec;
          if (g + 1 == gend) {
            int sn = s + 1;
            while (g + 1 >= sh.gbase[sn + 1]) ++sn;
            slot = sh.slot[sn] + lane * kVec;
          }
        }
#pragma unroll
        for (int r = 0; r < DIM; ++r) {
          y[r] = chunk_fma<DIM>(c[r % NB], ps, y[r]);
          if (r + NB < DIM)
            load_chunk<DIM, KEEP>(a, here, r + NB, c[r % NB]);
          else if (g + 1 < g1)
            load_chunk<DIM, KEEP>(a, slot, (r + NB) % DIM, c[r % NB]);
        }
      }
      if (g0 < g1)
#pragma unroll
        for (int k = 0; k < DIM; ++k) part[((warp + s) * DIM + k) * 32] = y[k];
    }
    double y[DIM];
#pragma unroll
    for (int k = 0; k < DIM; ++k) y[k] = 0.0;
#pragma unroll 1
    for (int k = 0; k < tail; ++k) {
      if (a.tails) {
        const double* b = reinterpret_cast<const double*>(tunit + k * kBlk);
        const unsigned l = reinterpret_cast<const unsigned short*>(b + E * 32)[lane];
        block_fma<DIM>([&](int e) { return b[e * 32 + lane]; }, ps + l * DIM, y);
      } else {
        const double* b = a.A + tslot + k * kSlice;
        block_fma<DIM>([&](int e) { return b[e * a.nslots]; }, ps + a.lidx[tslot + k * kSlice] * DIM, y);
      }
    }
    compute_sync(nth);
#pragma unroll 1
    for (unsigned m = parts; m; m &= m - 1) {
      const double* v = part + (__ffs((int)m) - 1 + warp) * DIM * 32;
#pragma unroll
      for (int k = 0; k < DIM; ++k) y[k] += v[k * 32];
    }
    // p.q
    if (mine) {
      double v[1] = {0.0};
      if (owner)
#pragma unroll
        for (int k = 0; k < DIM; ++k) v[0] = fma(ps[own * DIM + k], y[k], v[0]);
      warp_sum<1>(v);
      if (lane == 0) sh.red[0][warp] = v[0];
    }
    __syncthreads();  // p.q
    __syncthreads();
    if (st.fail) break;
    // r -= alpha q, z = M r published, |r|^2 and r.z
    ++zn;
    if (mine) {
      const double alpha = st.alpha;
      double v[2] = {0.0, 0.0};
      if (owner) {
        double z[DIM];
#pragma unroll
        for (int k = 0; k < DIM; ++k) {
          r[k] = fma(-alpha, y[k], r[k]);
          z[k] = rowc[k * rstride] * r[k];
        }
        publish_z64<DIM>(a, zn, row, z);
#pragma unroll
        for (int k = 0; k < DIM; ++k) {
          v[0] = fma(r[k], r[k], v[0]);
          v[1] = fma(r[k], z[k], v[1]);
        }
      }
      warp_sum<2>(v);
      if (lane == 0) {
        sh.red[0][warp] = v[0];
        sh.red[1][warp] = v[1];
      }
    }
    __syncthreads();  // |r|^2, r.z
    // while the sums travel: x += alpha p, and the z of the block's columns
    if (owner) {
      const double alpha = st.alpha;
#pragma unroll
      for (int k = 0; k < DIM; ++k) a.x[i0 + k] = fma(alpha, ps[own * DIM + k], a.x[i0 + k]);
    }
    ask_first();
    __syncthreads();
    if (st.fail || st.done) break;
  }
  // (nothing after the solve reads r but a caller of the residual)
  if (owner)
#pragma unroll
    for (int k = 0; k < DIM; ++k) a.r[i0 + k] = r[k];
}

// Most columns a row (of the largest block) in 2-D with more than nine slices:
// where the numbering scatters a row's neighbours every block forms p at nearly
// all the columns its rows name, and k_cg_persistent, which forms p once, is
// ahead.  us per iteration of plates numbered at random (28 columns a row),
// here against there: 44k rows, ten slices, 34.1 (31.7), 45.9k 34.4 (31.6), 50.3k,
// eleven, 37.8 (32.8), 52k 38.0 (32.3); within windows of 16,384 particles (24 to 27
// columns) the two are even, 45.9k 31.7 (31.6), or this is ahead, 57.8k 31.9
// (34.8).  Up to nine slices either may be ahead: 23.7k rows 23.0 (24.5), 33.9k
// 28.8 (29.1 to 29.7), 39.8k 29.3 or 32.1 (30.7).  In 3-D, nine elements to a block,
// what fits is ahead: 26^3 at random, 47 columns a row, 37.4 (69.4).
constexpr int kColumnsPerRow = 26, kColumnsSlices = 9;

// Launch shape with W compute warps in smem bytes: the staged vector, its
// columns, the partial sums, the diagonal, the slices' tail blocks and as many
// groups of each warp as fit.  `share`: only if all of them do, in blocks of which
// an SM holds two.
template <int DIM>
bool shape64_with(const lpm_handle* h, const void* fn, int W, int smem, bool share, PcgShape* sh) {
  const PcgPlan& pl = h->pcg;
  auto align = [](size_t b) { return (int)((b + 15) / 16 * 16); };
  int tails = 0, most = 0;  // most tail blocks of a slice, most groups of a block
  for (int b = 0; b < pl.G; ++b) {
    int g = 0;
    for (int s = plan_slice(b, pl.G, h->nslice); s < plan_slice(b + 1, pl.G, h->nslice); ++s) {
      const int w = (int)((h->sell_host[(size_t)s + 1] - h->sell_host[(size_t)s]) / kSlice);
      g += w / kVec;
      tails = std::max(tails, w % kVec);
    }
    most = std::max(most, g);
  }
  sh->T = W;
  sh->off_p = align(sizeof(Shared64));
  sh->off_list = sh->off_p + align(sizeof(double) * DIM * (size_t)pl.umax);
  sh->off_part = sh->off_list + align(sizeof(int) * (size_t)pl.umax);
  sh->off_row = sh->off_part + align(sizeof(double) * DIM * 32 * (size_t)(W + pl.S));
  sh->off_coarse = sh->off_row + align(sizeof(double) * DIM * 32 * (size_t)pl.S);  // the tail blocks
  const int tbytes = align((size_t)kPcgUnit64<DIM> / kVec * tails * (size_t)pl.S);
  if (sh->off_coarse > smem) return false;
  sh->tails = sh->off_coarse + tbytes <= smem ? tails : 0;
  sh->off_op = sh->off_coarse + (sh->tails ? tbytes : 0);
  const int units = (smem - sh->off_op) / kPcgUnit64<DIM>, need = (most + W - 1) / W;
  sh->gs = std::min(units / W, need);
  sh->gx = sh->gs < need ? units - sh->gs * W : 0;
  if (share && (sh->gs < need || sh->tails < tails)) return false;
  sh->bytes = (size_t)sh->off_op + (size_t)(sh->gs * W + sh->gx) * kPcgUnit64<DIM>;
  sh->threads = (W + 1) * 32;
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

// Once per handle.  Blocks of one slice take four warps and those of two seven,
// and half an SM, where their groups fit it, so that the solves of several small
// systems, from several threads, run beside each other.  us per iteration alone,
// with eight warps and so: a 41x41 plate 11.1 and 11.3, 61x80 11.0 and 11.0, 61x121
// 12.7 and 12.5, 75x110 11.7 and 12.3; of four handles solved at once (over all
// their iterations) a 41x41 plate 5.2 and 3.0, 61x121 12.4 and 6.0.  (With
// k_cg_persistent 5.4 and 7.1.)
template <int DIM>
bool shape64(const lpm_handle* h, const void* fn, PcgShape* sh) {
  const PcgPlan& pl = h->pcg;
  if (DIM == 2 && pl.S > kColumnsSlices && pl.umax > kColumnsPerRow * kSlice * pl.S) return false;
  return (pl.S <= kSharingSlices && shape64_with<DIM>(h, fn, pl.S == 1 ? 4 : 7, pl.half, true, sh)) ||
         shape64_with<DIM>(h, fn, fp64_warps(DIM, pl.S), pl.smem, false, sh);
}

template <int DIM>
int run_fp64_dim(lpm_handle* h, const double* A, double* x, double* r, const double* invd, bool keep) {
  Dev& d = h->d;
  PcgPlan& pl = h->pcg;
  using Fn = void (*)(PcgFp64Args);
  const Fn fn = keep ? k_pcg_fp64<DIM, true> : k_pcg_fp64<DIM, false>;
  PcgShape& sh = pl.fp64;
  if (!sh.state) sh.state = shape64<DIM>(h, (const void*)fn, &sh) ? 1 : -1;
  if (sh.state < 0) return 0;
  PcgFp64Args a{};
  a.sell_ptr = d.sell_ptr;
  a.ucnt = d.pl_ucnt;
  a.uown = d.pl_uown;
  a.ulist = d.pl_ulist;
  a.lidx = d.pl_lidx;
  a.A = A;
  a.invd = invd;
  a.x = x;
  a.r = r;
  a.zp = d.pl_zp;
  a.words = d.pl_words;
  a.cg = d.cg;
  a.nslots = h->nslots;
  a.n = h->n;
  a.nslice = h->nslice;
  a.umax = pl.umax;
  a.maxS = pl.S;
  a.W = sh.T;
  a.R = sh.gs;
  a.gx = sh.gx;
  a.tails = sh.tails;
  a.off_p = sh.off_p;
  a.off_list = sh.off_list;
  a.off_part = sh.off_part;
  a.off_row = sh.off_row;
  a.off_tail = sh.off_coarse;
  a.off_op = sh.off_op;
  // the records' tags, which start at 1
  LPM_CUDA(h, cudaMemsetAsync(d.pl_words, 0, kWordBytes, h->stream));
  LPM_CUDA(h, cudaMemsetAsync(d.pl_zp, 0, kZBytes64 * (size_t)h->n, h->stream));
  void* args[] = {&a};
  LPM_CUDA(h, cudaLaunchCooperativeKernel((const void*)fn, dim3(pl.G), dim3(sh.threads), args, sh.bytes, h->stream));
  LPM_LAUNCHED(h, "k_pcg_fp64");
  return 1;
}

}  // namespace

int pcg_run_fp64(lpm_handle* h, const double* A, double* x, double* r, const double* invd, bool keep) {
  const int st = pcg_plan(h, kPcg64Slices);
  if (st <= 0) return st;
  return h->dim == 3 ? run_fp64_dim<3>(h, A, x, r, invd, keep) : run_fp64_dim<2>(h, A, x, r, invd, keep);
}

}  // namespace lpm
