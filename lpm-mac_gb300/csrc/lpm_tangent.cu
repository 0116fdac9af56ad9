// Sparsity pattern (Particle::conns) and the analytical tangent.
//
// Pattern (assembly.h:236-266): conns(i) = sorted unique {k, m : k a layer-l
// bond partner of i, m a layer-l bond partner of k}.  Built on the device in
// three passes (count candidates, fill + sort + unique per particle,
// compact); integer work, identical to the reference's lists.
//
// Tangent (stiffness.h:67-101, 228-263; derivative.h): block K_ij for every
// j in conns(i).  The stored operator is A = K^T (see lpm_internal.cuh); a
// lane owns a row j of A and computes blocks K_ij, i in conns(j), each by a
// merge of the two particles' bond lists.
#include <algorithm>
#include <climits>
#include <numeric>

#include "lpm_device.cuh"

namespace lpm {
namespace {

__device__ __forceinline__ void layer_range(const int64_t* bptr, const int64_t* lptr, int i, int l, int64_t& b,
                                            int64_t& e) {
  b = l == 0 ? bptr[i] : lptr[i];
  e = l == 0 ? lptr[i] : bptr[i + 1];
}

__global__ void k_count_candidates(int n, const int64_t* __restrict__ bptr, const int64_t* __restrict__ lptr,
                                   const int* __restrict__ bp2, const int* __restrict__ blayer,
                                   int64_t* __restrict__ cnt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int64_t c = 0;
  for (int64_t b = bptr[i]; b < bptr[i + 1]; ++b) {
    int64_t kb, ke;
    layer_range(bptr, lptr, bp2[b], blayer[b], kb, ke);
    c += 1 + (ke - kb);
  }
  cnt[i] = c;
}

// Candidates of particle i, sorted and unique in place; writes their count.
// Their order before the sort does not matter, so a warp collects them a
// bond's segment at a time into shared memory and sorts them there
// (bitonic).  A particle of more candidates than kWarpCand is left to
// k_fill_candidates_long, one thread's heapsort in global memory.  By one
// thread's insertion sort in global memory all particles took 4.6 ms of 51^3
// (198 candidates each), with the warps 0.47.
constexpr int kWarpCand = 1024, kCandWarps = 4;
__global__ void __launch_bounds__(32 * kCandWarps) k_fill_candidates(int n, const int64_t* __restrict__ bptr,
                                                                    const int64_t* __restrict__ lptr,
                                                                    const int* __restrict__ bp2,
                                                                    const int* __restrict__ blayer,
                                                                    const int64_t* __restrict__ cand_ptr,
                                                                    int* __restrict__ cand,
                                                                    int64_t* __restrict__ ucnt) {
  __shared__ int sm[kCandWarps][kWarpCand];
  const int lane = threadIdx.x & 31, i = blockIdx.x * kCandWarps + (threadIdx.x >> 5);
  if (i >= n) return;
  const int m = (int)min(cand_ptr[i + 1] - cand_ptr[i], (int64_t)INT_MAX);
  if (m > kWarpCand) return;
  int* c = sm[threadIdx.x >> 5];
  const int64_t b0 = bptr[i], b1 = bptr[i + 1];
  // 32 bonds at a time: each lane's segment, then its place among them
  int at = 0;
  for (int64_t g = b0; g < b1; g += 32) {
    int64_t kb = 0, ke = 0;
    int k = 0, len = 0;
    if (g + lane < b1) {
      k = bp2[g + lane];
      layer_range(bptr, lptr, k, blayer[g + lane], kb, ke);
      len = 1 + (int)(ke - kb);
    }
    int s = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += t;
    }
    int to = at + s - len;
    if (len) {
      c[to++] = k;
      for (int64_t b = kb; b < ke; ++b) c[to++] = bp2[b];
    }
    at += __shfl_sync(0xffffffffu, s, 31);
  }
  int M = 32;
  while (M < m) M *= 2;
  for (int a = m + lane; a < M; a += 32) c[a] = INT_MAX;
  __syncwarp();
  for (int k = 2; k <= M; k *= 2)
    for (int q = k / 2; q > 0; q /= 2) {
      for (int t = lane; t < M / 2; t += 32) {
        const int lo = 2 * q * (t / q) + t % q, hi = lo + q;
        const int a = c[lo], b = c[hi];
        if ((a > b) == ((lo & k) == 0)) {
          c[lo] = b;
          c[hi] = a;
        }
      }
      __syncwarp();
    }
  int* out = cand + cand_ptr[i];
  int u = 0;
  for (int a0 = 0; a0 < m; a0 += 32) {
    const int a = a0 + lane;
    const bool first = a < m && (a == 0 || c[a] != c[a - 1]);
    const unsigned mask = __ballot_sync(0xffffffffu, first);
    if (first) out[u + __popc(mask & ((1u << lane) - 1u))] = c[a];
    u += __popc(mask);
  }
  if (lane == 0) ucnt[i] = u;
}
__global__ void k_fill_candidates_long(int n, const int64_t* __restrict__ bptr, const int64_t* __restrict__ lptr,
                                       const int* __restrict__ bp2, const int64_t* __restrict__ cand_ptr,
                                       int* __restrict__ cand, int64_t* __restrict__ ucnt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || cand_ptr[i + 1] - cand_ptr[i] <= kWarpCand) return;
  int* c = cand + cand_ptr[i];
  int64_t m = 0;
  for (int l = 0; l < NL; ++l) {
    int64_t lb, le;
    layer_range(bptr, lptr, i, l, lb, le);
    for (int64_t b = lb; b < le; ++b) {
      const int k = bp2[b];
      c[m++] = k;
      int64_t kb, ke;
      layer_range(bptr, lptr, k, l, kb, ke);
      for (int64_t b2 = kb; b2 < ke; ++b2) c[m++] = bp2[b2];
    }
  }
  auto sift = [&](int64_t r, int64_t e) {
    const int v = c[r];
    for (int64_t q; (q = 2 * r + 1) < e; r = q) {
      if (q + 1 < e && c[q] < c[q + 1]) ++q;
      if (v >= c[q]) break;
      c[r] = c[q];
    }
    c[r] = v;
  };
  for (int64_t r = m / 2 - 1; r >= 0; --r) sift(r, m);
  for (int64_t e = m - 1; e > 0; --e) {
    const int v = c[0];
    c[0] = c[e];
    c[e] = v;
    sift(0, e);
  }
  int64_t u = 0;
  for (int64_t a = 0; a < m; ++a)
    if (u == 0 || c[a] != c[u - 1]) c[u++] = c[a];
  ucnt[i] = u;
}

__global__ void k_compact_pattern(int n, const int64_t* __restrict__ cand_ptr, const int* __restrict__ cand,
                                  const int64_t* __restrict__ cptr, int* __restrict__ cidx) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int* c = cand + cand_ptr[i];
  const int64_t q0 = cptr[i], len = cptr[i + 1] - q0;
  for (int64_t a = 0; a < len; ++a) cidx[q0 + a] = c[a];
}

// Sliced layout: slot columns, row lengths and the diagonal slot.
__global__ void k_fill_sell(int n, const int64_t* __restrict__ cptr, const int* __restrict__ cidx,
                            const int64_t* __restrict__ sell_ptr, int* __restrict__ scol, int* __restrict__ rowlen,
                            int* __restrict__ diag_slot) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const int64_t q0 = cptr[j];
  const int len = (int)(cptr[j + 1] - q0);
  const SellRow row = sell_row(sell_ptr, j);
  int ds = -1;
  for (int k = 0; k < len; ++k) {
    const int c = cidx[q0 + k];
    scol[sell_slot(row, k)] = c;
    if (c == j) ds = (int)sell_slot(row, k);
  }
  // padding of the row's last group of four points at the row itself
  for (int k = len; k < sell_read_len(row, len); ++k) scol[sell_slot(row, k)] = j;
  rowlen[j] = len;
  diag_slot[j] = ds;
}

constexpr int kAsmThreads = 512;  // most warps of a slice: 16 groups

struct AsmView {
  const int64_t *bptr, *lptr, *sell_ptr;
  const int *scol, *rowlen, *sbond, *sp2, *opp;
  const double *cs, *cs_sum, *tsum, *msum, *Kn, *Tv, *bdamage;
  const double2* rec;  // per sorted bond {n, w Tv / 2}, and the sorted place of its opposite (bond_records), or null
  const int* sopp;
  double* A;
  int64_t nslots;
  int n, nslice, sym;
};

// The analytical tangent (derivative.h) restated per block K_ij, i != j, as
// a sum over layers l of
//   own    (i->j a layer-l bond b):   w_b[(-Kn n_b[s] + Tv S_j[s]) n_b[r] - (Kn+Tv) n_b[r] n_b[s]]
//   other  (same b, derivative.h:91-99 summed over the other bonds of i):
//          -1/2 [w_b Tv_b (S_i - n_b) + (T_i - w_b Tv_b n_b)][r] n_b[s]
//   paths  (bonds i->k, k->j of layer l, derivative.h:101-115 and 122-139):
//          -1/2 (w_kj Tv_kj + w_ik Tv_ik) n_ik[r] n_kj[s]
// with S_i = sum of i's layer-l direction cosines, T_i = sum w Tv n over i's
// layer-l bonds.  The diagonal block (derivative.h:8-45) is
//   K_ii[r][s] = sum_l M_i[r][s] + T_i[r] S_i[s]   (r <= s),  M_i = sum w (2Kn+Tv) n n^T,
// then mirrored as derivative.h:37-42 does ([1][0] stays 0 in the as-written
// variant).  Common neighbours k of i and j come from a merge of the two
// particles' partner-sorted layer-l bond lists.
__device__ __forceinline__ void seg(const int64_t* bptr, const int64_t* lptr, int i, int l, int64_t& b, int64_t& e) {
  b = l == 0 ? bptr[i] : lptr[i];
  e = l == 0 ? lptr[i] : bptr[i + 1];
}

template <int DIM>
__device__ __forceinline__ void diag_block(const AsmView& v, int i, double (&K)[3][3]) {
  double k00 = 0, k01 = 0, k02 = 0, k11 = 0, k12 = 0, k22 = 0;
#pragma unroll
  for (int l = 0; l < NL; ++l) {
    const double* M = v.msum + (NL * i + l) * 6;
    const double* T = v.tsum + (NL * i + l) * 3;
    const double* S = v.cs_sum + (NL * i + l) * 3;
    k00 += M[0] + T[0] * S[0];
    k01 += M[1] + T[0] * S[1];
    k02 += M[2] + T[0] * S[2];
    k11 += M[3] + T[1] * S[1];
    k12 += M[4] + T[1] * S[2];
    k22 += M[5] + T[2] * S[2];
  }
  K[0][0] = k00;
  K[0][1] = k01;
  K[0][2] = k02;
  K[1][0] = v.sym ? k01 : 0.0;
  K[1][1] = k11;
  K[1][2] = k12;
  K[2][0] = k02;
  K[2][1] = k12;
  K[2][2] = k22;
}

// A bond's direction cosines and half its damaged Tv.
struct BondRec {
  double n[3], t;
};
__device__ __forceinline__ BondRec bond_rec(const AsmView& v, int64_t b) {
  return BondRec{{v.cs[3 * b], v.cs[3 * b + 1], v.cs[3 * b + 2]}, 0.5 * ((1 - v.bdamage[b]) * v.Tv[b])};
}
// Of the bond at sorted place s, and of its opposite.
template <bool REC>
__device__ __forceinline__ BondRec own_rec(const AsmView& v, int64_t s) {
  if (!REC) return bond_rec(v, v.sbond[s]);
  const double2 a = __ldg(v.rec + 2 * s), b = __ldg(v.rec + 2 * s + 1);
  return BondRec{{a.x, a.y, b.x}, b.y};
}
template <bool REC>
__device__ __forceinline__ BondRec opp_rec(const AsmView& v, int64_t s) {
  return REC ? own_rec<true>(v, __ldg(v.sopp + s)) : bond_rec(v, v.opp[v.sbond[s]]);
}

__global__ void k_bond_records(int64_t nb, const int* __restrict__ sbond, const double* __restrict__ cs,
                               const double* __restrict__ Tv, const double* __restrict__ bdamage,
                               double2* __restrict__ rec) {
  for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < nb; s += (int64_t)gridDim.x * blockDim.x) {
    const int64_t b = sbond[s];
    rec[2 * s] = make_double2(cs[3 * b], cs[3 * b + 1]);
    rec[2 * s + 1] = make_double2(cs[3 * b + 2], 0.5 * ((1 - bdamage[b]) * Tv[b]));
  }
}
__global__ void k_sorted_place(int64_t nb, const int* __restrict__ sbond, int* __restrict__ place) {
  for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < nb; s += (int64_t)gridDim.x * blockDim.x)
    place[sbond[s]] = (int)s;
}
__global__ void k_sorted_opp(int64_t nb, const int* __restrict__ sbond, const int* __restrict__ opp,
                             const int* __restrict__ place, int* __restrict__ sopp) {
  for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < nb; s += (int64_t)gridDim.x * blockDim.x)
    sopp[s] = place[opp[sbond[s]]];
}

template <int DIM, bool REC>
__device__ __forceinline__ void off_block(const AsmView& v, int i, int j, double (&K)[3][3]) {
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) K[r][c] = 0.0;
#pragma unroll 1
  for (int l = 0; l < NL; ++l) {
    int64_t ia, ea, ib, eb;
    seg(v.bptr, v.lptr, i, l, ia, ea);
    seg(v.bptr, v.lptr, j, l, ib, eb);
    int64_t direct = -1;
    int pb = ib < eb ? __ldg(v.sp2 + ib) : INT_MAX;
    // merge of the partner-sorted lists; the direct bond i->j shows up as
    // partner j in i's list.  The lanes of a warp walk (integers) each to
    // its next common neighbour and then take its FP64 terms together.
#pragma unroll 1
    for (;;) {
      bool match = false;
#pragma unroll 1
      for (; ia < ea; ++ia) {
        const int pa = __ldg(v.sp2 + ia);
        if (pa == j) direct = ia;
        while (pb < pa) pb = ++ib < eb ? __ldg(v.sp2 + ib) : INT_MAX;
        if (pb == pa) {
          match = true;
          break;
        }
      }
      if (!match) break;
      const BondRec a = own_rec<REC>(v, ia++), b = opp_rec<REC>(v, ib);  // i -> k, k -> j
      const double h = a.t + b.t;
#pragma unroll
      for (int r = 0; r < DIM; ++r) {
        const double hr = h * a.n[r];
#pragma unroll
        for (int c = 0; c < DIM; ++c) K[r][c] = fma(-hr, b.n[c], K[r][c]);
      }
    }
    if (direct >= 0) {
      const BondRec a = own_rec<REC>(v, direct);
      const int64_t b = v.sbond[direct];
      const double wt = 2.0 * a.t, wn = 2.0 * ((1 - v.bdamage[b]) * v.Kn[b]) + wt;
      const double* Sj = v.cs_sum + (NL * j + l) * 3;
      const double* Si = v.cs_sum + (NL * i + l) * 3;
      const double* Ti = v.tsum + (NL * i + l) * 3;
      double p[DIM];
#pragma unroll
      for (int c = 0; c < DIM; ++c) p[c] = fma(wt, Sj[c], -(wn * a.n[c]));
#pragma unroll
      for (int r = 0; r < DIM; ++r) {
        const double o = fma(0.5, fma(wt, Si[r], Ti[r]), -(wt * a.n[r]));
#pragma unroll
        for (int c = 0; c < DIM; ++c) K[r][c] = fma(a.n[r], p[c], fma(-o, a.n[c], K[r][c]));
      }
    }
  }
}

template <int DIM, bool REC>
__device__ __forceinline__ void store_block(const AsmView& v, int64_t slot, int i, int j) {
  double K[3][3];
  if (i == j)
    diag_block<DIM>(v, i, K);
  else
    off_block<DIM, REC>(v, i, j, K);
#pragma unroll
  for (int r = 0; r < DIM; ++r)
#pragma unroll
    for (int s = 0; s < DIM; ++s) v.A[(r * DIM + s) * v.nslots + slot] = K[s][r];
}

// A block per slice of A = K^T: lane t owns row j = 32*slice + t, the warps
// share the row's blocks.  Each block K_ij is computed by its row's lane and
// its transpose stored in the row's slot.
//
// Bound by the FP64 pipe (13 operations per common neighbour and layer, 36 per
// direct bond: 0.6 ms of 51^3 particles), if the lanes' blocks see the same
// neighbourhood and so walk and multiply together.  On a lattice those are the
// blocks of equal i - j, not the k-th of each row: the first row past an edge
// of the lattice shifts them.  So the warps go through the offsets i - j of the
// slice's longest row (`off`, in shared memory), each lane taking the block of
// its own row at that offset if it has one, and then through the blocks at
// other offsets.  (Where a sample of the rows' offsets has fewer than half
// among the longest row's, the rows are taken as they are: a polycrystal of 27k
// particles 0.49 ms, by offsets 0.54.)  The records bring a bond's data in two loads instead of
// seven (sorted place, bond, its opposite, four arrays).
//
// Assembly and conditions, with one warp per slice taking the k-th blocks from
// the raw arrays, then with the warps and the records, then by offsets: a 7k
// plate 333, 82 and 67 us, a 21^3 cube 1203, 258 and 180 us, 51^3 2914, 1559
// and 1080 us, 101^3 17.8, 8.9 and 7.3 ms.
template <int DIM, bool REC>
__global__ void __launch_bounds__(kAsmThreads) k_assemble(AsmView v, int noff) {
  extern __shared__ int off[];  // [noff], ascending
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int j = blockIdx.x * kSlice + lane;
  const int len = j < v.n ? v.rowlen[j] : 0;
  const SellRow row = sell_row(v.sell_ptr, min(j, v.n - 1));
  int longest = len;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) longest = max(longest, __shfl_xor_sync(0xffffffffu, longest, o));
  const int src = __ffs(__ballot_sync(0xffffffffu, len == longest)) - 1;
  int m = min(longest, noff);  // offsets
  {
    const int js = blockIdx.x * kSlice + src;
    const SellRow rs = sell_row(v.sell_ptr, js);
    for (int k = threadIdx.x; k < m; k += blockDim.x) off[k] = v.scol[sell_slot(rs, k)] - js;
  }
  __syncthreads();
  auto place = [&](int o) {  // of the first offset not below o
    int lo = 0, hi = m;
    while (lo < hi) {
      const int t = (lo + hi) / 2;
      if (off[t] < o)
        lo = t + 1;
      else
        hi = t;
    }
    return lo;
  };
  auto listed = [&](int o) {
    const int t = place(o);
    return t < m && off[t] == o;
  };
  int found = 0, asked = 0;
#pragma unroll 1
  for (int q = 1; q < 4; ++q) {
    const bool has = len > 0, in = has && listed(v.scol[sell_slot(row, len * q / 4)] - j);
    asked += __popc(__ballot_sync(0xffffffffu, has));
    found += __popc(__ballot_sync(0xffffffffu, in));
  }
  if (2 * found < asked) m = 0;
#pragma unroll 1
  for (int t = warp; t < m; t += nw) {
    const int i = j + off[t];
    int lo = 0, hi = len;  // the first block of a column not below i
    while (lo < hi) {
      const int k = (lo + hi) / 2;
      if (v.scol[sell_slot(row, k)] < i)
        lo = k + 1;
      else
        hi = k;
    }
    if (lo < len && v.scol[sell_slot(row, lo)] == i) store_block<DIM, REC>(v, sell_slot(row, lo), i, j);
  }
#pragma unroll 1
  for (int k = warp; k < len; k += nw) {
    const int64_t slot = sell_slot(row, k);
    const int i = v.scol[slot];
    if (!listed(i - j)) store_block<DIM, REC>(v, slot, i, j);
  }
}

// |diag(K)|_2 (stiffness.h:269-270) and the DOFs to eliminate
// (stiffness.h:277: disp_constraint or damage_visual == 1).
template <int DIM>
__global__ void k_diag_norm_fixed(int n, const int* __restrict__ diag_slot, const double* __restrict__ A,
                                  int64_t nslots, const int* __restrict__ mask, const double* __restrict__ dvis,
                                  unsigned char* __restrict__ fixed, double* partials, unsigned int* ticket,
                                  double* norms) {
  double v[1] = {0.0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int s = diag_slot[i];
    const bool dead = fabs(dvis[i] - 1.0) < EPS;
#pragma unroll
    for (int r = 0; r < DIM; ++r) {
      if (s >= 0) {
        const double a = A[(r * DIM + r) * nslots + s];
        v[0] += a * a;
      }
      fixed[DIM * i + r] = (mask[3 * i + r] == 1 || dead) ? 1 : 0;
    }
  }
  double tot[1];
  if (grid_sum<1>(v, partials, ticket, tot) && threadIdx.x == 0) norms[2] = sqrt(tot[0]);
}

// Zero the rows and columns of fixed DOFs, norm on their diagonal
// (stiffness.h:273-291).  Entry (r, s) of block (j, i) of A is K(i s, j r).
// A block per slice, its warps sharing the rows' blocks (a warp per slice took
// 58 us of a 21^3 cube and 77 of 51^3, here 12 and 43).
template <int DIM>
__global__ void __launch_bounds__(256) k_apply_bc(int n, const int64_t* __restrict__ sell_ptr,
                                                  const int* __restrict__ scol, const int* __restrict__ rowlen,
                                                  const unsigned char* __restrict__ fixed, const double* norms,
                                                  double* __restrict__ A, int64_t nslots) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int j = blockIdx.x * kSlice + lane;
  if (j >= n) return;
  const double nd = norms[2];
  unsigned char fj[DIM];
#pragma unroll
  for (int r = 0; r < DIM; ++r) fj[r] = fixed[DIM * j + r];
  const int len = rowlen[j];
  const SellRow row = sell_row(sell_ptr, j);
  for (int k = warp; k < len; k += nw) {
    const int64_t slot = sell_slot(row, k);
    const int i = scol[slot];
#pragma unroll
    for (int r = 0; r < DIM; ++r)
#pragma unroll
      for (int s = 0; s < DIM; ++s)
        if (fj[r] || fixed[DIM * i + s]) A[(r * DIM + s) * nslots + slot] = (i == j && r == s) ? nd : 0.0;
  }
}

// 16-bit column offsets (column - row) of the slots the product reads for
// row j (sell_read_len).  The flag is set when one does not fit; the other
// slots are never read.
__global__ void k_col_offsets(int n, const int64_t* __restrict__ sell_ptr, const int* __restrict__ scol,
                              const int* __restrict__ rowlen, short* __restrict__ soff, int* flag) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const SellRow row = sell_row(sell_ptr, j);
  const int len = sell_read_len(row, rowlen[j]);
  bool bad = false;
  for (int k = 0; k < len; ++k) {
    const int64_t s = sell_slot(row, k);
    const int o = scol[s] - j;
    bad |= (o < -32768 || o > 32767);
    soff[s] = (short)o;
  }
  if (bad) atomicOr(flag, 1);
}

// The FP32 copy of the rows' slots and S_i = sum_j A_ij over row i's blocks,
// summed in FP64 and rounded once; padding slots are zero in both.  A block
// per slice, its warps sharing the groups, their sums added in the warps'
// order.  Bound by the FP64 pipe where the chip is full (an addition and a
// conversion an element: 281 us of 51^3 particles as two passes, 287 as one)
// and by latency where it is not: 99 us of 21^3 and 21 of a 61x121 plate with
// a thread per row, here 29 and 10.
constexpr int kConvertWarps = 8;
template <int DIM>
__global__ void __launch_bounds__(32 * kConvertWarps) k_convert(int n, const int64_t* __restrict__ sell_ptr,
                                                                const double* __restrict__ A, int64_t nslots,
                                                                float* __restrict__ B, float* __restrict__ S) {
  constexpr int E = DIM * DIM;
  __shared__ double sum[kConvertWarps][E][32];
  const int sl = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t base = sell_ptr[sl];
  const int w = (int)((sell_ptr[sl + 1] - base) / kSlice), g4 = w / kVec * kVec;
  double acc[E];
#pragma unroll
  for (int e = 0; e < E; ++e) acc[e] = 0.0;
#pragma unroll 1
  for (int g = warp * kVec; g < g4; g += kConvertWarps * kVec) {
    const int64_t s = base + (int64_t)g * kSlice + lane * kVec;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const double2* q = reinterpret_cast<const double2*>(A + e * nslots + s);
      const double2 lo = __ldcs(q), hi = __ldcs(q + 1);
      *reinterpret_cast<float4*>(B + e * nslots + s) = make_float4((float)lo.x, (float)lo.y, (float)hi.x, (float)hi.y);
      acc[e] += (lo.x + lo.y) + (hi.x + hi.y);
    }
  }
  for (int k = g4 + warp; k < w; k += kConvertWarps) {
    const int64_t s = base + (int64_t)k * kSlice + lane;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const double a = A[e * nslots + s];
      B[e * nslots + s] = (float)a;
      acc[e] += a;
    }
  }
#pragma unroll
  for (int e = 0; e < E; ++e) sum[warp][e][lane] = acc[e];
  __syncthreads();
  const int i = sl * kSlice + lane;
  if (i < n)
    for (int e = warp; e < E; e += kConvertWarps) {
      double t = sum[0][e][lane];
#pragma unroll
      for (int q = 1; q < kConvertWarps; ++q) t += sum[q][e][lane];
      S[(int64_t)i * E + e] = (float)t;
    }
}

}  // namespace

int build_pattern(lpm_handle* h) {
  Dev& d = h->d;
  const int n = h->n, T = 128;
  int64_t* cnt = (int64_t*)dev_alloc(h, sizeof(int64_t) * (size_t)n);
  int64_t* cand_ptr = (int64_t*)dev_alloc(h, sizeof(int64_t) * ((size_t)n + 1));
  if (!cnt || !cand_ptr) return LPM_ERR_NOMEM;
  k_count_candidates<<<grid_for(n, T), T, 0, h->stream>>>(n, d.bptr, d.lptr, d.bp2, d.blayer, cnt);
  LPM_LAUNCHED(h, "k_count_candidates");
  std::vector<int64_t> hc((size_t)n), hp((size_t)n + 1, 0);
  LPM_CUDA(h, cudaMemcpyAsync(hc.data(), cnt, sizeof(int64_t) * n, cudaMemcpyDeviceToHost, h->stream));
  LPM_CUDA(h, cudaStreamSynchronize(h->stream));
  for (int i = 0; i < n; ++i) hp[(size_t)i + 1] = hp[(size_t)i] + hc[(size_t)i];
  LPM_CUDA(h, cudaMemcpyAsync(cand_ptr, hp.data(), sizeof(int64_t) * (n + 1), cudaMemcpyHostToDevice, h->stream));
  int* cand = nullptr;
  LPM_CUDA(h, cudaMallocAsync((void**)&cand, sizeof(int) * (size_t)std::max<int64_t>(hp[(size_t)n], 1), h->stream));
  k_fill_candidates<<<grid_for(n, kCandWarps), 32 * kCandWarps, 0, h->stream>>>(n, d.bptr, d.lptr, d.bp2, d.blayer,
                                                                                cand_ptr, cand, cnt);
  LPM_LAUNCHED(h, "k_fill_candidates");
  if (*std::max_element(hc.begin(), hc.end()) > kWarpCand) {
    k_fill_candidates_long<<<grid_for(n, T), T, 0, h->stream>>>(n, d.bptr, d.lptr, d.bp2, cand_ptr, cand, cnt);
    LPM_LAUNCHED(h, "k_fill_candidates_long");
  }
  LPM_CUDA(h, cudaMemcpyAsync(hc.data(), cnt, sizeof(int64_t) * n, cudaMemcpyDeviceToHost, h->stream));
  LPM_CUDA(h, cudaStreamSynchronize(h->stream));
  std::vector<int64_t> cp((size_t)n + 1, 0);
  for (int i = 0; i < n; ++i) cp[(size_t)i + 1] = cp[(size_t)i] + hc[(size_t)i];
  h->nblk = cp[(size_t)n];
  if (h->nblk >= (int64_t)1 << 31) {
    cudaFreeAsync(cand, h->stream);
    h->err = "pattern has 2^31 or more blocks";
    return LPM_ERR_ARG;
  }
  // sliced layout: each slice is as long as its longest row (groups of four,
  // then a tail of at most three single blocks)
  h->nslice = (n + kSlice - 1) / kSlice;
  std::vector<int64_t> sp((size_t)h->nslice + 1, 0);
  for (int sl = 0; sl < h->nslice; ++sl) {
    int64_t mx = 0;
    for (int j = sl * kSlice; j < std::min(n, (sl + 1) * kSlice); ++j) mx = std::max(mx, hc[(size_t)j]);
    sp[(size_t)sl + 1] = sp[(size_t)sl] + mx * kSlice;
  }
  h->nslots = sp[(size_t)h->nslice];
  h->sell_host = sp;
  h->maxw = 0;
  for (int sl = 0; sl < h->nslice; ++sl)
    h->maxw = std::max(h->maxw, (int)((sp[(size_t)sl + 1] - sp[(size_t)sl]) / kSlice));
  if (h->nslots >= (int64_t)1 << 31) {
    cudaFreeAsync(cand, h->stream);
    h->err = "sliced operator has 2^31 or more slots";
    return LPM_ERR_ARG;
  }
  d.cptr = (int64_t*)dev_alloc(h, sizeof(int64_t) * ((size_t)n + 1));
  d.cidx = (int*)dev_alloc(h, sizeof(int) * (size_t)std::max<int64_t>(h->nblk, 1));
  d.diag_slot = (int*)dev_alloc(h, sizeof(int) * (size_t)n);
  d.sell_ptr = (int64_t*)dev_alloc(h, sizeof(int64_t) * ((size_t)h->nslice + 1));
  d.scol = (int*)dev_alloc(h, sizeof(int) * (size_t)std::max<int64_t>(h->nslots, 1));
  d.rowlen = (int*)dev_alloc(h, sizeof(int) * (size_t)n);
  if (!d.cptr || !d.cidx || !d.diag_slot || !d.sell_ptr || !d.scol || !d.rowlen) {
    cudaFreeAsync(cand, h->stream);
    return LPM_ERR_NOMEM;
  }
  LPM_CUDA(h, cudaMemcpyAsync(d.cptr, cp.data(), sizeof(int64_t) * (n + 1), cudaMemcpyHostToDevice, h->stream));
  LPM_CUDA(h, cudaMemcpyAsync(d.sell_ptr, sp.data(), sizeof(int64_t) * (h->nslice + 1), cudaMemcpyHostToDevice,
                              h->stream));
  LPM_CUDA(h, cudaMemsetAsync(d.scol, 0, sizeof(int) * (size_t)std::max<int64_t>(h->nslots, 1), h->stream));
  k_compact_pattern<<<grid_for(n, T), T, 0, h->stream>>>(n, cand_ptr, cand, d.cptr, d.cidx);
  LPM_LAUNCHED(h, "k_compact_pattern");
  k_fill_sell<<<grid_for(n, T), T, 0, h->stream>>>(n, d.cptr, d.cidx, d.sell_ptr, d.scol, d.rowlen, d.diag_slot);
  LPM_LAUNCHED(h, "k_fill_sell");
  LPM_CUDA(h, cudaFreeAsync(cand, h->stream));
  LPM_CUDA(h, cudaStreamSynchronize(h->stream));
  return LPM_OK;
}

// The bonds' records of an assembly: 1 made, 0 no memory for them, or an error.
static int bond_records(lpm_handle* h) {
  Dev& d = h->d;
  if (h->no_records || h->nb == 0) return 0;
  const int T = 256, G = grid_for((long long)h->nb, T, 152 * 32);
  if (!d.brec) {
    // the records and each one's opposite; given back where memory runs short later
    // (handle_malloc)
    double* rec = (double*)dev_alloc(h, sizeof(double) * 4 * (size_t)h->nb);
    int *sopp = rec ? (int*)dev_alloc(h, sizeof(int) * (size_t)h->nb) : nullptr, *place = nullptr;
    if (!sopp || cudaMallocAsync((void**)&place, sizeof(int) * (size_t)h->nb, h->stream) != cudaSuccess) {
      cudaGetLastError();
      h->err.clear();
      h->no_records = true;
      if (sopp) dev_free(h, sopp);
      if (rec) dev_free(h, rec);
      return 0;
    }
    d.brec = rec;
    d.sopp = sopp;
    k_sorted_place<<<G, T, 0, h->stream>>>(h->nb, d.sbond, place);
    LPM_LAUNCHED(h, "k_sorted_place");
    k_sorted_opp<<<G, T, 0, h->stream>>>(h->nb, d.sbond, d.opp, place, d.sopp);
    LPM_LAUNCHED(h, "k_sorted_opp");
    LPM_CUDA(h, cudaFreeAsync(place, h->stream));
  }
  k_bond_records<<<G, T, 0, h->stream>>>(h->nb, d.sbond, d.cs, d.Tv, d.bdamage, (double2*)d.brec);
  LPM_LAUNCHED(h, "k_bond_records");
  return 1;
}

int launch_assemble(lpm_handle* h, int tangent, int bc) {
  if (h->mf) return mf_assemble(h, tangent, bc);
  Dev& d = h->d;
  const int dim = h->dim;
  const size_t vals = (size_t)h->nslots * dim * dim;
  if (!d.A64) {
    d.A64 = (double*)dev_alloc(h, sizeof(double) * std::max<size_t>(vals, 1));
    if (!d.A64) return LPM_ERR_NOMEM;
    // padding slots stay zero for the life of the handle
    LPM_CUDA(h, cudaMemsetAsync(d.A64, 0, sizeof(double) * std::max<size_t>(vals, 1), h->stream));
  }
  const int ra = bond_records(h);
  if (ra < 0) return ra;
  AsmView v{d.bptr, d.lptr, d.sell_ptr, d.scol, d.rowlen, d.sbond, d.sp2, d.opp, d.cs, d.cs_sum, d.tsum, d.msum,
            d.Kn, d.Tv, d.bdamage, (const double2*)d.brec, d.sopp, d.A64, h->nslots, h->n, h->nslice,
            tangent == LPM_TANGENT_SYMMETRIC ? 1 : 0};
  {
    const int TA = 32 * std::min(kAsmThreads / 32, std::max(1, (h->maxw + kVec - 1) / kVec));
    const int noff = std::min(h->maxw, 48 * 1024 / (int)sizeof(int));
    const size_t sm = sizeof(int) * (size_t)noff;
    if (dim == 3)
      (ra ? k_assemble<3, true> : k_assemble<3, false>)<<<h->nslice, TA, sm, h->stream>>>(v, noff);
    else
      (ra ? k_assemble<2, true> : k_assemble<2, false>)<<<h->nslice, TA, sm, h->stream>>>(v, noff);
    LPM_LAUNCHED(h, "k_assemble");
  }
  if (bc == LPM_BC_ELIMINATE) {
    const int GR = grid_for(h->n, kRedThreads, kMaxRedBlocks);
    if (dim == 3)
      k_diag_norm_fixed<3><<<GR, kRedThreads, 0, h->stream>>>(h->n, d.diag_slot, d.A64, h->nslots, d.mask, d.dvis,
                                                              d.fixed, d.red.partials, d.red.ticket + 1, d.norms);
    else
      k_diag_norm_fixed<2><<<GR, kRedThreads, 0, h->stream>>>(h->n, d.diag_slot, d.A64, h->nslots, d.mask, d.dvis,
                                                              d.fixed, d.red.partials, d.red.ticket + 1, d.norms);
    LPM_LAUNCHED(h, "k_diag_norm_fixed");
    if (dim == 3)
      k_apply_bc<3><<<h->nslice, 256, 0, h->stream>>>(h->n, d.sell_ptr, d.scol, d.rowlen, d.fixed, d.norms, d.A64,
                                            h->nslots);
    else
      k_apply_bc<2><<<h->nslice, 256, 0, h->stream>>>(h->n, d.sell_ptr, d.scol, d.rowlen, d.fixed, d.norms, d.A64,
                                            h->nslots);
    LPM_LAUNCHED(h, "k_apply_bc");
  }
  h->have_K = true;
  h->a32_valid = false;
  h->coarse_valid = false;
  h->last_bc = bc;
  h->tangent = tangent;
  return LPM_OK;
}

// FP32 copy of the operator for the mixed-precision solve, with the block
// row sums the difference-form product needs.
int convert_A32(lpm_handle* h) {
  Dev& d = h->d;
  const int dim = h->dim;
  const size_t vals = (size_t)h->nslots * dim * dim;
  if (!d.A32) {
    d.A32 = (float*)dev_alloc(h, sizeof(float) * std::max<size_t>(vals, 1));
    if (!d.A32) return LPM_ERR_NOMEM;
  }
  if (!d.S32) {
    d.S32 = (float*)dev_alloc(h, sizeof(float) * std::max<size_t>((size_t)h->n * dim * dim, 1));
    if (!d.S32) return LPM_ERR_NOMEM;
  }
  if (!d.soff16) {  // the pattern is fixed for the handle: offsets once
    d.soff16 = (short*)dev_alloc(h, sizeof(short) * std::max<size_t>((size_t)h->nslots, 1));
    int* flag = (int*)dev_alloc(h, sizeof(int));
    if (!d.soff16 || !flag) return LPM_ERR_NOMEM;
    LPM_CUDA(h, cudaMemsetAsync(flag, 0, sizeof(int), h->stream));
    LPM_CUDA(h, cudaMemsetAsync(d.soff16, 0, sizeof(short) * std::max<size_t>((size_t)h->nslots, 1), h->stream));
    k_col_offsets<<<(h->n + 127) / 128, 128, 0, h->stream>>>(h->n, d.sell_ptr, d.scol, d.rowlen, d.soff16, flag);
    LPM_LAUNCHED(h, "k_col_offsets");
    int bad = 0;
    LPM_CUDA(h, cudaMemcpyAsync(&bad, flag, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
    LPM_CUDA(h, cudaStreamSynchronize(h->stream));
    h->soff16_ok = bad == 0;
  }
  if (dim == 3)
    k_convert<3><<<h->nslice, 32 * kConvertWarps, 0, h->stream>>>(h->n, d.sell_ptr, d.A64, h->nslots, d.A32, d.S32);
  else
    k_convert<2><<<h->nslice, 32 * kConvertWarps, 0, h->stream>>>(h->n, d.sell_ptr, d.A64, h->nslots, d.A32, d.S32);
  LPM_LAUNCHED(h, "k_convert");
  h->a32_valid = true;
  return LPM_OK;
}

}  // namespace lpm
