// A lattice's bonds from the caller's list: CSR by (owner, layer) in input
// order (bond_layers order), the opposite of each bond (particle.h:207-209),
// each segment's partner-sorted view (the tangent's merge), the initial
// lengths.  Integer work, and lengths by the same operations as the host's
// (bond_length), so the arrays are those a serial pass over the list makes.
//
// On the host this was serial over the bonds, each with a search in memory it
// did not have in cache, and most of lpm_create: 45 ms of 51^3 particles (2.4M
// bonds), now 6 with the pattern.  Here a counting sort: counts by atomics,
// one scan, places by atomics, then each segment (six or twelve bonds of a
// lattice) put in input order by one thread; 0.2 ms together.  Bound by the
// copy of the list to the device.
#include <algorithm>

#include "lpm_device.cuh"

namespace lpm {
namespace {

constexpr int kScan = 1024;  // keys of a block of the scan

// Bonds per (owner, layer); ids and layers are in range (lpm_create).
__global__ void k_bond_count(int64_t nb, const int* __restrict__ p1, const int* __restrict__ layer,
                             int* __restrict__ cnt) {
  const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (b < nb) atomicAdd(&cnt[(int64_t)p1[b] * NL + layer[b]], 1);
}

// Exclusive scan in three kernels: within blocks of kScan keys (the blocks'
// totals to sums), of the totals in one block, the totals added.
__device__ int block_scan(int v, int* sm) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int s = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, s, o);
    if (lane >= o) s += t;
  }
  if (lane == 31) sm[warp] = s;
  __syncthreads();
  if (warp == 0) {
    int w = sm[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += t;
    }
    sm[lane] = w;
  }
  __syncthreads();
  return s + (warp ? sm[warp - 1] : 0);
}
__global__ void __launch_bounds__(kScan) k_scan_blocks(int m, const int* __restrict__ cnt, int* __restrict__ at,
                                                       int* __restrict__ sums) {
  __shared__ int sm[32];
  const int k = blockIdx.x * kScan + threadIdx.x;
  const int v = k < m ? cnt[k] : 0, s = block_scan(v, sm);
  if (k < m) at[k] = s - v;
  if (threadIdx.x == kScan - 1) sums[blockIdx.x] = s;
}
__global__ void __launch_bounds__(kScan) k_scan_totals(int m, int* __restrict__ sums) {
  __shared__ int sm[32];
  int base = 0;
  for (int k0 = 0; k0 < m; k0 += kScan) {
    const int k = k0 + threadIdx.x, v = k < m ? sums[k] : 0, s = block_scan(v, sm);
    if (k < m) sums[k] = base + s - v;
    base += sm[31];
    __syncthreads();
  }
}

// The segments' starts (at: the scan within blocks), as the handle keeps them
// and as the cursors of the fill.
__global__ void k_bond_starts(int n, int64_t nb, const int* __restrict__ sums, int* __restrict__ at,
                              int64_t* __restrict__ bptr, int64_t* __restrict__ lptr, int* __restrict__ cursor) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k == 0) bptr[n] = nb;
  if (k >= n * NL) return;
  const int s = at[k] + sums[k / kScan];
  at[k] = cursor[k] = s;
  if (k % NL == 0)
    bptr[k / NL] = s;
  else
    lptr[k / NL] = s;
}
static_assert(NL == 2, "one boundary between a particle's layers");

__global__ void k_bond_fill(int64_t nb, const int* __restrict__ p1, const int* __restrict__ layer,
                            int* __restrict__ cursor, int* __restrict__ src) {
  const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nb) return;
  src[atomicAdd(&cursor[(int64_t)p1[b] * NL + layer[b]], 1)] = (int)b;
}

// [a, a + m) in the order of less(): insertion for a lattice's segments,
// else heapsort.
template <typename L>
__device__ void sort_segment(int* a, int m, L less) {
  if (m <= 64) {
    for (int k = 1; k < m; ++k) {
      const int v = a[k];
      int t = k - 1;
      for (; t >= 0 && less(v, a[t]); --t) a[t + 1] = a[t];
      a[t + 1] = v;
    }
    return;
  }
  auto sift = [&](int r, int e) {
    const int v = a[r];
    for (int c; (c = 2 * r + 1) < e; r = c) {
      if (c + 1 < e && less(a[c], a[c + 1])) ++c;
      if (!less(v, a[c])) break;
      a[r] = a[c];
    }
    a[r] = v;
  };
  for (int r = m / 2 - 1; r >= 0; --r) sift(r, m);
  for (int e = m - 1; e > 0; --e) {
    const int v = a[0];
    a[0] = a[e];
    a[e] = v;
    sift(0, e);
  }
}
__global__ void k_bond_order(int m, int64_t nb, const int* __restrict__ at, int* __restrict__ src) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= m) return;
  const int b0 = at[k], b1 = k + 1 < m ? at[k + 1] : (int)nb;
  sort_segment(src + b0, b1 - b0, [](int a, int b) { return a < b; });
}

__global__ void k_bond_gather(int64_t nb, const int* __restrict__ src, const int* __restrict__ p1,
                              const int* __restrict__ p2, const int* __restrict__ layer, const double* __restrict__ Kn,
                              const double* __restrict__ Tv, const double* __restrict__ x, int* __restrict__ bp2,
                              int* __restrict__ blayer, double* __restrict__ kn, double* __restrict__ tv,
                              double* __restrict__ dis0, double* __restrict__ dis, double* __restrict__ dis_last,
                              int* __restrict__ sbond) {
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nb) return;
  const int b = src[q], i = p1[b], j = p2[b];
  bp2[q] = j;
  blayer[q] = layer[b];
  kn[q] = Kn[b];
  tv[q] = Tv[b];
  const double d = bond_length(x[3 * i] - x[3 * j], x[3 * i + 1] - x[3 * j + 1], x[3 * i + 2] - x[3 * j + 2]);
  dis0[q] = dis[q] = dis_last[q] = d;
  sbond[q] = (int)q;
}

// The first bond of the partner in the same layer that points back; flag: there is none.
__global__ void k_bond_opposite(int64_t nb, const int* __restrict__ src, const int* __restrict__ p1,
                                const int64_t* __restrict__ bptr, const int64_t* __restrict__ lptr,
                                const int* __restrict__ bp2, const int* __restrict__ blayer, int* __restrict__ opp,
                                int* flag) {
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nb) return;
  const int i = p1[src[q]], j = bp2[q];
  const int64_t c0 = blayer[q] == 0 ? bptr[j] : lptr[j], c1 = blayer[q] == 0 ? lptr[j] : bptr[j + 1];
  int64_t c = c0;
  while (c < c1 && bp2[c] != i) ++c;
  if (c < c1)
    opp[q] = (int)c;
  else
    *flag = 1;
}

// Each segment's bonds by partner (then by place), and a particle's bonds.
__global__ void k_bond_sorted(int m, int64_t nb, const int* __restrict__ at, const int* __restrict__ bp2,
                              int* __restrict__ sbond, int* __restrict__ sp2, int* __restrict__ nbonds) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= m) return;
  const int b0 = at[k], b1 = k + 1 < m ? at[k + 1] : (int)nb;
  sort_segment(sbond + b0, b1 - b0, [&](int a, int b) { return bp2[a] < bp2[b] || (bp2[a] == bp2[b] && a < b); });
  for (int b = b0; b < b1; ++b) sp2[b] = bp2[sbond[b]];
  if (k % NL == 0) nbonds[k / NL] = (k + NL < m ? at[k + NL] : (int)nb) - b0;
}

// Initial critical stretch and particle property.
__global__ void k_ones(int n, double* __restrict__ a, double* __restrict__ b) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) a[i] = b[i] = 1.0;
}

}  // namespace

// d.x and the handle's bond arrays are allocated, d.x filled.
int build_bonds(lpm_handle* h, const int* p1, const int* p2, const int* layer, const double* Kn, const double* Tv) {
  Dev& d = h->d;
  const int n = h->n, m = n * NL, T = 256;
  const int64_t nb = h->nb;
  const size_t B = (size_t)std::max<int64_t>(nb, 1);
  const int blocks = (m + kScan - 1) / kScan;
  // the list, the keys' counts and starts, the cursors, the scan's totals, the flag
  const size_t ints = 3 * B + 3 * (size_t)m + (size_t)blocks + 1, dbl = (2 * B);
  char* tmp = nullptr;
  LPM_CUDA(h, cudaMallocAsync((void**)&tmp, sizeof(double) * dbl + sizeof(int) * ints, h->stream));
  double *kn = (double*)tmp, *tv = kn + B;
  int *q1 = (int*)(tv + B), *q2 = q1 + B, *ql = q2 + B, *cnt = ql + B, *at = cnt + m, *cursor = at + m,
      *sums = cursor + m, *flag = sums + blocks;
  auto run = [&]() -> int {
    LPM_CUDA(h, cudaMemsetAsync(cnt, 0, sizeof(int) * (3 * (size_t)m + (size_t)blocks + 1), h->stream));
    if (nb) {
      LPM_CUDA(h, cudaMemcpyAsync(q1, p1, sizeof(int) * nb, cudaMemcpyHostToDevice, h->stream));
      LPM_CUDA(h, cudaMemcpyAsync(q2, p2, sizeof(int) * nb, cudaMemcpyHostToDevice, h->stream));
      LPM_CUDA(h, cudaMemcpyAsync(ql, layer, sizeof(int) * nb, cudaMemcpyHostToDevice, h->stream));
      LPM_CUDA(h, cudaMemcpyAsync(kn, Kn, sizeof(double) * nb, cudaMemcpyHostToDevice, h->stream));
      LPM_CUDA(h, cudaMemcpyAsync(tv, Tv, sizeof(double) * nb, cudaMemcpyHostToDevice, h->stream));
    }
    const int GB = grid_for(nb, T), GM = grid_for(m, T);
    k_bond_count<<<GB, T, 0, h->stream>>>(nb, q1, ql, cnt);
    LPM_LAUNCHED(h, "k_bond_count");
    k_scan_blocks<<<blocks, kScan, 0, h->stream>>>(m, cnt, at, sums);
    LPM_LAUNCHED(h, "k_scan_blocks");
    k_scan_totals<<<1, kScan, 0, h->stream>>>(blocks, sums);
    LPM_LAUNCHED(h, "k_scan_totals");
    k_bond_starts<<<GM, T, 0, h->stream>>>(n, nb, sums, at, d.bptr, d.lptr, cursor);
    LPM_LAUNCHED(h, "k_bond_starts");
    k_bond_fill<<<GB, T, 0, h->stream>>>(nb, q1, ql, cursor, d.bsrc);
    LPM_LAUNCHED(h, "k_bond_fill");
    k_bond_order<<<GM, T, 0, h->stream>>>(m, nb, at, d.bsrc);
    LPM_LAUNCHED(h, "k_bond_order");
    k_bond_gather<<<GB, T, 0, h->stream>>>(nb, d.bsrc, q1, q2, ql, kn, tv, d.x, d.bp2, d.blayer, d.Kn, d.Tv, d.dis0,
                                           d.dis, d.dis_last, d.sbond);
    LPM_LAUNCHED(h, "k_bond_gather");
    k_bond_opposite<<<GB, T, 0, h->stream>>>(nb, d.bsrc, q1, d.bptr, d.lptr, d.bp2, d.blayer, d.opp, flag);
    LPM_LAUNCHED(h, "k_bond_opposite");
    k_bond_sorted<<<GM, T, 0, h->stream>>>(m, nb, at, d.bp2, d.sbond, d.sp2, d.nbonds);
    LPM_LAUNCHED(h, "k_bond_sorted");
    k_ones<<<grid_for(n, T), T, 0, h->stream>>>(n, d.crit, d.pp);
    LPM_LAUNCHED(h, "k_ones");
    int bad = 0;
    LPM_CUDA(h, cudaMemcpyAsync(&bad, flag, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
    LPM_CUDA(h, cudaStreamSynchronize(h->stream));
    if (bad) {
      h->err = kNoOpposite;
      return LPM_ERR_TOPOLOGY;
    }
    return LPM_OK;
  };
  const int st = run();
  cudaFreeAsync(tmp, h->stream);
  return st;
}

}  // namespace lpm
