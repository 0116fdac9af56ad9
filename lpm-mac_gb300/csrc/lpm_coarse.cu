// Coarse-space preconditioner of the mixed solve (lpm_set_preconditioner):
//   M^-1 = D^-1 + P A_c^-1 P^T,   A_c = P^T A P,
// additive two-level Schwarz with Jacobi as its one-level part.  The columns
// of P are the rigid-body modes (2-D: two translations and the rotation;
// 3-D: three translations and three rotations) of boxes of particles
// (aggregates), zero on eliminated DOFs.  Jacobi leaves the smooth,
// long-wavelength error of the lattice to the CG iterations; the coarse
// correction takes it out, so the iteration count stops growing with the
// lattice's size and depends on the box's instead.
//
// Set-up once per handle (host): the aggregates from the initial positions
// (boxes of an edge `box`, numbered in the order of their first particle),
// their members, each particle's offset from its aggregate's centroid, and
// the aggregate pairs the operator's pattern couples.  Once per assembly
// (device): A_c in FP64, one block per aggregate pair summing over the pair's
// rows in a fixed order; then, in one cooperative launch, modes without
// stiffness (an aggregate whose DOFs are all eliminated, the rotation of a
// lone particle) set aside and the inverse by blocked Gauss-Jordan elimination
// without pivoting (A_c is symmetric positive definite on the remaining
// modes).  The solve applies it in its own loop (lpm_pcg.cu, k_mx_persistent).
#include <algorithm>
#include <cmath>
#include <unordered_map>
#include <vector>

#include "lpm_device.cuh"
#include "lpm_coarse.cuh"
#include "lpm_grid.cuh"

namespace lpm {

// Most coarse DOFs: the dense inverse (8 MB in FP64 at 1,024) stays in L2.
constexpr int kCoarseMax = 1024;
// Coarse DOFs aimed at when the box edge is chosen automatically.
constexpr int kCoarseTarget = 480;

namespace {

// out[m] += v times mode m's entry in direction k for a particle at offset
// (dx, dy, dz): the three (2-D: two) entries that are not zero (mode_row).
template <int DIM>
__device__ __forceinline__ void add_modes(int k, double dx, double dy, double dz, double v,
                                          double (&out)[kModes<DIM>]) {
  out[k] += v;
  if (DIM == 2) {
    out[2] = fma(v, k == 0 ? -dy : dx, out[2]);
  } else if (k == 0) {
    out[4] = fma(v, dz, out[4]);
    out[5] = fma(v, -dy, out[5]);
  } else if (k == 1) {
    out[3] = fma(v, -dz, out[3]);
    out[5] = fma(v, dx, out[5]);
  } else {
    out[3] = fma(v, dy, out[3]);
    out[4] = fma(v, -dx, out[4]);
  }
}

// A_c block (a, b) = sum over i in a, blocks (i, j) with j in b, of
// P_i^T A_ij P_j.  A block per pair: the threads take the pair's rows (the
// members of a with a block in b) in turn, walk each row's slots in order
// and, row by row, form A_ij P_j summed over the row before P_i^T is applied;
// the threads' sums are folded by a fixed tree.  Bound by the FP64 pipe and
// by the walk past the slots of other aggregates; with P_i^T applied slot by
// slot, all modes' products taken and a warp per pair it was 10 ms for the
// 41^3 cube.
constexpr int kPairThreads = 128;
template <int DIM>
__global__ void __launch_bounds__(kPairThreads) k_coarse_pairs(const int* __restrict__ pairs,
                                                               const int* __restrict__ prow_ptr,
                                                               const int* __restrict__ prow,
                                                               const int* __restrict__ agg,
                                                               const float* __restrict__ off,
                                                               const unsigned char* __restrict__ fixed,
                                                               const int64_t* __restrict__ sell_ptr,
                                                               const int* __restrict__ scol,
                                                               const int* __restrict__ rowlen,
                                                               const double* __restrict__ A, int64_t nslots, int nc,
                                                               double* __restrict__ Ac) {
  constexpr int NM = kModes<DIM>;
  const int a = pairs[2 * blockIdx.x], b = pairs[2 * blockIdx.x + 1];
  double c[NM][NM];
#pragma unroll
  for (int m = 0; m < NM; ++m)
#pragma unroll
    for (int q = 0; q < NM; ++q) c[m][q] = 0.0;
  for (int t = prow_ptr[blockIdx.x] + threadIdx.x; t < prow_ptr[blockIdx.x + 1]; t += kPairThreads) {
    const int i = prow[t];
    double ap[DIM][NM];  // (A P)_ib
#pragma unroll
    for (int r = 0; r < DIM; ++r)
#pragma unroll
      for (int q = 0; q < NM; ++q) ap[r][q] = 0.0;
    const int len = rowlen[i];
    const SellRow sr = sell_row(sell_ptr, i);
#pragma unroll 4
    for (int k = 0; k < len; ++k) {
      const int64_t s = sell_slot(sr, k);
      const int j = __ldg(&scol[s]);
      if (__ldg(&agg[j]) != b) continue;
      const double dx = off[3 * j], dy = off[3 * j + 1], dz = off[3 * j + 2];
#pragma unroll
      for (int q = 0; q < DIM; ++q) {
        if (fixed && fixed[(int64_t)DIM * j + q]) continue;
#pragma unroll
        for (int r = 0; r < DIM; ++r)
          add_modes<DIM>(q, dx, dy, dz, A[(int64_t)(r * DIM + q) * nslots + s], ap[r]);
      }
    }
    const double dx = off[3 * i], dy = off[3 * i + 1], dz = off[3 * i + 2];
#pragma unroll
    for (int q = 0; q < NM; ++q) {
      double col[NM];
#pragma unroll
      for (int m = 0; m < NM; ++m) col[m] = c[m][q];
#pragma unroll
      for (int r = 0; r < DIM; ++r)
        if (!(fixed && fixed[(int64_t)DIM * i + r])) add_modes<DIM>(r, dx, dy, dz, ap[r][q], col);
#pragma unroll
      for (int m = 0; m < NM; ++m) c[m][q] = col[m];
    }
  }
  __shared__ double part[kPairThreads / 32][NM * NM];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int m = 0; m < NM; ++m)
#pragma unroll
    for (int q = 0; q < NM; ++q) {
      double v = c[m][q];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
      if (lane == 0) part[warp][m * NM + q] = v;
    }
  __syncthreads();
  for (int e = threadIdx.x; e < NM * NM; e += kPairThreads) {
    double v = part[0][e];
    for (int w = 1; w < kPairThreads / 32; ++w) v += part[w][e];
    Ac[(int64_t)(a * NM + e / NM) * nc + b * NM + e % NM] = v;
  }
}

// The inverse of A_c by Gauss-Jordan elimination without pivoting, kInv
// columns at a time, ping-ponged between two buffers (step k reads one and
// writes the other).  With D the diagonal block of step k, P = D^-1 A_kj:
//   A_kj <- P,  A_ik <- -A_ik D^-1,  A_ij <- A_ij - A_ik P,  A_kk <- D^-1.
// A column at a time this was a grid barrier and a pass over the matrix per
// column, 3.8 ms at 480 coarse DOFs of which the barriers were most; in
// blocks it is two barriers and a rank-16 update per 16 columns, bound by
// the FP64 pipe (2 nc^3 operations).  The last block of the grid takes no
// part in the update: it works out the next step's D and inverts it
// meanwhile, a serial chain of 16 divisions.  The whole set-up of a 61x121
// plate (480 coarse DOFs) went from 3.9 to 0.77 ms, of a 41^3 cube from 18 to
// 3.3 ms.
//
// First, modes without stiffness (a diagonal entry at most 1e-12 of the
// largest) are set aside: their rows and columns become the identity's for
// the elimination, and the inverse's are cleared; `active` records which
// are kept.  A mode that the ones before it span (an aggregate with fewer free
// DOFs than modes) shows as a pivot of nothing but rounding, 1e-16 of the mode's
// diagonal entry, where those of slender bars still have 4e-6: at most kDependent
// of it, the mode is set aside then.  (P A_c^-1 P^T is that of the modes' space,
// whichever of them span it.)  The result is symmetrized, (B + B^T)/2, into the other buffer
// (X after an odd number of steps, else Y): elimination leaves the computed
// inverse of an ill-conditioned A_c slightly unsymmetric, and CG needs a
// symmetric preconditioner.
constexpr int kInv = 16;         // columns per step
constexpr int kInvRows = 16, kInvCols = 32;  // tile of the update
constexpr int kInvThreads = 256;
constexpr double kDependent = 1e-13;

// D^-1 of the block of step k after the update of step k - 1 (k > 0) applied
// to it, into dinv (global, kInv x kInv, identity beyond the matrix and for modes
// set aside; diag: the modes' diagonal entries).
__device__ void invert_diagonal(int nc, int k, const double* src, const double* panel, double* dinv,
                                double (&d)[kInv][kInv + 1], const double* diag, int* active) {
  const int r = threadIdx.x / kInv, c = threadIdx.x % kInv, i = k * kInv + r, j = k * kInv + c;
  const bool in = i < nc && j < nc;
  __shared__ double rp;
  __shared__ int dependent;
  double v = in ? __ldcg(&src[(int64_t)i * nc + j]) : (r == c ? 1.0 : 0.0);
  if (panel && in) {  // A_ij - A_i(k-1) P
    const int k0 = (k - 1) * kInv;
    for (int t = 0; t < kInv; ++t)
      v -= __ldcg(&src[(int64_t)i * nc + k0 + t]) * __ldcg(&panel[(int64_t)(k0 + t) * nc + j]);
  }
  d[r][c] = v;
  __syncthreads();
  for (int p = 0; p < kInv; ++p) {
    if (threadIdx.x == 0) {
      const int m = k * kInv + p;
      dependent = m < nc && fabs(d[p][p]) <= kDependent * fabs(__ldcg(&diag[m]));
      if (dependent) active[m] = 0;
      rp = 1.0 / d[p][p];
    }
    __syncthreads();
    const double q = rp, a = d[r][c], f = d[r][p], g = d[p][c];
    const bool aside = dependent;
    __syncthreads();
    if (aside)
      d[r][c] = r != p && c != p ? a : r == c ? 1.0 : 0.0;
    else if (r == p)
      d[r][c] = c == p ? q : a * q;
    else
      d[r][c] = c == p ? -a * q : a - f * q * g;
    __syncthreads();
  }
  dinv[threadIdx.x] = d[r][c];
}

__global__ void __launch_bounds__(kInvThreads) k_coarse_invert(int nc, double* X, double* Y, double* dinv,
                                                               double* diag, int* active, unsigned long long* gbar,
                                                               long long spin_limit, int* fault) {
  __shared__ double D[kInv][kInv + 1], L[kInvRows][kInv + 1], P[kInv][kInvCols];
  __shared__ double smax[kInvThreads / 32];
  const int64_t nn = (int64_t)nc * nc;
  const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
  const int last = gridDim.x - 1;  // the block that inverts; with one block it does everything
  unsigned long long target = 0;
  auto barrier = [&]() {
    target += gridDim.x;
    if (grid_barrier(gbar, target, spin_limit)) return true;
    if (threadIdx.x == 0) atomicExch(fault, 1);
    return false;
  };
  // modes without stiffness
  {
    double m = 0.0;
    for (int q = threadIdx.x; q < nc; q += blockDim.x) m = fmax(m, fabs(__ldcg(&X[(int64_t)q * nc + q])));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) smax[threadIdx.x >> 5] = m;
    __syncthreads();
    m = 0.0;
    for (int w = 0; w < kInvThreads / 32; ++w) m = fmax(m, smax[w]);
    for (int64_t q = t0; q < nc; q += stride) {
      const double a = __ldcg(&X[q * nc + q]);
      active[q] = fabs(a) > 1e-12 * m ? 1 : 0;
      diag[q] = active[q] ? a : 1.0;
    }
    if (!barrier()) return;
    for (int64_t e = t0; e < nn; e += stride) {
      const int r = (int)(e / nc), c = (int)(e % nc);
      if (!__ldcg(&active[r]) || !__ldcg(&active[c])) X[e] = r == c ? 1.0 : 0.0;
    }
    if (!barrier()) return;
  }
  if (blockIdx.x == last) invert_diagonal(nc, 0, X, nullptr, dinv, D, diag, active);
  if (!barrier()) return;
  const int steps = (nc + kInv - 1) / kInv;
  const int rows = (nc + kInvRows - 1) / kInvRows, cols = (nc + kInvCols - 1) / kInvCols;
  const int workers = last > 0 ? last : 1;
  for (int k = 0; k < steps; ++k) {
    const double* src = (k & 1) ? Y : X;
    double* dst = (k & 1) ? X : Y;
    const double* dk = dinv + (k & 1) * kInv * kInv;
    const int k0 = k * kInv, kb = min(kInv, nc - k0);
    // the row panel P, and D^-1 in its place
    for (int64_t e = t0; e < (int64_t)kb * nc; e += stride) {
      const int r = (int)(e / nc), j = (int)(e % nc);
      double v = 0.0;
      if (j >= k0 && j < k0 + kb) {
        v = __ldcg(&dk[r * kInv + j - k0]);
      } else if (__ldcg(&active[k0 + r])) {
        for (int t = 0; t < kb; ++t) v += __ldcg(&dk[r * kInv + t]) * __ldcg(&src[(int64_t)(k0 + t) * nc + j]);
      }
      dst[(int64_t)(k0 + r) * nc + j] = v;
    }
    if (!barrier()) return;
    if ((int)blockIdx.x == last && k + 1 < steps)
      invert_diagonal(nc, k + 1, src, dst, dinv + ((k + 1) & 1) * kInv * kInv, D, diag, active);
    if ((int)blockIdx.x < workers)
      for (int tile = blockIdx.x; tile < rows * cols; tile += workers) {
        const int i0 = tile / cols * kInvRows, j0 = tile % cols * kInvCols;
        __syncthreads();
        for (int e = threadIdx.x; e < kInvRows * kInv; e += kInvThreads) {
          const int r = e / kInv, t = e % kInv;
          L[r][t] = i0 + r < nc && t < kb && __ldcg(&active[k0 + t]) ? __ldcg(&src[(int64_t)(i0 + r) * nc + k0 + t])
                                                                      : 0.0;
        }
        // the k-th columns take D^-1 (in dst's row panel) and start from zero
        for (int e = threadIdx.x; e < kInv * kInvCols; e += kInvThreads) {
          const int t = e / kInvCols, j = j0 + e % kInvCols;
          P[t][e % kInvCols] = t < kb && j < nc ? __ldcg(&dst[(int64_t)(k0 + t) * nc + j]) : 0.0;
        }
        __syncthreads();
        for (int e = threadIdx.x; e < kInvRows * kInvCols; e += kInvThreads) {
          const int r = e / kInvCols, c = e % kInvCols, i = i0 + r, j = j0 + c;
          if (i >= nc || j >= nc || (i >= k0 && i < k0 + kb)) continue;
          double v = j >= k0 && j < k0 + kb ? 0.0 : __ldcg(&src[(int64_t)i * nc + j]);
#pragma unroll
          for (int t = 0; t < kInv; ++t) v -= L[r][t] * P[t][c];
          dst[(int64_t)i * nc + j] = v;
        }
      }
    if (!barrier()) return;
  }
  const double* res = (steps & 1) ? Y : X;
  double* out = (steps & 1) ? X : Y;
  for (int64_t e = t0; e < nn; e += stride) {
    const int i = (int)(e / nc), j = (int)(e % nc);
    out[e] = (!__ldcg(&active[i]) || !__ldcg(&active[j])) ? 0.0 : 0.5 * (__ldcg(&res[e]) + __ldcg(&res[(int64_t)j * nc + i]));
  }
}

// The same coarse correction for FP64 vectors, as three launches (the
// tangent solves' BiCGSTAB, whose loop runs from the host): y = P^T r with a
// block per aggregate, e = A_c^-1 y with a block per aggregate, then
// z = invd r + P e per row.
template <int DIM>
__global__ void __launch_bounds__(256) k_coarse_restrict64(int nagg, const int* __restrict__ mem_ptr,
                                                           const int* __restrict__ mem, const float* __restrict__ off,
                                                           const unsigned char* __restrict__ fixed,
                                                           const double* __restrict__ r, double* __restrict__ y) {
  constexpr int NM = kModes<DIM>;
  for (int ag = blockIdx.x; ag < nagg; ag += gridDim.x) {
    double acc[NM];
#pragma unroll
    for (int m = 0; m < NM; ++m) acc[m] = 0.0;
    for (int t = mem_ptr[ag] + threadIdx.x; t < mem_ptr[ag + 1]; t += blockDim.x) {
      const int i = mem[t];
#pragma unroll
      for (int k = 0; k < DIM; ++k) {
        const int64_t q = (int64_t)DIM * i + k;
        if (fixed[q]) continue;
        double w[NM];
        mode_row<DIM, double>(k, off[3 * i], off[3 * i + 1], off[3 * i + 2], w);
#pragma unroll
        for (int m = 0; m < NM; ++m) acc[m] += w[m] * r[q];
      }
    }
    block_sum<NM>(acc);
    if (threadIdx.x == 0)
#pragma unroll
      for (int m = 0; m < NM; ++m) y[ag * NM + m] = acc[m];
  }
}

template <int DIM>
__global__ void __launch_bounds__(256) k_coarse_solve64(int nagg, const double* __restrict__ Ainv,
                                                        const double* __restrict__ y, double* __restrict__ e) {
  constexpr int NM = kModes<DIM>;
  const int nc = nagg * NM;
  for (int ag = blockIdx.x; ag < nagg; ag += gridDim.x) {
    double acc[NM];
#pragma unroll
    for (int m = 0; m < NM; ++m) acc[m] = 0.0;
    for (int c = threadIdx.x; c < nc; c += blockDim.x)
#pragma unroll
      for (int m = 0; m < NM; ++m) acc[m] += Ainv[(int64_t)(ag * NM + m) * nc + c] * y[c];
    block_sum<NM>(acc);
    if (threadIdx.x == 0)
#pragma unroll
      for (int m = 0; m < NM; ++m) e[ag * NM + m] = acc[m];
  }
}

template <int DIM>
__global__ void k_coarse_prolong64(int n, const int* __restrict__ agg, const float* __restrict__ off,
                                   const unsigned char* __restrict__ fixed, const double* __restrict__ invd,
                                   const double* __restrict__ r, const double* __restrict__ e,
                                   double* __restrict__ z) {
  constexpr int NM = kModes<DIM>;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int ag = agg[i];
#pragma unroll
  for (int k = 0; k < DIM; ++k) {
    const int64_t q = (int64_t)DIM * i + k;
    double zi = invd[q] * r[q];
    if (!fixed[q]) {
      double w[NM];
      mode_row<DIM, double>(k, off[3 * i], off[3 * i + 1], off[3 * i + 2], w);
#pragma unroll
      for (int m = 0; m < NM; ++m) zi += w[m] * e[ag * NM + m];
    }
    z[q] = zi;
  }
}

}  // namespace

// The aggregates: boxes of edge `box` from the lowest corner of the
// particles' bounding box (box <= 0: the edge that gives about
// kCoarseTarget coarse DOFs for the box volume), numbered in the order of
// their first particle.  Writes agg[n] and the edge used; returns the count.
int coarse_boxes(int dim, int n, const double* x0, double box, int* agg, double* edge_out) {
  const int nm = dim == 3 ? 6 : 3;
  double lo[3], hi[3];
  for (int k = 0; k < 3; ++k) {
    lo[k] = hi[k] = n ? x0[k] : 0.0;
    for (int i = 0; i < n; ++i) {
      lo[k] = std::min(lo[k], x0[3 * i + k]);
      hi[k] = std::max(hi[k], x0[3 * i + k]);
    }
  }
  double edge = box;
  if (!(edge > 0.0)) {
    double vol = 1.0;
    for (int k = 0; k < dim; ++k) vol *= std::max(hi[k] - lo[k], 1e-300);
    edge = std::pow(vol / std::max(1, kCoarseTarget / nm), 1.0 / dim);
    if (!(edge > 0.0) || !std::isfinite(edge)) edge = 1.0;  // no extent (one particle): one box
  }
  std::unordered_map<int64_t, int> box_id;
  for (int i = 0; i < n; ++i) {
    int64_t key = 0;
    for (int k = 0; k < dim; ++k) key = key * 2000003 + (int64_t)std::floor((x0[3 * i + k] - lo[k]) / edge);
    auto it = box_id.emplace(key, (int)box_id.size()).first;
    agg[i] = it->second;
  }
  if (edge_out) *edge_out = edge;
  return (int)box_id.size();
}

int coarse_setup(lpm_handle* h) {
  Dev& d = h->d;
  const int n = h->n, dim = h->dim, nm = dim == 3 ? 6 : 3;
  std::vector<double> x0((size_t)3 * n);
  LPM_CUDA(h, cudaMemcpyAsync(x0.data(), d.x0, sizeof(double) * 3 * n, cudaMemcpyDeviceToHost, h->stream));
  std::vector<int64_t> cptr((size_t)n + 1);
  std::vector<int> cidx((size_t)h->nblk);
  LPM_CUDA(h, cudaMemcpyAsync(cptr.data(), d.cptr, sizeof(int64_t) * (n + 1), cudaMemcpyDeviceToHost, h->stream));
  LPM_CUDA(h, cudaMemcpyAsync(cidx.data(), d.cidx, sizeof(int) * h->nblk, cudaMemcpyDeviceToHost, h->stream));
  LPM_CUDA(h, cudaStreamSynchronize(h->stream));
  std::vector<int> agg((size_t)n);
  double edge = 0.0;
  const int nagg = coarse_boxes(dim, n, x0.data(), h->cbox, agg.data(), &edge);
  if ((long long)nagg * nm > kCoarseMax) {
    h->err = "coarse preconditioner: " + std::to_string(nagg) + " aggregates exceed " +
             std::to_string(kCoarseMax / nm) + "; give a larger box";
    return LPM_ERR_ARG;
  }
  std::vector<int> mem_ptr((size_t)nagg + 1, 0), mem((size_t)n);
  for (int i = 0; i < n; ++i) mem_ptr[(size_t)agg[(size_t)i] + 1]++;
  for (int a = 0; a < nagg; ++a) mem_ptr[(size_t)a + 1] += mem_ptr[(size_t)a];
  std::vector<int> fill(mem_ptr.begin(), mem_ptr.end() - 1);
  std::vector<double> cen((size_t)3 * nagg, 0.0);
  for (int i = 0; i < n; ++i) {
    const int a = agg[(size_t)i];
    mem[(size_t)fill[(size_t)a]++] = i;
    for (int k = 0; k < 3; ++k) cen[(size_t)3 * a + k] += x0[(size_t)3 * i + k];
  }
  std::vector<float> off((size_t)3 * n);
  for (int a = 0; a < nagg; ++a)
    for (int k = 0; k < 3; ++k) cen[(size_t)3 * a + k] /= std::max(1, mem_ptr[(size_t)a + 1] - mem_ptr[(size_t)a]);
  for (int i = 0; i < n; ++i)
    for (int k = 0; k < 3; ++k)
      off[(size_t)3 * i + k] = (float)(x0[(size_t)3 * i + k] - cen[(size_t)3 * agg[(size_t)i] + k]);
  // aggregate pairs coupled by the pattern, in order, each with its rows
  // (the members of a with a block in b, ascending)
  std::vector<int> pairs, prow_ptr(1, 0), prow;
  std::vector<int> seen_row((size_t)nagg, -1);
  std::vector<std::vector<int>> rows_of((size_t)nagg);
  std::vector<int> nbr;
  for (int a = 0; a < nagg; ++a) {
    nbr.clear();
    for (int t = mem_ptr[(size_t)a]; t < mem_ptr[(size_t)a + 1]; ++t) {
      const int i = mem[(size_t)t];
      for (int64_t q = cptr[(size_t)i]; q < cptr[(size_t)i + 1]; ++q) {
        const int b = agg[(size_t)cidx[(size_t)q]];
        if (seen_row[(size_t)b] == i) continue;
        if (rows_of[(size_t)b].empty()) nbr.push_back(b);
        seen_row[(size_t)b] = i;
        rows_of[(size_t)b].push_back(i);
      }
    }
    std::sort(nbr.begin(), nbr.end());
    for (int b : nbr) {
      pairs.push_back(a);
      pairs.push_back(b);
      prow.insert(prow.end(), rows_of[(size_t)b].begin(), rows_of[(size_t)b].end());
      prow_ptr.push_back((int)prow.size());
      rows_of[(size_t)b].clear();
    }
  }
  const int nc = nagg * nm;
  const int64_t ndof = (int64_t)n * dim;
  d.cagg = (int*)dev_alloc(h, sizeof(int) * n);
  d.cmem_ptr = (int*)dev_alloc(h, sizeof(int) * (nagg + 1));
  d.cmem = (int*)dev_alloc(h, sizeof(int) * n);
  d.cpair = (int*)dev_alloc(h, sizeof(int) * std::max<size_t>(pairs.size(), 1));
  d.cprow_ptr = (int*)dev_alloc(h, sizeof(int) * prow_ptr.size());
  d.cprow = (int*)dev_alloc(h, sizeof(int) * std::max<size_t>(prow.size(), 1));
  d.coff = (float*)dev_alloc(h, sizeof(float) * 3 * n);
  d.cA = (double*)dev_alloc(h, sizeof(double) * (size_t)nc * nc);
  d.cA2 = (double*)dev_alloc(h, sizeof(double) * (size_t)nc * nc);
  d.cact = (int*)dev_alloc(h, sizeof(int) * nc);
  d.cyc = (double*)dev_alloc(h, sizeof(double) * nc);
  d.cec = (double*)dev_alloc(h, sizeof(double) * nc);
  d.cz = (float*)dev_alloc(h, sizeof(float) * ndof);
  d.cfault = (int*)dev_alloc(h, sizeof(int));
  d.cdinv = (double*)dev_alloc(h, sizeof(double) * 2 * kInv * kInv);
  if (!d.cagg || !d.cmem_ptr || !d.cmem || !d.cpair || !d.cprow_ptr || !d.cprow || !d.coff || !d.cA || !d.cA2 ||
      !d.cact || !d.cyc || !d.cec || !d.cz || !d.cfault || !d.cdinv)
    return LPM_ERR_NOMEM;
  LPM_CUDA(h, cudaMemcpyAsync(d.cagg, agg.data(), sizeof(int) * n, cudaMemcpyHostToDevice, h->stream));
  LPM_CUDA(h, cudaMemcpyAsync(d.cmem_ptr, mem_ptr.data(), sizeof(int) * (nagg + 1), cudaMemcpyHostToDevice,
                              h->stream));
  LPM_CUDA(h, cudaMemcpyAsync(d.cmem, mem.data(), sizeof(int) * n, cudaMemcpyHostToDevice, h->stream));
  if (!pairs.empty())
    LPM_CUDA(h, cudaMemcpyAsync(d.cpair, pairs.data(), sizeof(int) * pairs.size(), cudaMemcpyHostToDevice,
                                h->stream));
  LPM_CUDA(h, cudaMemcpyAsync(d.coff, off.data(), sizeof(float) * 3 * n, cudaMemcpyHostToDevice, h->stream));
  LPM_CUDA(h, cudaMemcpyAsync(d.cprow_ptr, prow_ptr.data(), sizeof(int) * prow_ptr.size(), cudaMemcpyHostToDevice,
                              h->stream));
  if (!prow.empty())
    LPM_CUDA(h, cudaMemcpyAsync(d.cprow, prow.data(), sizeof(int) * prow.size(), cudaMemcpyHostToDevice, h->stream));
  LPM_CUDA(h, cudaStreamSynchronize(h->stream));
  h->cnagg = nagg;
  h->cnc = nc;
  h->cnpair = (int)(pairs.size() / 2);
  h->cedge = edge;
  h->coarse_valid = false;
  return pcg_coarse_plan(h, agg, nagg);
}

// A_c of the current operator and its symmetrized inverse (in d.cAinv).
int coarse_assemble(lpm_handle* h) {
  Dev& d = h->d;
  if (!d.cagg) {
    const int st = coarse_setup(h);
    if (st) return st;
  }
  const int nc = h->cnc;
  const unsigned char* fixed = h->last_bc == LPM_BC_ELIMINATE ? d.fixed : nullptr;
  LPM_CUDA(h, cudaMemsetAsync(d.cA, 0, sizeof(double) * (size_t)nc * nc, h->stream));
  if (h->cnpair > 0) {
    if (h->dim == 3)
      k_coarse_pairs<3><<<h->cnpair, kPairThreads, 0, h->stream>>>(d.cpair, d.cprow_ptr, d.cprow, d.cagg, d.coff, fixed,
                                                                  d.sell_ptr, d.scol, d.rowlen, d.A64, h->nslots, nc,
                                                                  d.cA);
    else
      k_coarse_pairs<2><<<h->cnpair, kPairThreads, 0, h->stream>>>(d.cpair, d.cprow_ptr, d.cprow, d.cagg, d.coff, fixed,
                                                                  d.sell_ptr, d.scol, d.rowlen, d.A64, h->nslots, nc,
                                                                  d.cA);
    LPM_LAUNCHED(h, "k_coarse_pairs");
  }
  // a block per SM: the barriers cost more with more
  const int grid = std::max(1, sm_count(h));
  LPM_CUDA(h, cudaMemsetAsync(d.gbar, 0, sizeof(unsigned long long), h->stream));
  LPM_CUDA(h, cudaMemsetAsync(d.cfault, 0, sizeof(int), h->stream));
  long long spin = kPcgSpinLimit;
  int ncv = nc;
  // (d.cyc, the solves' y, holds the diagonal meanwhile)
  void* args[] = {&ncv, &d.cA, &d.cA2, &d.cdinv, &d.cyc, &d.cact, &d.gbar, &spin, &d.cfault};
  LPM_CUDA(h, cudaLaunchCooperativeKernel((const void*)k_coarse_invert, dim3(grid), dim3(kInvThreads), args, 0,
                                          h->stream));
  LPM_LAUNCHED(h, "k_coarse_invert");
  int fault = 0;
  LPM_CUDA(h, cudaMemcpyAsync(&fault, d.cfault, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
  LPM_CUDA(h, cudaStreamSynchronize(h->stream));
  if (fault) {
    h->err = "coarse preconditioner: a grid-barrier wait gave up in the inversion";
    return LPM_ERR_STATE;
  }
  d.cAinv = ((nc + kInv - 1) / kInv & 1) ? d.cA : d.cA2;
  h->coarse_valid = true;
  return LPM_OK;
}

}  // namespace lpm

namespace lpm {

// The coarse correction applies to the tangent solves when the user chose it
// and the last assembly is the symmetric tangent with the displacement BCs
// eliminated (its eliminated DOFs contain the constrained ones, on which the
// correction is zero).
bool coarse_usable(const lpm_handle* h) {
  return h->precond == LPM_PRECOND_COARSE && h->have_K && !h->mf && h->tangent == LPM_TANGENT_SYMMETRIC &&
         h->last_bc == LPM_BC_ELIMINATE;
}

int coarse_apply64(lpm_handle* h, const double* r, const double* invd, double* z) {
  Dev& d = h->d;
  if (!h->coarse_valid) {
    const int st = coarse_assemble(h);
    if (st) return st;
  }
  const int nagg = h->cnagg;
  if (h->dim == 3) {
    k_coarse_restrict64<3><<<nagg, 256, 0, h->stream>>>(nagg, d.cmem_ptr, d.cmem, d.coff, d.fixed, r, d.cyc);
    k_coarse_solve64<3><<<nagg, 256, 0, h->stream>>>(nagg, d.cAinv, d.cyc, d.cec);
    k_coarse_prolong64<3><<<grid_for(h->n, 256), 256, 0, h->stream>>>(h->n, d.cagg, d.coff, d.fixed, invd, r, d.cec, z);
  } else {
    k_coarse_restrict64<2><<<nagg, 256, 0, h->stream>>>(nagg, d.cmem_ptr, d.cmem, d.coff, d.fixed, r, d.cyc);
    k_coarse_solve64<2><<<nagg, 256, 0, h->stream>>>(nagg, d.cAinv, d.cyc, d.cec);
    k_coarse_prolong64<2><<<grid_for(h->n, 256), 256, 0, h->stream>>>(h->n, d.cagg, d.coff, d.fixed, invd, r, d.cec, z);
  }
  LPM_LAUNCHED(h, "k_coarse_apply64");
  h->stats.kernel_launches += 2;
  return LPM_OK;
}

}  // namespace lpm
