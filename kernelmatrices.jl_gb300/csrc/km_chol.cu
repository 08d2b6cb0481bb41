// Batched FP64 Cholesky spread over the chip: the leaf blocks K_j of the HODLR matrix
// (bdiag Cholesky of symmetricfactorize!, src/HODLR/src/symfact.jl:14-20) as two launches per NB
// columns, so that few large leaves fill every SM.
//
// A leaf of m points takes m^3 / 6 multiply-adds and an SM issues two a clock, so one CTA per
// leaf left 2 leaves of 500 points on 2 SMs for 7.2 ms and 64 leaves of 469 on 64 SMs for 6.1 ms.
// Here a step solves the rows below its NB x NB diagonal block (k_chol_panel), then updates the
// trailing triangle in 32 x 32 tiles, one CTA each, the first of which also factors the next
// diagonal block (k_chol_update).  The Nystrom panel rides along: A = L^{-1} Phi by the same steps
// on the r columns of Phi (a separate solve kernel took 1.6 ms for 256 leaves of 256 points, rank 72,
// a third of it in 32-step substitutions with one useful lane at a time).  Measured: 2 leaves of 500
// 7.21 -> 1.84 ms, 64 of 469 6.14 -> 3.5 ms, 256 of 256 2.85 -> 2.19 ms.
//
// Every element sees the operations of the blocked right-looking algorithm in the same order
// whatever the split: inside a block column c takes the updates of columns 0, 1, ... < c and one
// division by its pivot; a trailing element takes one fused multiply-add chain per step,
// subtracted once.  The factor's bits do not depend on the number of CTAs.
#include <algorithm>
#include <climits>

#include "km_kernels.h"

namespace km {

namespace {

constexpr int kTile = 32;

// One matrix of the batch: read at step 0 from `in`, later from `out` (lower triangles, leading
// dimension m; nothing above the diagonal of `out` is read or written).
struct CholMat {
  const double* in;
  double* out;
  int m;
  const double* pin;  // r columns of length m to be solved with the factor (read at step 0, then
  double* pout;       // from pout; leading dimension m): A = L^{-1} Phi
};

struct LeafMats {
  const double* K;
  double* Lf;
  const double* Phi;
  double* A;
  int r;
  DTree t;
  __device__ CholMat operator()(int64_t j) const {
    const int64_t off = d_leaf_koff(t, j), s = d_leaf_start(t, j) * r;
    return CholMat{K + off, Lf + off, d_leaf_size(t, j), Phi + s, A + s};
  }
};

// Cholesky factor of the NB x NB diagonal block at column k0, entries in D (row-major, leading
// dimension NB + 1, lower triangle), by 4 warps, lane = row.  Warp w updates the columns c = w mod 4
// (each quarter of the SM has its own FP64 pipe); the warp of the next column updates it first and
// forms its square root and divisions while the others are still updating: one barrier a column.
// The loops stay rolled: with the block in registers of one warp the unrolled code, run once,
// waited for its own instructions (58 us for 32 columns, now 36 us: NB times a square root, a
// division and an update).
template <int NB>
__device__ void chol_diag(double* D, const CholMat& M, int k0, int* __restrict__ info) {
  constexpr int LD = NB + 1;
  __shared__ int first_bad;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, m = M.m, kb = min(NB, m - k0);
  // column j (updated value y of row `lane`) into its final form
  auto finish = [&](int j, double y) {
    const double p = __shfl_sync(0xffffffffu, y, j);
    // p > 0 on the bits (an FP64 comparison is one more instruction of the FP64 pipe on the chain)
    const long long pb = __double_as_longlong(p);
    const bool ok = pb > 0 && pb <= 0x7ff0000000000000ll;
    if (!ok && lane == 0) atomicMin(&first_bad, k0 + j + 1);
    const double sd = ok ? sqrt(p) : 1.0;
    // (a zero numerator in an idle lane would send the warp through the slow division)
    const bool below = lane > j && lane < kb;
    const double x = below ? y : 1.0;
    const double v = x / sd;
    if (below || lane == j) D[lane * LD + j] = below ? v : sd;
  };
  if (threadIdx.x == 0) first_bad = INT_MAX;
  __syncthreads();
  if (w == 0) finish(0, lane < kb ? D[lane * LD] : 0.0);
  __syncthreads();
  auto update = [&](int c, int j) {
    if (lane >= c && lane < kb) D[lane * LD + c] = __fma_rn(-D[lane * LD + j], D[c * LD + j], D[lane * LD + c]);
  };
  for (int j = 0; j < kb; ++j) {
    const bool live = lane >= j && lane < kb;
    if (w == (j & 3) && live) M.out[(int64_t)(k0 + j) * m + k0 + lane] = D[lane * LD + j];
    const int c = j + 1 + ((w - j - 1) & 3);
    if (c == j + 1) {
      // next column first; this warp's other columns take column j in the next step
      if (c < kb)
        finish(c, lane >= c && lane < kb ? __fma_rn(-D[lane * LD + j], D[c * LD + j], D[lane * LD + c]) : 0.0);
    } else {
      for (int q = c; q < kb; q += 4) {
        if (j > 0 && c == j + 4) update(q, j - 1);
        update(q, j);
      }
    }
    __syncthreads();
  }
  if (threadIdx.x == 0 && first_bad != INT_MAX && *info == 0) *info = first_bad;
}

template <typename Mats, int NB>
__global__ void __launch_bounds__(128) k_chol_first(Mats mats, int* __restrict__ info) {
  __shared__ double D[NB * (NB + 1)];
  const CholMat M = mats(blockIdx.x);
  const int lane = threadIdx.x & 31, kb = min(NB, M.m);
  for (int c = threadIdx.x >> 5; c < kb; c += 4)
    if (lane >= c && lane < kb) D[lane * (NB + 1) + c] = M.in[(int64_t)c * M.m + lane];
  __syncthreads();
  chol_diag<NB>(D, M, 0, info + blockIdx.x);
}

// Rows below the diagonal block at column k0: x D' = a, and the block's rows of the r solved columns
// (their transposes are rows of the same kind): grid (matrix, 32-row chunk; the first `nrow` chunks
// below the block, then those of the columns), 4 warps, lane = row.  Warp l mod 4 finishes column
// l; every warp updates every fourth column, so the warp that finishes column l + 1 is the one that
// updated it: one barrier a column.  The rows of the factor divide by the pivot, the solved columns
// multiply by its reciprocal, as the triangular solve kernel does.
template <typename Mats, int NB>
__global__ void __launch_bounds__(128) k_chol_panel(Mats mats, int k0, int nrow, int r) {
  __shared__ double D[NB * (NB + 1)], V[32 * (NB + 1)], inv[NB];
  constexpr int LD = NB + 1;
  const CholMat M = mats(blockIdx.x);
  const int m = M.m, kb = min(NB, m - k0);
  const bool solve = (int)blockIdx.y >= nrow;
  const int row0 = solve ? ((int)blockIdx.y - nrow) * 32 : k0 + NB + (int)blockIdx.y * 32;
  if (kb <= 0 || (!solve && row0 >= m)) return;  // (rows below the block: it has all NB columns)
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, i = row0 + lane;
  double* v = V + lane * LD;
  if (solve) {
    const double* src = k0 == 0 ? M.pin : M.pout;
    for (int q = w; q < 32; q += 4)
      if (lane < kb) V[q * LD + lane] = row0 + q < r ? src[(int64_t)(row0 + q) * m + k0 + lane] : 1.0;
    if (w == 0 && lane < kb) inv[lane] = 1.0 / M.out[(int64_t)(k0 + lane) * m + k0 + lane];
  } else {
    const double* src = k0 == 0 ? M.in : M.out;
    for (int c = w; c < NB; c += 4) v[c] = i < m ? src[(int64_t)(k0 + c) * m + i] : 1.0;
  }
  for (int c = w; c < kb; c += 4)
    if (lane >= c && lane < kb) D[lane * LD + c] = M.out[(int64_t)(k0 + c) * m + k0 + lane];
  __syncthreads();
  if (w == 0) v[0] = solve ? __dmul_rn(v[0], inv[0]) : v[0] / D[0];
  __syncthreads();
  for (int l = 0; l < kb; ++l) {
    const double x = v[l];
    if (w == (l & 3) && !solve && i < m) M.out[(int64_t)(k0 + l) * m + i] = x;
    const int c = l + 1 + ((w - l - 1) & 3);
    if (c == l + 1) {
      // next column first; this warp's other columns take column l in the next step
      if (c < kb) {
        const double y = __fma_rn(-x, D[c * LD + l], v[c]);
        v[c] = solve ? __dmul_rn(y, inv[c]) : y / D[c * LD + c];
      }
    } else {
      const bool two = l > 0 && c == l + 4;
      const double xp = two ? v[l - 1] : 0.0;
      for (int q = c; q < kb; q += 4) {
        double y = v[q];
        if (two) y = __fma_rn(-xp, D[q * LD + l - 1], y);
        v[q] = __fma_rn(-x, D[q * LD + l], y);
      }
    }
    __syncthreads();
  }
  if (solve)
    for (int q = w; q < 32; q += 4)
      if (lane < kb && row0 + q < r) M.pout[(int64_t)(row0 + q) * m + k0 + lane] = V[q * LD + lane];
}

// Trailing update of one 32 x 32 tile: A[i, c] -= sum_l P[i, l] P[c, l] of the lower triangle (P the
// step's panel rows), or A[i, q] -= sum_l P[i, l] X[l, q] of the solved columns (X their rows of the
// step): grid (tile; the ntri tiles of the triangle, then row tiles x column tiles, matrix), 128
// threads with 2 x 4 outputs each.  The CTA of the first tile goes on to factor the next diagonal
// block, which lies inside it.
template <typename Mats, int NB>
__global__ void __launch_bounds__(128) k_chol_update(Mats mats, int k0, int ntri, int nb, int r, int* __restrict__ info) {
  __shared__ double Pi[kTile * (NB + 1)], Pc[kTile * (NB + 1)];
  constexpr int LD = NB + 1;
  const CholMat M = mats(blockIdx.y);
  const int m = M.m, r0 = k0 + NB, mr = m - r0;
  const bool solve = (int)blockIdx.x >= ntri;
  int bi, bc;
  if (solve) {
    bc = ((int)blockIdx.x - ntri) / nb;
    bi = (int)blockIdx.x - ntri - bc * nb;
  } else {
    bi = (int)((sqrtf(8.f * blockIdx.x + 1.f) - 1.f) * 0.5f);
    while (bi * (bi + 1) / 2 > (int)blockIdx.x) --bi;
    while ((bi + 1) * (bi + 2) / 2 <= (int)blockIdx.x) ++bi;
    bc = blockIdx.x - bi * (bi + 1) / 2;
  }
  if (bi * kTile >= mr) return;
  const int i0 = r0 + bi * kTile, c0 = solve ? bc * kTile : r0 + bc * kTile;
  const int clim = solve ? r : m;
  const double* src = solve ? (k0 == 0 ? M.pin : M.pout) : (k0 == 0 ? M.in : M.out);
  double* dst = solve ? M.pout : M.out;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  for (int l = w; l < NB; l += 4) {
    const double* col = M.out + (int64_t)(k0 + l) * m;
    Pi[lane * LD + l] = i0 + lane < m ? col[i0 + lane] : 0.0;
    if (!solve) Pc[lane * LD + l] = c0 + lane < m ? col[c0 + lane] : 0.0;
  }
  if (solve)
    for (int q = w; q < kTile; q += 4)
      if (lane < NB) Pc[q * LD + lane] = c0 + q < r ? M.pout[(int64_t)(c0 + q) * m + k0 + lane] : 0.0;
  const int ti = tid & 15, tc = tid >> 4;
  // columns tc + 8 q: those beyond the last, and the half of a diagonal tile above the diagonal
  // (rows below 16, columns from 16 on), are left out
  const int nq = min(4, (clim - c0 + 7) / 8);
  const bool diag = !solve && bi == bc;
  double a[2][4];
#pragma unroll
  for (int p = 0; p < 2; ++p)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = i0 + ti + 16 * p, c = c0 + tc + 8 * q;
      a[p][q] = (i < m && c < clim && (solve || i >= c)) ? src[(int64_t)c * m + i] : 0.0;
    }
  __syncthreads();
  double acc[2][4] = {};
#pragma unroll 4
  for (int l = 0; l < NB; ++l) {
    double x[2], y[4];
#pragma unroll
    for (int p = 0; p < 2; ++p) x[p] = Pi[(ti + 16 * p) * LD + l];
#pragma unroll
    for (int q = 0; q < 4; ++q) y[q] = Pc[(tc + 8 * q) * LD + l];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (q < nq) {
        if (!(diag && q >= 2)) acc[0][q] = __fma_rn(x[0], y[q], acc[0][q]);
        acc[1][q] = __fma_rn(x[1], y[q], acc[1][q]);
      }
  }
#pragma unroll
  for (int p = 0; p < 2; ++p)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = i0 + ti + 16 * p, c = c0 + tc + 8 * q;
      a[p][q] = __dsub_rn(a[p][q], acc[p][q]);
      if (i < m && c < clim && (solve || i >= c)) dst[(int64_t)c * m + i] = a[p][q];
    }
  if (blockIdx.x > 0) return;
  __syncthreads();
#pragma unroll
  for (int p = 0; p < 2; ++p)
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (tc + 8 * q < NB) Pi[(ti + 16 * p) * LD + tc + 8 * q] = a[p][q];
  __syncthreads();
  chol_diag<NB>(Pi, M, r0, info + blockIdx.y);
}

template <typename Mats, int NB>
int chol_steps(const Mats& mats, int64_t nmat, int mmax, int r, int* info, cudaStream_t st) {
  int launches = 1;
  k_chol_first<Mats, NB><<<(unsigned)nmat, 128, 0, st>>>(mats, info);
  for (int k0 = 0; k0 < mmax; k0 += NB) {
    const int rows = std::max(mmax - k0 - NB, 0), nb = (rows + kTile - 1) / kTile, nr = (r + 31) / 32;
    if (nb + nr > 0) {
      k_chol_panel<Mats, NB><<<dim3((unsigned)nmat, (unsigned)(nb + nr)), 128, 0, st>>>(mats, k0, nb, r);
      ++launches;
    }
    if (nb > 0) {
      const int ntri = nb * (nb + 1) / 2;
      k_chol_update<Mats, NB><<<dim3((unsigned)(ntri + nb * nr), (unsigned)nmat), 128, 0, st>>>(mats, k0, ntri, nb, r,
                                                                                               info);
      ++launches;
    }
  }
  return launches;
}

// C = R1 R2' (R1, R2 upper triangular) or, with the lower triangle of C'C wanted, L22 = I - C'C
// (zeros above the diagonal): 32 x 32 tiles, grid (tile, tile, node), 256 threads.
template <bool GRAM>
__global__ void __launch_bounds__(256) k_gnode_product(const GNodeDesc* __restrict__ nodes) {
  __shared__ double As[32 * 33], Bs[32 * 33];
  const GNodeDesc N = nodes[blockIdx.z];
  const int r = N.r, i0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
  if (i0 >= r || c0 >= r) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double acc[4] = {};  // row i0 + lane, columns c0 + w + 8 q
  if (!GRAM || i0 >= c0) {
    for (int l0 = GRAM ? 0 : max(i0, c0); l0 < r; l0 += 32) {
      __syncthreads();
      for (int u = w; u < 32; u += 8) {
        if (GRAM) {  // entry (l, i) of C: As[i][l]
          As[u * 33 + lane] = (l0 + lane < r && i0 + u < r) ? N.C[l0 + lane + (int64_t)(i0 + u) * r] : 0.0;
          Bs[u * 33 + lane] = (l0 + lane < r && c0 + u < r) ? N.C[l0 + lane + (int64_t)(c0 + u) * r] : 0.0;
        } else {     // entry (i, l) of R1, (c, l) of R2, zero below the diagonal
          As[lane * 33 + u] = (i0 + lane <= l0 + u && l0 + u < r) ? N.R1[i0 + lane + (int64_t)(l0 + u) * r] : 0.0;
          Bs[lane * 33 + u] = (c0 + lane <= l0 + u && l0 + u < r) ? N.R2[c0 + lane + (int64_t)(l0 + u) * r] : 0.0;
        }
      }
      __syncthreads();
#pragma unroll 8
      for (int l = 0; l < 32; ++l) {
        const double a = As[lane * 33 + l];
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[q] = __fma_rn(a, Bs[(w + 8 * q) * 33 + l], acc[q]);
      }
    }
  }
  const int i = i0 + lane;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int c = c0 + w + 8 * q;
    if (i < r && c < r) {
      if (GRAM) N.L22[i + (int64_t)c * r] = i < c ? 0.0 : (i == c ? 1.0 : 0.0) - acc[q];
      else N.C[i + (int64_t)c * r] = acc[q];
    }
  }
}

struct NodeMats22 {
  const GNodeDesc* nodes;
  __device__ CholMat operator()(int64_t q) const { return CholMat{nodes[q].L22, nodes[q].L22, nodes[q].r, nullptr, nullptr}; }
};

}  // namespace

// Node capacitances of the general factorisation: C = R1 R2', L22 = chol(I - C'C) (lower).
// info[q]: failing column (1-based) of node q, zero on entry.  One CTA a node, as before, took
// 70 ms at rank 496 (an FP64-bound 2/3 r^3 multiply-adds on one SM); tiles over all SMs 3.1 ms.
int launch_gnode(const GNodeDesc* nodes, int n, int maxr, int* info, cudaStream_t st) {
  const unsigned nt = (unsigned)((maxr + 31) / 32);
  k_gnode_product<false><<<dim3(nt, nt, (unsigned)n), 256, 0, st>>>(nodes);
  k_gnode_product<true><<<dim3(nt, nt, (unsigned)n), 256, 0, st>>>(nodes);
  return 2 + chol_steps<NodeMats22, 32>(NodeMats22{nodes}, n, maxr, 0, info, st);
}

// block widths and size limit of the shared-memory panel (m + NB) x (NB + 1) of the one-CTA kernel
// that float pairs use: a wider block at the same size would round differently
static int leaf_chol_width(int64_t m) {
  for (int64_t nb : {32, 16, 8})
    if ((m + nb) * (nb + 1) * (int64_t)sizeof(double) <= 200 * 1024) return (int)nb;
  return 0;
}

bool leaf_chol_f64_solves(const Tree& t) { return leaf_chol_width(t.max_leaf) == 32; }

int launch_leaf_chol_f64(const double* K, double* Lf, const double* Phi, double* A, int r, const Tree& t, int* info,
                         cudaStream_t st) {
  const LeafMats mats{K, Lf, Phi, A, r, dtree(t)};
  const int m = (int)t.max_leaf;
  switch (leaf_chol_width(m)) {
    case 32: return chol_steps<LeafMats, 32>(mats, t.nleaf, m, r, info, st);
    case 16: return chol_steps<LeafMats, 16>(mats, t.nleaf, m, 0, info, st);
    case 8: return chol_steps<LeafMats, 8>(mats, t.nleaf, m, 0, info, st);
  }
  return 0;
}

}  // namespace km
