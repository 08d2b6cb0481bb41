// Batched FP64 Cholesky spread over the chip: the leaf blocks K_j of the HODLR matrix
// (bdiag Cholesky of symmetricfactorize!, src/HODLR/src/symfact.jl:14-20) as two launches per NB
// columns, so that few large leaves fill every SM.
//
// A leaf of m points takes m^3 / 6 multiply-adds and an SM issues two a clock, so one CTA per
// leaf left 2 leaves of 500 points on 2 SMs for 7.2 ms and 64 leaves of 469 on 64 SMs for 6.1 ms.
// Here a step solves the rows below its NB x NB diagonal block (k_chol_panel), then updates the
// trailing triangle in 32 x 32 tiles, one CTA each, the first of which also factors the next
// diagonal block (k_chol_update).  Measured: 2 leaves of 500
// 7.21 -> 1.84 ms, 64 of 469 6.14 -> 3.5 ms, 256 of 256 2.85 -> 2.19 ms.
//
// Every element sees the operations of the blocked right-looking algorithm in the same order
// whatever the split: inside a block column c takes the updates of columns 0, 1, ... < c and one
// division by its pivot; a trailing element takes one fused multiply-add chain per step,
// subtracted once.  The factor's bits do not depend on the number of CTAs.
#include <algorithm>

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
};

struct LeafMats {
  const double* K;
  double* Lf;
  DTree t;
  __device__ CholMat operator()(int64_t j) const {
    const int64_t off = d_leaf_koff(t, j);
    return CholMat{K + off, Lf + off, d_leaf_size(t, j)};
  }
};

// Cholesky factor of the NB x NB diagonal block at column k0 by one warp, a row per lane in
// registers: the pivot and the multipliers travel by shuffles, no barrier (about 8 us at NB = 32,
// a chain of NB square roots and divisions).  d: row `lane` of the block, columns <= lane.
template <int NB>
__device__ void chol_diag(double (&d)[NB], const CholMat& M, int k0, int* __restrict__ info) {
  const int lane = threadIdx.x & 31, m = M.m, kb = min(NB, m - k0);
  int bad = 0;
#pragma unroll
  for (int j = 0; j < NB; ++j) {
    if (j < kb) {
      const double p = __shfl_sync(0xffffffffu, d[j], j);
      const bool ok = p > 0.0;
      if (!ok && bad == 0) bad = k0 + j + 1;
      const double sd = ok ? sqrt(p) : 1.0;
      d[j] = lane == j ? sd : d[j] / sd;
#pragma unroll
      for (int c = j + 1; c < NB; ++c) d[c] = __fma_rn(-d[j], __shfl_sync(0xffffffffu, d[j], c), d[c]);
    }
  }
  if (lane < kb) {
#pragma unroll
    for (int c = 0; c < NB; ++c)
      if (c <= lane) M.out[(int64_t)(k0 + c) * m + k0 + lane] = d[c];
  }
  if (lane == 0 && bad && *info == 0) *info = bad;
}

template <typename Mats, int NB>
__global__ void __launch_bounds__(32) k_chol_first(Mats mats, int* __restrict__ info) {
  const CholMat M = mats(blockIdx.x);
  const int lane = threadIdx.x, kb = min(NB, M.m);
  double d[NB];
#pragma unroll
  for (int c = 0; c < NB; ++c) d[c] = (c <= lane && lane < kb) ? M.in[(int64_t)c * M.m + lane] : 0.0;
  chol_diag<NB>(d, M, 0, info + blockIdx.x);
}

// Rows below the diagonal block at column k0: x D' = a, grid (matrix, row chunk), a row per thread.
template <typename Mats, int NB>
__global__ void __launch_bounds__(128) k_chol_panel(Mats mats, int k0) {
  __shared__ double D[NB * (NB + 1)];
  constexpr int LD = NB + 1;
  const CholMat M = mats(blockIdx.x);
  const int m = M.m, row0 = k0 + NB + (int)(blockIdx.y * blockDim.x);
  if (row0 >= m) return;  // the block has all NB columns: rows exist below it
  const double* src = k0 == 0 ? M.in : M.out;
  const int i = row0 + threadIdx.x;
  double v[NB];
#pragma unroll
  for (int c = 0; c < NB; ++c) v[c] = i < m ? src[(int64_t)(k0 + c) * m + i] : 0.0;
  for (int e = threadIdx.x; e < NB * NB; e += blockDim.x) {
    const int r = e % NB, c = e / NB;
    if (r >= c) D[r * LD + c] = M.out[(int64_t)(k0 + c) * m + k0 + r];
  }
  __syncthreads();
  if (i >= m) return;
#pragma unroll
  for (int l = 0; l < NB; ++l) {
    v[l] /= D[l * LD + l];
#pragma unroll
    for (int c = l + 1; c < NB; ++c) v[c] = __fma_rn(-v[l], D[c * LD + l], v[c]);
  }
#pragma unroll
  for (int c = 0; c < NB; ++c) M.out[(int64_t)(k0 + c) * m + i] = v[c];
}

// Trailing update A[i, c] -= sum_l P[i, l] P[c, l] of one 32 x 32 tile, P the step's panel rows:
// grid (tile of the lower triangle, matrix), 128 threads with 2 x 4 outputs each.  The CTA of the
// first tile goes on to factor the next diagonal block, which lies inside it.
template <typename Mats, int NB>
__global__ void __launch_bounds__(128) k_chol_update(Mats mats, int k0, int* __restrict__ info) {
  __shared__ double Pi[kTile * (NB + 1)], Pc[kTile * (NB + 1)];
  constexpr int LD = NB + 1;
  const CholMat M = mats(blockIdx.y);
  const int m = M.m, r0 = k0 + NB, mr = m - r0;
  int bi = (int)((sqrtf(8.f * blockIdx.x + 1.f) - 1.f) * 0.5f);
  while (bi * (bi + 1) / 2 > (int)blockIdx.x) --bi;
  while ((bi + 1) * (bi + 2) / 2 <= (int)blockIdx.x) ++bi;
  const int bc = blockIdx.x - bi * (bi + 1) / 2;
  if (bi * kTile >= mr) return;
  const int i0 = r0 + bi * kTile, c0 = r0 + bc * kTile;
  const double* src = k0 == 0 ? M.in : M.out;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  for (int l = w; l < NB; l += 4) {
    const double* col = M.out + (int64_t)(k0 + l) * m;
    Pi[lane * LD + l] = i0 + lane < m ? col[i0 + lane] : 0.0;
    Pc[lane * LD + l] = c0 + lane < m ? col[c0 + lane] : 0.0;
  }
  const int ti = tid & 15, tc = tid >> 4;
  double a[2][4];
#pragma unroll
  for (int p = 0; p < 2; ++p)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = i0 + ti + 16 * p, c = c0 + tc + 8 * q;
      a[p][q] = (i < m && i >= c) ? src[(int64_t)c * m + i] : 0.0;
    }
  __syncthreads();
  double acc[2][4] = {};
#pragma unroll 8
  for (int l = 0; l < NB; ++l) {
    double x[2], y[4];
#pragma unroll
    for (int p = 0; p < 2; ++p) x[p] = Pi[(ti + 16 * p) * LD + l];
#pragma unroll
    for (int q = 0; q < 4; ++q) y[q] = Pc[(tc + 8 * q) * LD + l];
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[p][q] = __fma_rn(x[p], y[q], acc[p][q]);
  }
#pragma unroll
  for (int p = 0; p < 2; ++p)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = i0 + ti + 16 * p, c = c0 + tc + 8 * q;
      a[p][q] -= acc[p][q];
      if (i < m && i >= c) M.out[(int64_t)c * m + i] = a[p][q];
    }
  if (blockIdx.x > 0) return;
  __syncthreads();
#pragma unroll
  for (int p = 0; p < 2; ++p)
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (tc + 8 * q < NB) Pi[(ti + 16 * p) * LD + tc + 8 * q] = a[p][q];
  __syncthreads();
  if (w > 0) return;
  const int kb = min(NB, mr);
  double d[NB];
#pragma unroll
  for (int c = 0; c < NB; ++c) d[c] = (c <= lane && lane < kb) ? Pi[lane * LD + c] : 0.0;
  chol_diag<NB>(d, M, r0, info + blockIdx.y);
}

template <typename Mats, int NB>
int chol_steps(const Mats& mats, int64_t nmat, int mmax, int* info, cudaStream_t st) {
  int launches = 1;
  k_chol_first<Mats, NB><<<(unsigned)nmat, 32, 0, st>>>(mats, info);
  for (int k0 = 0; k0 + NB < mmax; k0 += NB) {
    const int rows = mmax - k0 - NB, nb = (rows + kTile - 1) / kTile;
    // one warp per CTA while that gives at most four CTAs an SM, so that the rows of few matrices
    // are solved by many SMs
    const int nt = nmat * ((rows + 31) / 32) <= 4 * 152 ? 32 : 128;
    k_chol_panel<Mats, NB><<<dim3((unsigned)nmat, (unsigned)((rows + nt - 1) / nt)), nt, 0, st>>>(mats, k0);
    k_chol_update<Mats, NB><<<dim3((unsigned)(nb * (nb + 1) / 2), (unsigned)nmat), 128, 0, st>>>(mats, k0, info);
    launches += 2;
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
  __device__ CholMat operator()(int64_t q) const { return CholMat{nodes[q].L22, nodes[q].L22, nodes[q].r}; }
};

}  // namespace

// Node capacitances of the general factorisation: C = R1 R2', L22 = chol(I - C'C) (lower).
// info[q]: failing column (1-based) of node q, zero on entry.  One CTA a node, as before, took
// 70 ms at rank 496 (an FP64-bound 2/3 r^3 multiply-adds on one SM); tiles over all SMs 3.1 ms.
int launch_gnode(const GNodeDesc* nodes, int n, int maxr, int* info, cudaStream_t st) {
  const unsigned nt = (unsigned)((maxr + 31) / 32);
  k_gnode_product<false><<<dim3(nt, nt, (unsigned)n), 256, 0, st>>>(nodes);
  k_gnode_product<true><<<dim3(nt, nt, (unsigned)n), 256, 0, st>>>(nodes);
  return 2 + chol_steps<NodeMats22, 32>(NodeMats22{nodes}, n, maxr, info, st);
}

int launch_leaf_chol_f64(const double* K, double* Lf, const Tree& t, int* info, cudaStream_t st) {
  const LeafMats mats{K, Lf, dtree(t)};
  const int m = (int)t.max_leaf;
  // block widths and size limit of the shared-memory panel (m + NB) x (NB + 1) of the one-CTA
  // kernel that float pairs use: a wider block at the same size would round differently
  auto fits = [&](int64_t nb) { return (m + nb) * (nb + 1) * (int64_t)sizeof(double) <= 200 * 1024; };
  if (fits(32)) return chol_steps<LeafMats, 32>(mats, t.nleaf, m, info, st);
  if (fits(16)) return chol_steps<LeafMats, 16>(mats, t.nleaf, m, info, st);
  if (fits(8)) return chol_steps<LeafMats, 8>(mats, t.nleaf, m, info, st);
  return 0;
}

}  // namespace km
