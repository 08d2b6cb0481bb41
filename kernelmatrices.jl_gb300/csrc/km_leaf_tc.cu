// Mixed-precision leaf stage on the tensor cores: blocked Cholesky of the augmented leaf matrix
//
//     [ K_j     ]   =   [ L_j ] [ L_j' A_j ]        A_j = L_j^{-1} Phi_j
//     [ Phi_j'  ]       [ A_j']
//
// so that one factorisation gives the leaf factor L_j (leaf Cholesky, src/HODLR/src/symfact.jl:17)
// and the transformed leaf panel A_j = L_j^{-1} Phi_j (the leaf-level invapply!,
// src/HODLR/src/utils.jl:54-65, BlockDiagonal.jl:62-66) in float pairs.  The rows of Phi_j' are
// the columns of A_j as stored (m x r column-major), so "row g" of the lower part is column g of
// the panel buffer.
//
// Per 64-column block (step) of every leaf:
//   * k_lc_diag (CUDA cores, one CTA per leaf): Cholesky D of the 64 x 64 diagonal block and,
//     in the same column sweep, X = D^{-1} (float pairs, shared memory); the rows of X cut into
//     bf16 slices for the next kernel;
//   * k_lc_trsm (tensor cores, one CTA per 128-row tile of the rows below the block: trailing
//     rows of K_j, then the rows of Phi_j'): the block column P = A X' (the triangular solve
//     P D' = A with the explicit inverse of the diagonal block) as a split product, written back
//     and cut into slices (with row exponents) for the update;
//   * k_lc_update (tensor cores, one CTA per 128 x 64 tile of the trailing rows / columns):
//     C -= P P' from the slices.
// A float-pair value is cut into kSlices bf16 slices with a row exponent (km_tc.cuh); both
// products take the 28 slice products with i + j <= 6, accumulated per diagonal i + j in tensor
// memory (exact integer sums in fp32), and the epilogues add the 7 diagonal sums in float pairs
// and scale them by 2^(e_row + e_col).  The leaf matrices enter in float pairs (written by the
// mixed-form leaf evaluation).
#include "km_kernels.h"
#include "km_tc.cuh"

namespace km {

using tc::kSlices;

constexpr int kLcNB = 64;              // panel width = K of the products
constexpr int kLcTileM = 128;          // rows of a tile (MMA M)
constexpr int kLcTileN = 64;           // columns of a tile (MMA N)
constexpr int kLcTcThreads = 512;      // 16 warps: warp w reads tensor-memory lanes 32 (w % 4) .. + 31,
                                       // columns 16 (w / 4) .. + 15 of a tile
constexpr int kLcDiagThreads = 512;
constexpr int kLcProbeThreads = 256;
constexpr uint32_t kLcTmemCols = 512;  // kSlices x kLcTileN = 448 accumulator columns
constexpr uint32_t kATileBytes = kLcTileM * kLcNB * 2;  // one slice of a 128-row tile
constexpr uint32_t kBTileBytes = kLcTileN * kLcNB * 2;  // one slice of a 64-row tile
constexpr long long kTcWaitLimit = 1ll << 21;           // mbarrier polls before giving up
constexpr int kLcMaxLeaf = 1024;
constexpr int kLcMaxRank = 256;

__host__ __device__ inline int64_t lc_rows_padded(int64_t rows) { return (rows + 127) / 128 * 128; }

// bf16 element index of (slice s, row rho, column c) in a slice array of rp rows: core matrix
// (rho / 8, c / 8) of slice s is 64 consecutive elements, core matrices ordered by slice, then
// row group, then column group.
__host__ __device__ inline int64_t lc_slice_index(int s, int64_t rp, int64_t rho, int c) {
  return ((((int64_t)s * (rp / 8) + rho / 8) * 8 + c / 8) * 64) + (rho % 8) * 8 + (c % 8);
}

// Writes the kSlices slices of 8 consecutive values (columns 8 kc .. 8 kc + 7 of row rho).
__device__ __forceinline__ void store_slices8(uint16_t* base, int64_t rp, int64_t rho, int kc, const ff (&x)[8],
                                              int e) {
  uint32_t w[kSlices][4];
#pragma unroll
  for (int cc = 0; cc < 8; cc += 2) {
    float t0[kSlices], t1[kSlices];
    tc::split_slices(x[cc], e, t0);
    tc::split_slices(x[cc + 1], e, t1);
#pragma unroll
    for (int s = 0; s < kSlices; ++s) w[s][cc / 2] = tc::bf16_pack2(t0[s], t1[s]);
  }
#pragma unroll
  for (int s = 0; s < kSlices; ++s)
    *reinterpret_cast<uint4*>(base + lc_slice_index(s, rp, rho, 8 * kc)) =
        make_uint4(w[s][0], w[s][1], w[s][2], w[s][3]);
}

// Split products of one 128 x 64 tile: A slices (kSlices x kATileBytes) times B slices
// (kSlices x kBTileBytes) into kSlices accumulators of kLcTileN columns, one per diagonal i + j.
__device__ __forceinline__ void lc_issue_products(uint32_t tmem, uint32_t smA, uint32_t smB) {
  constexpr uint32_t idesc = tc::idesc_bf16(kLcTileM, kLcTileN);
#pragma unroll 1
  for (int d = 0; d < kSlices; ++d) {
    bool first = true;
#pragma unroll 1
    for (int i = 0; i <= d; ++i) {
      const int j = d - i;
#pragma unroll
      for (int ks = 0; ks < kLcNB / 16; ++ks) {
        const uint64_t ad = tc::smem_desc(smA + i * kATileBytes + ks * 256, 128, 1024);
        const uint64_t bd = tc::smem_desc(smB + j * kBTileBytes + ks * 256, 128, 1024);
        tc::mma_bf16(tmem + d * kLcTileN, ad, bd, idesc, !first);
        first = false;
      }
    }
  }
}

// The 8 float-pair values of accumulator columns j0 .. j0 + 7 of this thread's lane: the 7
// diagonal sums combined and scaled by 2^(erow + ecol[jj]).
__device__ __forceinline__ void lc_tile_values(uint32_t tl, int j0, int erow, const int* ecol, ff (&out)[8]) {
  float s[kSlices][8];
#pragma unroll
  for (int d = 0; d < kSlices; ++d) tc::tmem_ld8(tl + d * kLcTileN + j0, s[d]);
  tc::tmem_wait_ld();
#pragma unroll
  for (int jj = 0; jj < 8; ++jj) {
    float sd[kSlices];
#pragma unroll
    for (int d = 0; d < kSlices; ++d) sd[d] = s[d][jj];
    out[jj] = tc::ff_ldexp(tc::combine_diagonals(sd), erow + ecol[jj]);
  }
}

// ---------------------------------------------------------------------------------------------
// Diagonal block: grid = nleaf, block = kLcDiagThreads, dynamic shared memory 2 x 64 x 65 float
// pairs.  D = chol(B) and X = D^{-1} for the block B = rows / columns [c0, c0 + nb) of the
// matrix being factored (row j of X is finalised at step j, then rows i > j subtract L_ij X_j);
// beyond nb both are the identity.  The chain of square roots and reciprocals bounds it: with two block
// barriers a column 256 leaves took 118 us a block, by panels of 4 columns (the same operations on every
// entry in the same order) 77 us.  Writes D to Lf and the slices of the rows of X (64 rows,
// the canonical layout) with their exponents.
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kLcDiagThreads) k_lc_diag(ff* __restrict__ Lf, DTree t, int c0,
                                                            uint16_t* __restrict__ xsl, int* __restrict__ xexp,
                                                            int* __restrict__ info) {
  extern __shared__ __align__(16) unsigned char lc_smem_d[];
  constexpr int LD = kLcNB + 1;
  ff* D = reinterpret_cast<ff*>(lc_smem_d);
  ff* X = D + kLcNB * LD;
  const int64_t leaf = blockIdx.x;
  const int m = d_leaf_size(t, leaf);
  if (c0 >= m) return;
  const int nb = min(kLcNB, m - c0);
  const int64_t koff = d_leaf_koff(t, leaf);
  const int tid = threadIdx.x, NT = blockDim.x;
  for (int e = tid; e < kLcNB * kLcNB; e += NT) {
    const int i = e % kLcNB, c = e / kLcNB;
    ff v(0.0);
    if (i < nb && c < nb) {
      if (i >= c) v = Lf[koff + (int64_t)(c0 + c) * m + c0 + i];
    } else if (i == c) {
      v = ff(1.0);
    }
    D[i * LD + c] = v;
    X[i * LD + c] = ff(i == c ? 1.0 : 0.0);
  }
  // Panels of 4 columns.  In step p the four warps of one SM quarter apply panel p - 1 to panel p, a
  // column each, and warp 0 factors panel p in registers; warps 1 and 2, a thread per column of X, apply
  // the rows of panel p - 2 to those of panel p - 1 and finish these; the other warps apply panel p - 1 to
  // the columns of D behind panel p and the rows of panel p - 2 of X to its rows from panel p on.
  __shared__ ff srinv[kLcNB];
  constexpr int kP = 4;
  const int w = tid >> 5, lane = tid & 31, np = (nb + kP - 1) / kP;
  // the workers: warps 3, 5, 6, 7, 9, 10, 11, 13, 14, 15
  const int wi = (w & 3) == 0 || w < 3 ? -1 : w == 3 ? 0 : 3 * (w >> 2) - 3 + (w & 3), nwi = 10;
  int bad = 0;
  __syncthreads();
  for (int p = 0; p <= np; ++p) {
    const int c0p = kP * p, k0 = c0p - kP, q0 = k0 - kP;  // panels p, p - 1, p - 2
    if ((w & 3) == 0 && p < np) {
      const int c = c0p + (w >> 2);
      if (p > 0 && c < nb) {
        ff v[2];
#pragma unroll
        for (int s = 0; s < 2; ++s) v[s] = D[(lane + 32 * s) * LD + c];
#pragma unroll
        for (int k = k0; k < k0 + kP; ++k) {
          const ff mc = D[c * LD + k];
#pragma unroll
          for (int s = 0; s < 2; ++s) v[s] -= D[(lane + 32 * s) * LD + k] * mc;
        }
#pragma unroll
        for (int s = 0; s < 2; ++s)
          if (lane + 32 * s >= c && lane + 32 * s < nb) D[(lane + 32 * s) * LD + c] = v[s];
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");  // (warps 0, 4, 8, 12)
      if (w == 0) {
        ff v[kP][2];
#pragma unroll
        for (int j = 0; j < kP; ++j)
#pragma unroll
          for (int s = 0; s < 2; ++s) v[j][s] = D[(lane + 32 * s) * LD + min(c0p + j, kLcNB - 1)];
        const bool upper = c0p < 32;  // the pivots' half of the rows
#pragma unroll
        for (int j = 0; j < kP; ++j) {
          const int cj = c0p + j;
          if (cj >= nb) break;
          const ff d = shfl_idx(upper ? v[j][0] : v[j][1], cj & 31);
          const bool ok = d > 0.0;
          const ff sd = ok ? sqrt(d) : ff(1.0);
          const ff rinv = ff(1.0) / sd;
          if (!ok && bad == 0) bad = c0 + cj + 1;
          ff x[2];
#pragma unroll
          for (int s = 0; s < 2; ++s) {
            const int i = lane + 32 * s;
            x[s] = ff(v[j][s] * rinv);
            if (i == cj) D[i * LD + cj] = sd;
            else if (i > cj && i < nb) D[i * LD + cj] = x[s];
          }
          if (lane == 0) srinv[cj] = rinv;
#pragma unroll
          for (int q = j + 1; q < kP; ++q) {
            const ff mc = shfl_idx(upper ? x[0] : x[1], (c0p + q) & 31);
#pragma unroll
            for (int s = 0; s < 2; ++s) v[q][s] -= x[s] * mc;
          }
        }
      }
    } else if (w == 1 || w == 2) {
      const int c = tid - 32;
      if (p > 0) {
        ff a[kP], y[kP];
#pragma unroll
        for (int j = 0; j < kP; ++j) a[j] = X[min(k0 + j, kLcNB - 1) * LD + c];
        if (p > 1)
#pragma unroll
          for (int k = q0; k < q0 + kP; ++k) {
            const ff x = X[k * LD + c];
            if (c <= k)
#pragma unroll
              for (int j = 0; j < kP; ++j) a[j] -= D[min(k0 + j, kLcNB - 1) * LD + k] * x;
          }
#pragma unroll
        for (int j = 0; j < kP; ++j) {
          if (k0 + j >= nb) break;
#pragma unroll
          for (int q = 0; q < j; ++q)
            if (c <= k0 + q) a[j] -= D[(k0 + j) * LD + k0 + q] * y[q];
          y[j] = ff(a[j] * srinv[k0 + j]);
          if (c <= k0 + j) X[(k0 + j) * LD + c] = y[j];
        }
      }
    } else if (wi >= 0) {
      if (p > 0)
        for (int c = c0p + kP + wi; c < nb; c += nwi)
          for (int i = (c & 32) + lane; i < nb; i += 32) {
            if (i < c) continue;
            ff v = D[i * LD + c];
#pragma unroll
            for (int k = k0; k < k0 + kP; ++k) v -= D[i * LD + k] * D[c * LD + k];
            D[i * LD + c] = v;
          }
      if (p > 1)
        for (int i = c0p + wi; i < nb; i += nwi)
          for (int c = lane; c < q0 + kP; c += 32) {
            ff v = X[i * LD + c];
#pragma unroll
            for (int k = q0; k < q0 + kP; ++k)
              if (c <= k) v -= D[i * LD + k] * X[k * LD + c];
            X[i * LD + c] = v;
          }
    }
    __syncthreads();
  }
  // L in the lower triangle of the diagonal block; the strictly lower part of X = D^{-1} in its
  // (otherwise unused) strictly upper triangle, X[i][c] at row c0 + c, column c0 + i, for the
  // block solves of k_leaf_tri_few and k_leaf_tri_wide (X's diagonal is 1 / D_ii, recomputed there the same way)
  for (int e = tid; e < nb * nb; e += NT) {
    const int i = e % nb, c = e / nb;
    if (i >= c) Lf[koff + (int64_t)(c0 + c) * m + c0 + i] = D[i * LD + c];
    else Lf[koff + (int64_t)(c0 + c) * m + c0 + i] = X[c * LD + i];
  }
  if (tid == 0 && bad != 0 && info[leaf] == 0) info[leaf] = bad;
  // rows of X: four threads per row, 16 columns each
  uint16_t* dst = xsl + leaf * (int64_t)(kSlices * kLcNB * kLcNB);
  for (int rr = tid >> 2; rr < kLcNB; rr += NT >> 2) {
    const int qq = tid & 3;
    float amax = 0.f;
    ff xv[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      xv[k] = X[rr * LD + 16 * qq + k];
      amax = fmaxf(amax, fabsf(xv[k].hi));
    }
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    const int e = tc::row_exponent(amax);
    if (qq == 0) xexp[leaf * kLcNB + rr] = e;
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      ff xg[8];
#pragma unroll
      for (int cc = 0; cc < 8; ++cc) xg[cc] = xv[8 * g + cc];
      store_slices8(dst, kLcNB, rr, 2 * qq + g, xg, e);
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Block column below the diagonal block: grid = (nleaf, row tiles), block = kLcTcThreads,
// dynamic shared memory kSlices x (kATileBytes + kBTileBytes).  Rows [128 rt, 128 rt + 128) of
// the rows below (trailing rows of K_j, then the r rows of Phi_j', then zero padding up to RP).
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kLcTcThreads, 1) k_lc_trsm(ff* __restrict__ Lf, ff* __restrict__ G, int r,
                                                             DTree t, int c0, const uint16_t* __restrict__ xsl,
                                                             const int* __restrict__ xexp,
                                                             uint16_t* __restrict__ slices, int* __restrict__ rexp,
                                                             int64_t slice_stride, int64_t exp_stride,
                                                             int* __restrict__ info) {
  extern __shared__ __align__(1024) unsigned char smraw[];
  constexpr int LD = kLcNB + 1;
  __shared__ __align__(8) uint64_t bar[2];
  __shared__ uint32_t tslot;
  __shared__ int serr;
  __shared__ int bexp[kLcNB];
  __shared__ int aexp[kLcTileM];
  const int64_t leaf = blockIdx.x;
  const int rt = blockIdx.y;
  const int m = d_leaf_size(t, leaf);
  if (c0 >= m) return;
  const int nb = min(kLcNB, m - c0);
  const int T = m - c0 - nb;
  const int R = T + r;
  const int64_t RP = lc_rows_padded(R);
  if ((int64_t)kLcTileM * rt >= RP) return;
  const int64_t koff = d_leaf_koff(t, leaf);
  const int64_t qoff = d_leaf_start(t, leaf) * r;
  uint16_t* sl = slices + leaf * slice_stride;
  int* ex = rexp + leaf * exp_stride;
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  uint16_t* sA = reinterpret_cast<uint16_t*>(smraw);
  uint16_t* sB = sA + kSlices * kATileBytes / 2;
  ff* Pst = reinterpret_cast<ff*>(smraw);  // after the products: P, kLcTileM x LD
  const uint32_t smA = tc::smem_u32(sA), smB = tc::smem_u32(sB);

  if (tid == 0) {
    tc::mbar_init(&bar[0], 1);
    tc::mbar_init(&bar[1], 1);
    tc::mbar_fence_init();
    serr = 0;
  }
  if (w == 0) {
    tc::tmem_alloc(&tslot, kLcTmemCols);
    tc::tmem_relinquish();
  }
  if (tid < kLcNB) bexp[tid] = xexp[leaf * kLcNB + tid];
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = tslot;
  if (tid == 0) {
    tc::mbar_arrive_expect_tx(&bar[0], kSlices * kBTileBytes);
    const uint16_t* xs = xsl + leaf * (int64_t)(kSlices * kLcNB * kLcNB);
    for (int s = 0; s < kSlices; ++s)
      tc::bulk_g2s(reinterpret_cast<unsigned char*>(sB) + s * kBTileBytes, xs + (int64_t)s * kLcNB * kLcNB,
                   kBTileBytes, &bar[0]);
  }
  // A slices: four threads per row, 16 columns each
  const int i4 = tid >> 2, qq = tid & 3;
  const int64_t rho4 = (int64_t)kLcTileM * rt + i4;
  const bool valid4 = rho4 < R;
  {
    ff a[16];
    float amax = 0.f;
#pragma unroll
    for (int cc = 0; cc < 16; ++cc) {
      const int c = 16 * qq + cc;
      ff v(0.0);
      if (valid4 && c < nb)
        v = rho4 < T ? Lf[koff + (int64_t)(c0 + c) * m + c0 + nb + rho4] : G[qoff + (rho4 - T) * m + c0 + c];
      a[cc] = v;
      amax = fmaxf(amax, fabsf(v.hi));
    }
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    const int e = tc::row_exponent(amax);
    if (qq == 0) aexp[i4] = e;
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      ff xg[8];
#pragma unroll
      for (int cc = 0; cc < 8; ++cc) xg[cc] = a[8 * g + cc];
      store_slices8(sA, kLcTileM, i4, 2 * qq + g, xg, e);
    }
  }
  tc::fence_proxy_async_smem();
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  if (tid == 0) {
    if (tc::mbar_wait(&bar[0], 0, kTcWaitLimit)) {
      tc::tc_fence_after();
      lc_issue_products(tmem, smA, smB);
    } else {
      serr = 1;
    }
    tc::mma_commit(&bar[1]);
  }
  __syncwarp();
  if (!tc::mbar_wait(&bar[1], 0, kTcWaitLimit)) atomicExch(&serr, 1);
  tc::tc_fence_after();
  __syncthreads();  // serr is the same in every thread from here on
  if (serr) {
    if (tid == 0) {  // copies and products still in flight finish before the exit
      tc::mbar_wait(&bar[0], 0, kTcWaitLimit);
      tc::mbar_wait(&bar[1], 0, kTcWaitLimit);
      info[leaf] = -1;
    }
  } else {
    // P = A X' into shared memory (over the A slices, which the products have read)
    const int q = w & 3, h = w >> 2;
    const int i = 32 * q + lane;
    const uint32_t tl = tmem + ((uint32_t)(32 * q) << 16);
#pragma unroll 1
    for (int cc = 0; cc < 2; ++cc) {
      const int j0 = 16 * h + 8 * cc;
      ff pv[8];
      lc_tile_values(tl, j0, aexp[i], bexp + j0, pv);
#pragma unroll
      for (int jj = 0; jj < 8; ++jj) Pst[i * LD + j0 + jj] = pv[jj];
    }
    __syncthreads();
    // P back to Lf / G, its row exponent and slices for the update step
    ff pv[16];
    float amax = 0.f;
#pragma unroll
    for (int cc = 0; cc < 16; ++cc) {
      const int c = 16 * qq + cc;
      const ff v = (valid4 && c < nb) ? Pst[i4 * LD + c] : ff(0.0);
      pv[cc] = v;
      amax = fmaxf(amax, fabsf(v.hi));
    }
    if (valid4) {
#pragma unroll
      for (int cc = 0; cc < 16; ++cc) {
        const int c = 16 * qq + cc;
        if (c < nb) {
          if (rho4 < T)
            Lf[koff + (int64_t)(c0 + c) * m + c0 + nb + rho4] = pv[cc];
          else
            G[qoff + (rho4 - T) * m + c0 + c] = pv[cc];
        }
      }
    }
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    const int e = tc::row_exponent(amax);
    if (qq == 0) ex[rho4] = e;
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      ff xg[8];
#pragma unroll
      for (int cc = 0; cc < 8; ++cc) xg[cc] = pv[8 * g + cc];
      store_slices8(sl, RP, rho4, 2 * qq + g, xg, e);
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (w == 0) tc::tmem_dealloc(tmem, kLcTmemCols);
}

// ---------------------------------------------------------------------------------------------
// Trailing update step: grid = (nleaf, row tiles, column tiles), block = kLcTcThreads.
// Shared memory: kSlices A slices (kATileBytes each), then kSlices B slices (kBTileBytes each).
// A thread updates 16 entries of C (tile row 32 (w % 4) + lane, columns 16 (w / 4) .. + 15),
// loading the first eight while the products run and the next eight one chunk ahead.
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kLcTcThreads, 1) k_lc_update(ff* __restrict__ Lf, ff* __restrict__ G, int r,
                                                               DTree t, int c0, const uint16_t* __restrict__ slices,
                                                               const int* __restrict__ rexp, int64_t slice_stride,
                                                               int64_t exp_stride, int* __restrict__ info) {
  extern __shared__ __align__(1024) unsigned char smraw[];
  __shared__ __align__(8) uint64_t bar[2];
  __shared__ uint32_t tslot;
  __shared__ int cexp[kLcTileN];
  __shared__ int serr;
  const int64_t leaf = blockIdx.x;
  const int rt = blockIdx.y, ct = blockIdx.z;
  const int m = d_leaf_size(t, leaf);
  if (c0 >= m) return;
  const int nb = min(kLcNB, m - c0);
  const int T = m - c0 - nb;
  const int R = T + r;
  if (T <= 0 || kLcTileM * rt >= R || kLcTileN * ct >= T) return;
  const int rlast = min(kLcTileM * rt + kLcTileM - 1, R - 1);
  if (rlast < T && rlast < kLcTileN * ct) return;  // tile strictly above the diagonal
  const int64_t RP = lc_rows_padded(R);
  const int64_t koff = d_leaf_koff(t, leaf);
  const int64_t qoff = d_leaf_start(t, leaf) * r;
  const uint16_t* sl = slices + leaf * slice_stride;
  const int* ex = rexp + leaf * exp_stride;
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const uint32_t smA = tc::smem_u32(smraw);
  const uint32_t smB = smA + kSlices * kATileBytes;

  if (tid == 0) {
    tc::mbar_init(&bar[0], 1);
    tc::mbar_init(&bar[1], 1);
    tc::mbar_fence_init();
    serr = 0;
  }
  if (w == 0) {
    tc::tmem_alloc(&tslot, kLcTmemCols);
    tc::tmem_relinquish();
  }
  if (tid < kLcTileN) {
    const int64_t j = (int64_t)kLcTileN * ct + tid;
    cexp[tid] = j < RP ? ex[j] : 0;
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = tslot;

  if (tid == 0) {
    tc::mbar_arrive_expect_tx(&bar[0], kSlices * (kATileBytes + kBTileBytes));
    for (int s = 0; s < kSlices; ++s) {
      tc::bulk_g2s(smraw + s * kATileBytes, sl + lc_slice_index(s, RP, (int64_t)kLcTileM * rt, 0), kATileBytes,
                   &bar[0]);
      tc::bulk_g2s(smraw + kSlices * kATileBytes + s * kBTileBytes,
                   sl + lc_slice_index(s, RP, (int64_t)kLcTileN * ct, 0), kBTileBytes, &bar[0]);
    }
  }
  const int q = w & 3, h = w >> 2;
  const int64_t rho = (int64_t)kLcTileM * rt + 32 * q + lane;
  const bool rvalid = rho < R;
  const int erow = rvalid ? ex[rho] : 0;
  auto c_index = [&](int j) -> int64_t {  // -1: not updated by this thread
    if (!rvalid || j >= T || (rho < T && rho < j)) return -1;
    return rho < T ? koff + (int64_t)(c0 + nb + j) * m + c0 + nb + rho : qoff + (rho - T) * m + c0 + nb + j;
  };
  auto c_load = [&](int64_t o) -> ff {
    if (o < 0) return ff(0.0);
    return rho < T ? Lf[o] : G[o];
  };
  ff cbuf[8];
#pragma unroll
  for (int jj = 0; jj < 8; ++jj) cbuf[jj] = c_load(c_index(kLcTileN * ct + 16 * h + jj));
  if (tid == 0) {
    if (tc::mbar_wait(&bar[0], 0, kTcWaitLimit)) {
      tc::tc_fence_after();
      lc_issue_products(tmem, smA, smB);
    } else {
      serr = 1;
    }
    tc::mma_commit(&bar[1]);
  }
  __syncwarp();
  if (!tc::mbar_wait(&bar[1], 0, kTcWaitLimit)) atomicExch(&serr, 1);
  tc::tc_fence_after();
  __syncthreads();  // serr is the same in every thread from here on
  if (serr) {
    if (tid == 0) {  // copies and products still in flight finish before the exit
      tc::mbar_wait(&bar[0], 0, kTcWaitLimit);
      tc::mbar_wait(&bar[1], 0, kTcWaitLimit);
      info[leaf] = -1;
    }
  } else {
    const uint32_t tl = tmem + ((uint32_t)(32 * q) << 16);
#pragma unroll 1
    for (int cc = 0; cc < 2; ++cc) {
      const int j0 = 16 * h + 8 * cc;
      ff nbuf[8];
#pragma unroll
      for (int jj = 0; jj < 8; ++jj) nbuf[jj] = cc == 0 ? c_load(c_index(kLcTileN * ct + j0 + 8 + jj)) : ff(0.0);
      ff v[8];
      lc_tile_values(tl, j0, erow, cexp + j0, v);
#pragma unroll
      for (int jj = 0; jj < 8; ++jj) {
        const int64_t o = c_index(kLcTileN * ct + j0 + jj);
        if (o < 0) continue;
        const ff out = cbuf[jj] - v[jj];
        if (rho < T)
          Lf[o] = out;
        else
          G[o] = out;
      }
#pragma unroll
      for (int jj = 0; jj < 8; ++jj) cbuf[jj] = nbuf[jj];
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (w == 0) tc::tmem_dealloc(tmem, kLcTmemCols);
}

// ---------------------------------------------------------------------------------------------
// Probe of the split product (C ABI: km_probe_tc_gemm): C = A B' for A 128 x 64 and B 64 x 64
// (row-major doubles).  mode 0: A and B hold integers |v| <= 128, used as the single slice;
// C is the tensor cores' fp32 sum.  mode 1: the float-pair split product of arbitrary values.
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kLcProbeThreads, 1) k_tc_probe(const double* __restrict__ A,
                                                                 const double* __restrict__ B, int mode,
                                                                 double* __restrict__ C, int* __restrict__ status) {
  extern __shared__ __align__(1024) unsigned char smraw[];
  __shared__ __align__(8) uint64_t bar;
  __shared__ uint32_t tslot;
  __shared__ int rexp[kLcTileM + kLcTileN];
  __shared__ int serr;
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  uint16_t* sA = reinterpret_cast<uint16_t*>(smraw);
  uint16_t* sB = sA + kSlices * kATileBytes / 2;
  if (tid == 0) {
    tc::mbar_init(&bar, 1);
    tc::mbar_fence_init();
    serr = 0;
  }
  if (w == 0) {
    tc::tmem_alloc(&tslot, kLcTmemCols);
    tc::tmem_relinquish();
  }
  if (tid < kLcTileM + kLcTileN) {
    const bool isA = tid < kLcTileM;
    const int row = isA ? tid : tid - kLcTileM;
    const double* src = isA ? A + row * kLcNB : B + row * kLcNB;
    uint16_t* dst = isA ? sA : sB;
    const int64_t rp = isA ? kLcTileM : kLcTileN;
    float amax = 0.f;
    for (int c = 0; c < kLcNB; ++c) amax = fmaxf(amax, fabsf((float)src[c]));
    const int e = mode == 0 ? 7 : tc::row_exponent(amax);  // mode 0: v = t 2^-7 2^7 = t
    rexp[tid] = e;
    for (int kc = 0; kc < kLcNB / 8; ++kc) {
      ff x[8];
      for (int cc = 0; cc < 8; ++cc) x[cc] = ff(src[8 * kc + cc]);
      store_slices8(dst, rp, row, kc, x, e);
    }
  }
  tc::fence_proxy_async_smem();
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = tslot;
  const uint32_t smA = tc::smem_u32(sA), smB = tc::smem_u32(sB);
  if (tid == 0) {
    if (mode == 0) {
      constexpr uint32_t idesc = tc::idesc_bf16(kLcTileM, kLcTileN);
      for (int ks = 0; ks < kLcNB / 16; ++ks)
        tc::mma_bf16(tmem, tc::smem_desc(smA + ks * 256, 128, 1024), tc::smem_desc(smB + ks * 256, 128, 1024),
                     idesc, ks > 0);
    } else {
      lc_issue_products(tmem, smA, smB);
    }
    tc::mma_commit(&bar);
  }
  __syncwarp();
  if (!tc::mbar_wait(&bar, 0, kTcWaitLimit)) atomicExch(&serr, 1);
  tc::tc_fence_after();
  __syncthreads();  // serr is the same in every thread from here on
  if (serr) {
    if (tid == 0) status[0] = 1;
  } else {
    const int q = w & 3, h = w >> 2;
    const int row = 32 * q + lane;
    const uint32_t tl = tmem + ((uint32_t)(32 * q) << 16);
    for (int cc = 0; cc < 4; ++cc) {
      const int j0 = 32 * h + 8 * cc;
      float s[kSlices][8];
#pragma unroll
      for (int d = 0; d < kSlices; ++d) tc::tmem_ld8(tl + d * kLcTileN + j0, s[d]);
      tc::tmem_wait_ld();
#pragma unroll
      for (int jj = 0; jj < 8; ++jj) {
        double out;
        if (mode == 0) {
          out = (double)s[0][jj];
        } else {
          float sd[kSlices];
#pragma unroll
          for (int d = 0; d < kSlices; ++d) sd[d] = s[d][jj];
          out = (double)tc::ff_ldexp(tc::combine_diagonals(sd), rexp[row] + rexp[kLcTileM + j0 + jj]);
        }
        C[row * kLcTileN + j0 + jj] = out;
      }
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (w == 0) tc::tmem_dealloc(tmem, kLcTmemCols);
}

// ---------------------------------------------------------------------------------------------
// launchers: step p covers columns [64 p, 64 p + 64) of every leaf; the update of step p exists
// when some leaf has rows left after the block
// ---------------------------------------------------------------------------------------------
static int64_t lc_rp_max(const Tree& t, int r) { return lc_rows_padded(t.max_leaf + r); }

// ---------------------------------------------------------------------------------------------
// Leaf triangular solves with the factor of the tensor-core stage: L x = b (op 0) or L' x = b
// (op 1) by 64-row blocks, x_q = X_q (b_q - L_q,<q x_<q) with X_q the inverse of diagonal block q
// kept by k_lc_diag (strictly lower part in the block's upper triangle, diagonal 1 / D_ii), so
// that both steps are block products spread over all threads: no sequential chain over rows
// (the substitution of k_leaf_tri runs one warp per column through each block).  After x_q the
// remaining rows are updated at once (right-looking).  Same arithmetic as the TC stage's own
// block column products, which use the same inverses.
//
// Few columns, 4 a CTA: reading L bounds it.  Thread (row i of a 64 x 64 tile, part g) multiplies the
// tile's columns g, g + 4, ...; a tile that lies along the rows in memory goes from memory to the
// registers of these threads, one that lies across goes through shared memory, and the next tile is on
// its way meanwhile.  The four parts are added in shared memory.  With four loads in flight a thread, row
// by row, 256 leaves of 256 took 230 us for 16 columns, now 146; 512 leaves of 256 100 us for one, now 50.
// grid (nleaf, ceil(k / 4)), block 256.
// ---------------------------------------------------------------------------------------------
constexpr int kTfCols = 4, kTwLd = kLcNB + 1;

// x of 64-row block q by substitution in place of the product with its inverse (kIllBlock, km_kernels.h): a warp per
// column (column c at xs[c mp]), rows lane and lane + 32, L's block through T (64 x 65), the diagonal as
// reciprocals.  Called by all 256 threads; begins and ends with a barrier.
__device__ __noinline__ void block_subst_ff(const ff* L, ff* T, ff* xs, int m, int mp, int q, int nc, int op) {
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, fast = tid & 63;
  const int i0 = kLcNB * q, nb = min(kLcNB, m - i0);
  __syncthreads();
  for (int sl = tid >> 6; sl < kLcNB; sl += 4)
    if (sl <= fast && fast < nb) {
      const ff v = L[(int64_t)(i0 + sl) * m + i0 + fast];
      T[sl * kTwLd + fast] = sl == fast ? ff(1.0) / v : v;
    }
  __syncthreads();
  // columns w and w + 8 together: two independent chains (at most 16 columns)
  if (w < nc) {
    const bool two = w + 8 < nc;
    ff* x[2] = {xs + w * mp + i0, xs + (two ? w + 8 : w) * mp + i0};
    acc_t<ff> v[2][2];
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int s = 0; s < 2; ++s) v[c][s] = x[c][lane + 32 * s];
    for (int u = 0; u < nb; ++u) {
      const int l = op == 0 ? u : nb - 1 - u;
      const ff inv = T[l * kTwLd + l];
      ff xl[2];
#pragma unroll
      for (int c = 0; c < 2; ++c)
        if (c == 0 || two) xl[c] = shfl_idx(accv(l < 32 ? v[c][0] : v[c][1]) * inv, l & 31);
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int i = lane + 32 * s;
        if (i == l) {
          v[0][s] = xl[0];
          v[1][s] = xl[1];
        } else if (op == 0 ? (i > l && i < nb) : i < l) {
          const ff a = op == 0 ? T[l * kTwLd + i] : T[i * kTwLd + l];
          v[0][s] -= a * xl[0];
          if (two) v[1][s] -= a * xl[1];
        }
      }
    }
#pragma unroll
    for (int s = 0; s < 2; ++s)
      if (lane + 32 * s < nb) {
        x[0][lane + 32 * s] = accv(v[0][s]);
        if (two) x[1][lane + 32 * s] = accv(v[1][s]);
      }
  }
  __syncthreads();
}

// CHECK: diagonal blocks with an ill-conditioned inverse are substituted (kIllBlock, km_kernels.h)
template <bool CHECK>
__global__ void __launch_bounds__(256, 3) k_leaf_tri_few(const ff* __restrict__ Lf, DTree t, int op, ff* __restrict__ X,
                                                      int64_t ldx, int k) {
  extern __shared__ __align__(16) unsigned char lc_smem_s[];
  const int64_t leaf = blockIdx.x;
  const int m = d_leaf_size(t, leaf), nbk = (m + kLcNB - 1) / kLcNB, mp = nbk * kLcNB;
  const int64_t s = d_leaf_start(t, leaf);
  const ff* L = Lf + d_leaf_koff(t, leaf);
  const int c0 = blockIdx.y * kTfCols, nc = min(kTfCols, k - c0);
  const int tid = threadIdx.x, fast = tid & 63, g = tid >> 6;
  ff* xs = reinterpret_cast<ff*>(lc_smem_s);  // kTfCols x mp, column c at xs[c mp], zero below row m
  ff* red = xs + kTfCols * mp;                // part, column, row: 4 x kTfCols x 64
  ff* T = red + 4 * kTfCols * kLcNB;          // 64 x 65, element (l, row) at T[l kTwLd + row]
  for (int c = 0; c < nc; ++c)
    for (int i = tid; i < mp; i += 256) xs[c * mp + i] = i < m ? X[(int64_t)(c0 + c) * ldx + s + i] : ff(0.0);
  // tile (block q, rows of block b): L[b rows][q columns] (op 0) or its transpose, b == q: the inverse.
  // In memory L runs along the rows, the inverse (upper triangle) across, for op 1 the other way round.
  ff pre[16];
  auto fetch = [&](int q, int b) {
    const bool across = (b == q) == (op == 0);
    const int col0 = kLcNB * (across ? b : q) + g, row = kLcNB * (across ? q : b) + fast;
    const int cols = row < m ? m - col0 : 0;  // columns col0, col0 + 4, ... below this many
    const ff* p = L + (int64_t)col0 * m + row;
#pragma unroll
    for (int u = 0; u < 16; ++u, p += 4 * m) pre[u] = 4 * u < cols ? *p : ff(0.0);
  };
  const float ill = kIllBlock / L[0].hi;
  fetch(op == 0 ? 0 : nbk - 1, op == 0 ? 0 : nbk - 1);
  __syncthreads();
  for (int step = 0; step < nbk; ++step) {
    const int q = op == 0 ? step : nbk - 1 - step, left = nbk - step;
    for (int v = 0; v < left; ++v) {
      const int b = op == 0 ? q + v : q - v;
      ff cur[16];  // columns g + 4 u of row `fast` of the tile
      bool above = false;
#pragma unroll
      for (int u = 0; u < 16; ++u) cur[u] = pre[u];
      if (v == 0) {  // a triangle, its diagonal the reciprocal (fast <= column or row g + 4 u)
        ff d(1.f, 0.f);
#pragma unroll
        for (int u = 0; u < 16; ++u)
          if (fast == g + 4 * u && kLcNB * q + fast < m) d = cur[u];
        d = ff(1.0) / d;
#pragma unroll
        for (int u = 0; u < 16; ++u) {
          cur[u] = fast < g + 4 * u ? cur[u] : fast == g + 4 * u ? d : ff(0.0);
          if (CHECK) above |= !(fabsf(cur[u].hi) <= ill) && kLcNB * q + fast < m;  // (one in rows beyond the leaf)
        }
      }
      bool by_rows = false;
      if ((v == 0) == (op == 0)) {
#pragma unroll
        for (int u = 0; u < 16; ++u) T[fast * kTwLd + g + 4 * u] = cur[u];
        if (CHECK) by_rows = __syncthreads_or(above);
        else __syncthreads();
#pragma unroll
        for (int u = 0; u < 16; ++u) cur[u] = T[(g + 4 * u) * kTwLd + fast];
      } else if (CHECK && v == 0) {
        by_rows = __syncthreads_or(above);
      }
      if (v + 1 < left) fetch(q, op == 0 ? b + 1 : b - 1);
      else if (left > 1) fetch(op == 0 ? q + 1 : q - 1, op == 0 ? q + 1 : q - 1);
      if (CHECK && by_rows) {
        block_subst_ff(L, T, xs, m, mp, q, nc, op);
        continue;
      }
      for (int c = 0; c < nc; ++c) {
        const ff* x = xs + c * mp + kLcNB * q + g;
        acc_t<ff> a{};
#pragma unroll
        for (int u = 0; u < 16; ++u) a += cur[u] * x[4 * u];
        red[(g * kTfCols + c) * kLcNB + fast] = accv(a);
      }
      __syncthreads();
      if (g < nc) {
        const ff* p = red + g * kLcNB + fast;
        constexpr int sp = kTfCols * kLcNB;
        const ff sum = (p[0] + p[sp]) + (p[2 * sp] + p[3 * sp]);
        ff* out = xs + g * mp + kLcNB * b + fast;
        *out = v == 0 ? sum : *out - sum;
      }
      __syncthreads();
    }
  }
  for (int c = 0; c < nc; ++c)
    for (int i = tid; i < m; i += 256) X[(int64_t)(c0 + c) * ldx + s + i] = xs[c * mp + i];
}

// The same solves for many right-hand sides, 12 columns a CTA: 64 x 64 tiles of L (or L'), and of the
// diagonal blocks' inverses, go through shared memory, and the next tile is on its way from memory
// while the present one is multiplied.  Thread (row 32 (w & 1) + lane, columns 3 (w >> 1) .. + 2): per
// two rows of x five loads from shared memory feed six multiply-adds, so that the FP32 pipe bounds the
// kernel (12 instructions a multiply-add).  512 leaves of 488, 72 columns: the substitution of
// k_leaf_tri took 4.4 ms, this 2.6 ms; the FP32 floor is 1.5 ms.  The chunks of a leaf are neighbours in
// the grid and find its tiles in L2.  A diagonal block with an ill-conditioned inverse is substituted
// (kIllBlock, km_kernels.h).  grid nleaf ceil(k / 12), block 256.
constexpr int kTwCols = 12;

__global__ void __launch_bounds__(256, 2) k_leaf_tri_wide(const ff* __restrict__ Lf, DTree t, int op, ff* __restrict__ X,
                                                          int64_t ldx, int k) {
  extern __shared__ __align__(16) unsigned char lc_smem_w[];
  struct __align__(16) pair {
    ff a, b;
  };
  const int nch = (k + kTwCols - 1) / kTwCols;
  const int64_t leaf = blockIdx.x / nch;
  const int c0 = (int)(blockIdx.x % nch) * kTwCols, nc = min(kTwCols, k - c0);
  const int m = d_leaf_size(t, leaf), mp = (m + kLcNB - 1) & ~(kLcNB - 1);
  const int64_t s = d_leaf_start(t, leaf);
  const ff* L = Lf + d_leaf_koff(t, leaf);
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  ff* xs = reinterpret_cast<ff*>(lc_smem_w);  // kTwCols x mp, column c at xs[c mp], zero below row m
  ff* T = xs + kTwCols * mp;                  // 64 x 65, element (l, row) at T[l kTwLd + row]
  for (int c = w; c < kTwCols; c += 8)
    for (int i = lane; i < mp; i += 32) xs[c * mp + i] = c < nc && i < m ? X[(int64_t)(c0 + c) * ldx + s + i] : ff(0.0);
  const int nbk = mp / kLcNB;
  ff pre[16];
  // tile (block q, rows of block b): L[b rows][q columns] (op 0) or its transpose, b == q: the inverse.
  // In memory L runs along the rows, the inverse (upper triangle) across, for op 1 the other way round.
  const int fast = tid & 63, slow = tid >> 6;
  auto fetch = [&](int q, int b) {
    const bool across = (b == q) == (op == 0);
    const int col0 = kLcNB * (across ? b : q) + slow, row = kLcNB * (across ? q : b) + fast;
    const int cols = row < m ? m - col0 : 0;  // columns col0, col0 + 4, ... below this many
    const ff* p = L + (int64_t)col0 * m + row;
#pragma unroll
    for (int u = 0; u < 16; ++u, p += 4 * m) pre[u] = 4 * u < cols ? *p : ff(0.0);
  };
  // true if a thread's part of the inverse has an entry above kIllBlock / L[0][0]
  const float ill = kIllBlock / L[0].hi;
  auto put = [&](int q, int b) {
    const bool across = (b == q) == (op == 0);
    bool above = false;
    if (b == q) {
      ff d(1.f, 0.f);
#pragma unroll
      for (int u = 0; u < 16; ++u)
        if (fast == slow + 4 * u && kLcNB * q + fast < m) d = pre[u];
      d = ff(1.0) / d;
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        const int sl = slow + 4 * u;  // kept: l <= i (op 0) or l >= i (op 1), fast <= sl for both
        const ff v = fast < sl ? pre[u] : fast == sl ? d : ff(0.0);
        above |= !(fabsf(v.hi) <= ill) && kLcNB * q + fast < m;  // (one in rows beyond the leaf)
        T[across ? fast * kTwLd + sl : sl * kTwLd + fast] = v;
      }
    } else {
      ff* to = across ? T + fast * kTwLd + slow : T + slow * kTwLd + fast;
      const int step = across ? 4 : 4 * kTwLd;
#pragma unroll
      for (int u = 0; u < 16; ++u) to[u * step] = pre[u];
    }
    return above;
  };
  const int i = 32 * (w & 1) + lane;
  ff* xc = xs + 3 * (w >> 1) * mp;
  fetch(op == 0 ? 0 : nbk - 1, op == 0 ? 0 : nbk - 1);
  for (int step = 0; step < nbk; ++step) {
    const int q = op == 0 ? step : nbk - 1 - step, left = nbk - step;
    for (int v = 0; v < left; ++v) {
      const int b = op == 0 ? q + v : q - v;
      __syncthreads();
      const bool by_rows = __syncthreads_or(put(q, b));
      if (v + 1 < left) fetch(q, op == 0 ? b + 1 : b - 1);
      else if (left > 1) fetch(op == 0 ? q + 1 : q - 1, op == 0 ? q + 1 : q - 1);
      if (by_rows) {  // (a diagonal block)
        block_subst_ff(L, T, xs, m, mp, q, nc, op);
        continue;
      }
      acc_t<ff> a[3] = {};
      // the inverse is a triangle: 32 of its rows need half of the tile
      const int l0 = v == 0 && op == 1 ? 32 * (w & 1) : 0;
      // (nothing beyond the leaf: columns in pairs, rows by warps)
      const bool live = kLcNB * b + 32 * (w & 1) < m;
      const int l1 = live ? min(v == 0 && op == 0 ? 32 * (w & 1) + 32 : kLcNB, (m - kLcNB * q + 1) & ~1) : 0;
      const ff* x = xc + kLcNB * q;
#pragma unroll 4
      for (int l = l0; l < l1; l += 2) {
        const ff t0 = T[l * kTwLd + i], t1 = T[(l + 1) * kTwLd + i];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const pair y = *reinterpret_cast<const pair*>(x + c * mp + l);
          a[c] += t0 * y.a;
          a[c] += t1 * y.b;
        }
      }
      if (v == 0) __syncthreads();
      ff* out = xc + kLcNB * b + i;
      if (live)
#pragma unroll
        for (int c = 0; c < 3; ++c) out[c * mp] = v == 0 ? accv(a[c]) : out[c * mp] - accv(a[c]);
    }
  }
  __syncthreads();
  for (int c = w; c < nc; c += 8)
    for (int j = lane; j < m; j += 32) X[(int64_t)(c0 + c) * ldx + s + j] = xs[c * mp + j];
}

bool launch_leaf_tri_blk(const ff* Lf, const Tree& t, int op, ff* X, int64_t ldx, int k, cudaStream_t st) {
  if (k <= 0) return true;
  if (t.max_leaf > kLcMaxLeaf || (op != 0 && op != 1)) return false;
  const int64_t nb = (t.max_leaf + kLcNB - 1) / kLcNB, mp = nb * kLcNB, few = (k + kTfCols - 1) / kTfCols;
  // Many leaves whose triangle fills little of its tiles, up to 37 points and 65 and 66: the substitution (16
  // columns, a backward call: 4096 leaves of 16 0.44 ms, by tiles 0.63; 2048 of 65 0.75 against 0.93).  With few
  // CTAs the tiles are faster (32 of 65, 100 columns: 0.15 against 0.17 ms).
  if (t.max_leaf * (t.max_leaf + 1) * 100 < 18 * kLcNB * kLcNB * nb * (nb + 1) && t.nleaf * few > 8 * 152)
    return launch_leaf_tri<ff>(Lf, t, op, X, 1, t.n, 0, X, 1, t.n, 0, k, st);
  // 12 columns a CTA take as long as 2.1 chunks of 4 columns (256 leaves of 256: 81 us against 31, 50, 90,
  // 124 us for 1, 4, 8, 12 columns; 16 columns 155 against 146, 24 columns 156 against 220), unless the SMs
  // hold all chunks of 4 at once (one leaf of 1024, 33 columns: the call 634 us against 424)
  if (2 * ((k + kTwCols - 1) / kTwCols) >= few || t.nleaf * few <= 152) {
    const size_t sm = ((size_t)kTfCols * mp + (size_t)4 * kTfCols * kLcNB + (size_t)kLcNB * kTwLd) * sizeof(ff);
    const dim3 grid((unsigned)t.nleaf, (unsigned)few);
    // (from 32 columns on the substitution has been the rule: none of its accuracy is given up)
    if (k < 32) {
      smem_limit((const void*)k_leaf_tri_few<false>, sm);
      k_leaf_tri_few<false><<<grid, 256, sm, st>>>(Lf, dtree(t), op, X, ldx, k);
    } else {
      smem_limit((const void*)k_leaf_tri_few<true>, sm);
      k_leaf_tri_few<true><<<grid, 256, sm, st>>>(Lf, dtree(t), op, X, ldx, k);
    }
    return true;
  }
  const size_t sm = ((size_t)kTwCols * mp + (size_t)kLcNB * kTwLd) * sizeof(ff);
  smem_limit((const void*)k_leaf_tri_wide, sm);
  k_leaf_tri_wide<<<(unsigned)(t.nleaf * ((k + kTwCols - 1) / kTwCols)), 256, sm, st>>>(Lf, dtree(t), op, X, ldx, k);
  return true;
}

bool leaf_chol_tc_supported(const Tree& t, int r) {
  return t.max_leaf >= 1 && t.max_leaf <= kLcMaxLeaf && r >= 1 && r <= kLcMaxRank;
}

// Scratch per leaf: the slices of the rows below the block (kSlices x RP x 64 bf16) and of X
// (kSlices x 64 x 64 bf16), then the row exponents of both.
int64_t leaf_chol_tc_scratch_bytes(const Tree& t, int r) {
  const int64_t rp = lc_rp_max(t, r);
  return t.nleaf * ((rp * kLcNB + (int64_t)kLcNB * kLcNB) * kSlices * (int64_t)sizeof(uint16_t) +
                    (rp + kLcNB) * (int64_t)sizeof(int));
}

int leaf_chol_tc_steps(const Tree& t) { return (int)((t.max_leaf + kLcNB - 1) / kLcNB); }

bool leaf_chol_tc_has_update(const Tree& t, int p) { return t.max_leaf - (int64_t)kLcNB * (p + 1) > 0; }

struct LcArgs {
  uint16_t* slices;
  uint16_t* xsl;
  int* rexp;
  int* xexp;
  int64_t slice_stride, exp_stride;
};

static LcArgs lc_args(const Tree& t, int r, void* scratch) {
  const int64_t rp = lc_rp_max(t, r);
  LcArgs a;
  a.slice_stride = rp * kLcNB * kSlices;
  a.exp_stride = rp;
  a.slices = reinterpret_cast<uint16_t*>(scratch);
  a.xsl = a.slices + t.nleaf * a.slice_stride;
  a.rexp = reinterpret_cast<int*>(a.xsl + t.nleaf * (int64_t)kSlices * kLcNB * kLcNB);
  a.xexp = a.rexp + t.nleaf * rp;
  return a;
}

void launch_leaf_chol_tc_diag(ff* Lf, int r, const Tree& t, int p, void* scratch, int* info, cudaStream_t st) {
  const LcArgs a = lc_args(t, r, scratch);
  const size_t smd = (size_t)2 * kLcNB * (kLcNB + 1) * sizeof(ff);
  smem_limit((const void*)k_lc_diag, smd);
  k_lc_diag<<<(unsigned)t.nleaf, kLcDiagThreads, smd, st>>>(Lf, dtree(t), kLcNB * p, a.xsl, a.xexp, info);
}

void launch_leaf_chol_tc_trsm(ff* Lf, ff* G, int r, const Tree& t, int p, void* scratch, int* info,
                              cudaStream_t st) {
  const LcArgs a = lc_args(t, r, scratch);
  const int c0 = kLcNB * p;
  const size_t sm = (size_t)kSlices * (kATileBytes + kBTileBytes);
  smem_limit((const void*)k_lc_trsm, sm);
  const int64_t rmax = t.max_leaf - c0 - 1 + r;  // rows below the block of the largest leaf, nb >= 1
  dim3 grid((unsigned)t.nleaf, (unsigned)((rmax + kLcTileM - 1) / kLcTileM));
  k_lc_trsm<<<grid, kLcTcThreads, sm, st>>>(Lf, G, r, dtree(t), c0, a.xsl, a.xexp, a.slices, a.rexp, a.slice_stride,
                                            a.exp_stride, info);
}

void launch_leaf_chol_tc_update(ff* Lf, ff* G, int r, const Tree& t, int p, void* scratch, int* info,
                                cudaStream_t st) {
  const LcArgs a = lc_args(t, r, scratch);
  const size_t sm = (size_t)kSlices * (kATileBytes + kBTileBytes);
  const int c0 = kLcNB * p;
  const int64_t tmax = t.max_leaf - c0 - kLcNB;
  if (tmax <= 0) return;
  dim3 grid((unsigned)t.nleaf, (unsigned)((tmax + r + kLcTileM - 1) / kLcTileM),
            (unsigned)((tmax + kLcTileN - 1) / kLcTileN));
  smem_limit((const void*)k_lc_update, sm);
  k_lc_update<<<grid, kLcTcThreads, sm, st>>>(Lf, G, r, dtree(t), c0, a.slices, a.rexp, a.slice_stride,
                                              a.exp_stride, info);
}

}  // namespace km

extern "C" int km_probe_tc_gemm(int device, const double* A, const double* B, int mode, double* C) {
  using namespace km;
  if (!A || !B || !C || (mode != 0 && mode != 1)) return KM_ERR_BAD_ARG;
  if (cudaSetDevice(device) != cudaSuccess) return KM_ERR_CUDA;
  double *dA = nullptr, *dB = nullptr, *dC = nullptr;
  int* dst = nullptr;
  const size_t na = (size_t)kLcTileM * kLcNB, nbb = (size_t)kLcTileN * kLcNB, nc = (size_t)kLcTileM * kLcTileN;
  int rc = KM_OK;
  if (cudaMalloc(&dA, na * 8) != cudaSuccess || cudaMalloc(&dB, nbb * 8) != cudaSuccess ||
      cudaMalloc(&dC, nc * 8) != cudaSuccess || cudaMalloc(&dst, sizeof(int)) != cudaSuccess) {
    rc = KM_ERR_OOM;
  } else {
    cudaMemcpy(dA, A, na * 8, cudaMemcpyHostToDevice);
    cudaMemcpy(dB, B, nbb * 8, cudaMemcpyHostToDevice);
    cudaMemset(dst, 0, sizeof(int));
    const size_t smu = (size_t)kSlices * (kATileBytes + kBTileBytes);
    smem_limit((const void*)k_tc_probe, smu);
    k_tc_probe<<<1, kLcProbeThreads, smu>>>(dA, dB, mode, dC, dst);
    int stv = 0;
    if (cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess) {
      rc = KM_ERR_CUDA;
    } else {
      cudaMemcpy(&stv, dst, sizeof(int), cudaMemcpyDeviceToHost);
      cudaMemcpy(C, dC, nc * 8, cudaMemcpyDeviceToHost);
      if (stv) rc = KM_ERR_TIMEOUT;
    }
  }
  cudaFree(dA);
  cudaFree(dB);
  cudaFree(dC);
  cudaFree(dst);
  return rc;
}
