// Leaf-level kernels: triangular solves/products with the leaf Cholesky factors and the
// projections Q_leaf' y / expansions Q_leaf g through the leaf Householder reflectors.
//
// These replace the blockwise loops ldiv!/mul!(BDiagonal(leafW), .) of the reference
// (src/HODLR/src/BlockDiagonal.jl:51-70, used by src/HODLR/src/utils.jl:54-65 and
// src/HODLR/src/baseoverloads.jl:95-150).  One CTA handles one leaf and a chunk of right-hand
// sides staged in shared memory; the triangular solves are blocked by 32 rows so that the
// dependency chain is a 32-step shuffle solve per block and the bulk of the work is an
// independent multiply-add update (FP64 throughput bound).
#include <algorithm>
#include <type_traits>

#include "km_kernels.h"

namespace km {

// ---------------------------------------------------------------------------------------------
// Blocked leaf triangular kernels, L lower triangular (column-major m x m):
//   op 0: X = L^{-1} B   op 1: X = L^{-T} B   op 2: X = L B   op 3: X = L^T B
// grid = (nleaf, ceil(ncols / NC)), block = 256.
// ---------------------------------------------------------------------------------------------
template <typename T, int NC>
__device__ void leaf_tri_body(const T* __restrict__ L, int m, int op, const T* Bp, int64_t ldb, T* Xp,
                              int64_t ldx, int nc, T* sm) {
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  T* xs = sm;                   // NC x m  (column c at xs[c*m])
  T* ys = xs + NC * m;          // NC x m  (products only)
  T* D = ys + ((op >= 2) ? NC * m : 0);  // 32 x 33
  for (int e = tid; e < NC * m; e += blockDim.x) {
    const int c = e / m, i = e % m;
    xs[e] = (c < nc) ? Bp[(int64_t)c * ldb + i] : T(0.0);
  }
  __syncthreads();
  if (op == 0 || op == 1) {
    const int nblk = (m + 31) / 32;
    for (int q = 0; q < nblk; ++q) {
      const int i0 = (op == 0) ? q * 32 : (nblk - 1 - q) * 32;
      const int ib = min(32, m - i0);
      for (int e = tid; e < 32 * 32; e += blockDim.x) {
        const int i = e & 31, l = e >> 5;
        if (i < ib && l <= i) {
          const T v = L[(int64_t)(i0 + l) * m + i0 + i];
          D[i * 33 + l] = (l == i) ? T(1.0) / v : v;  // diagonal kept as its reciprocal
        }
      }
      __syncthreads();
      // diagonal block, one warp per column, lanes = rows of the block
      for (int c = w; c < nc; c += 8) {
        acc_t<T> xa = (lane < ib) ? xs[c * m + i0 + lane] : T(0.0);  // row `lane`, updates pending
        T x = T(0.0);                                                  // row `lane`, solved
        if (op == 0) {
          for (int l = 0; l < ib; ++l) {
            if (lane == l) x = accv(xa) * D[l * 33 + l];
            const T xl = shfl_idx(x, l);
            if (lane > l && lane < ib) xa -= D[lane * 33 + l] * xl;
          }
        } else {
          for (int l = ib - 1; l >= 0; --l) {
            if (lane == l) x = accv(xa) * D[l * 33 + l];
            const T xl = shfl_idx(x, l);
            if (lane < l) xa -= D[l * 33 + lane] * xl;
          }
        }
        if (lane < ib) xs[c * m + i0 + lane] = x;
      }
      __syncthreads();
      // update of the remaining rows with the solved block: items of (row, 4 columns), so that
      // each loaded L entry feeds 4 multiply-adds and all threads stay busy as the remaining
      // rows shrink
      const int R = (op == 0) ? m - (i0 + ib) : i0;
      const int r0 = (op == 0) ? i0 + ib : 0;
      const int ng = (nc + 3) >> 2;
      for (int e = tid; e < R * ng; e += blockDim.x) {
        const int g = e / R, i = r0 + (e - g * R), cb = 4 * g;
        const T* xc = xs + cb * m + i0;
        acc_t<T> acc[4] = {};
        auto ld = [&](int l) {
          return (op == 0) ? L[(int64_t)(i0 + l) * m + i]   // L[i, i0 + l]
                           : L[(int64_t)i * m + i0 + l];    // L[i0 + l, i]
        };
        int l = 0;
        for (; l + 3 < ib; l += 4) {  // four entries loaded ahead of their multiply-adds
          const T a0 = ld(l), a1 = ld(l + 1), a2 = ld(l + 2), a3 = ld(l + 3);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (cb + j < nc) {
              acc[j] += a0 * xc[j * m + l];
              acc[j] += a1 * xc[j * m + l + 1];
              acc[j] += a2 * xc[j * m + l + 2];
              acc[j] += a3 * xc[j * m + l + 3];
            }
        }
        for (; l < ib; ++l) {
          const T a = ld(l);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (cb + j < nc) acc[j] += a * xc[j * m + l];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (cb + j < nc) xs[(cb + j) * m + i] -= accv(acc[j]);
      }
      __syncthreads();
    }
    for (int e = tid; e < nc * m; e += blockDim.x) {
      const int c = e / m, i = e % m;
      Xp[(int64_t)c * ldx + i] = xs[e];
    }
  } else {
    for (int i = tid; i < m; i += blockDim.x) {
      acc_t<T> acc[NC] = {};
      if (op == 2) {  // row i of L: L[i, l], l <= i
        for (int l = 0; l <= i; ++l) {
          const T a = L[(int64_t)l * m + i];
#pragma unroll
          for (int c = 0; c < NC; ++c) acc[c] += a * xs[c * m + l];
        }
      } else {        // row i of L^T = column i of L, rows l >= i
        const T* col = L + (int64_t)i * m;
        for (int l = i; l < m; ++l) {
          const T a = col[l];
#pragma unroll
          for (int c = 0; c < NC; ++c) acc[c] += a * xs[c * m + l];
        }
      }
#pragma unroll
      for (int c = 0; c < NC; ++c) ys[c * m + i] = accv(acc[c]);
    }
    __syncthreads();
    for (int e = tid; e < nc * m; e += blockDim.x) {
      const int c = e / m, i = e % m;
      Xp[(int64_t)c * ldx + i] = ys[e];
    }
  }
}

template <typename T, int NC>
__global__ void __launch_bounds__(256) k_leaf_tri(const T* __restrict__ Lf, DTree t, int op,
                                                  LeafOperand B, LeafOperand X, int ncols) {
  extern __shared__ __align__(16) unsigned char smraw[];
  T* sm = reinterpret_cast<T*>(smraw);
  const int64_t leaf = blockIdx.x;
  const int m = d_leaf_size(t, leaf);
  const int64_t s = d_leaf_start(t, leaf);
  const int c0 = blockIdx.y * NC;
  const int nc = min(NC, ncols - c0);
  const int64_t ldb = B.ld_is_m ? m : B.ld, ldx = X.ld_is_m ? m : X.ld;
  leaf_tri_body<T, NC>(Lf + d_leaf_koff(t, leaf), m, op,
                       reinterpret_cast<const T*>(B.ptr) + s * B.bmul + (int64_t)c0 * ldb, ldb,
                       reinterpret_cast<T*>(X.ptr) + s * X.bmul + (int64_t)c0 * ldx, ldx, nc, sm);
}

// Same operation on arbitrary column blocks: descriptor d covers leaf d.leaf's rows of a block.
template <int NC>
__global__ void __launch_bounds__(256) k_leaf_tri_desc(const double* __restrict__ Lf, DTree t, int op,
                                                       const LeafDesc* __restrict__ descs) {
  extern __shared__ __align__(16) unsigned char smraw[];
  double* sm = reinterpret_cast<double*>(smraw);
  const LeafDesc d = descs[blockIdx.x];
  const int c0 = blockIdx.y * NC;
  if (c0 >= d.ncols) return;
  const int nc = min(NC, d.ncols - c0);
  const int m = d_leaf_size(t, d.leaf);
  double* p = d.ptr + (int64_t)c0 * d.ld;
  leaf_tri_body<double, NC>(Lf + d_leaf_koff(t, d.leaf), m, op, p, d.ld, p, d.ld, nc, sm);
}


// ---------------------------------------------------------------------------------------------
// Q_leaf' y (proj) and y += sign * Q_leaf g (expand) with the explicit leaf bases Q (m x r,
// column-major at start*r).  grid = (nleaf, ceil(k / 16)), block 256.
// ---------------------------------------------------------------------------------------------
// VP[leaf][c] = Q_leaf' y_c for a chunk of up to 16 columns and the basis columns q0 .. q0 + rq - 1.
// The leaf is processed in chunks of 64 rows: Q (64 x rq, padded rows) and y (16 x 64) are staged in
// shared memory, then thread t owns basis column t % rq and the columns of group t / rq, with up to
// 6 accumulators; where there are at least twice as many groups as columns, the groups of a column
// share its rows and their sums are added in order at the end.  Few leaves split the basis columns
// over CTAs: 2 leaves of 500 points, 25 columns, rank 32 took 250 us on 4 CTAs, now 40 us.
constexpr int kProjRows = 64;
constexpr int kProjCols = 16;

template <typename T>
__global__ void __launch_bounds__(256) k_leaf_qproj(const T* __restrict__ Q, int r, DTree t, const T* __restrict__ Y,
                                                    int64_t ldy, T* __restrict__ VP, int k, int rq) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int q0 = blockIdx.z * rq;
  if (r - q0 < rq) rq = r - q0;
  const int ldq = rq + 1;
  T* qs = reinterpret_cast<T*>(smraw);   // kProjRows x (rq + 1): element (i, q) at i * ldq + q
  T* ys = qs + kProjRows * ldq;           // kProjCols x kProjRows
  const int64_t leaf = blockIdx.x;
  const int m = d_leaf_size(t, leaf);
  const int64_t s = d_leaf_start(t, leaf);
  const int c0 = blockIdx.y * kProjCols;
  const int nc = min(kProjCols, k - c0);
  const int tid = threadIdx.x;
  const int G = blockDim.x / rq;                // groups (>= 3 for rq <= 80)
  const int q = tid % rq, g = tid / rq;
  const int parts = max(1, G / nc);             // row parts of a column
  const int cper = parts > 1 ? 1 : (nc + G - 1) / G;  // <= 6
  const int part = parts > 1 ? g / nc : 0;
  const int cb = parts > 1 ? g % nc : g * cper, ce = min(nc, cb + cper);
  const bool active = g < G && part < parts;
  acc_t<T> acc[6] = {};
  const T* Ql = Q + s * r + (int64_t)q0 * m;
  for (int i0 = 0; i0 < m; i0 += kProjRows) {
    const int rows = min(kProjRows, m - i0);
    __syncthreads();
    for (int e = tid; e < rows * rq; e += blockDim.x) {
      const int qq = e / rows, i = e - qq * rows;
      qs[i * ldq + qq] = Ql[(int64_t)qq * m + i0 + i];
    }
    for (int e = tid; e < nc * rows; e += blockDim.x) {
      const int c = e / rows, i = e - c * rows;
      ys[c * kProjRows + i] = Y[(int64_t)(c0 + c) * ldy + s + i0 + i];
    }
    __syncthreads();
    // cper columns a thread, unrolled for that number (a multiply-add that is switched off still
    // takes its pipe); a last group with fewer columns repeats its last one
    auto dots = [&](auto count) {
      constexpr int CP = decltype(count)::value;
      int at[CP];
#pragma unroll
      for (int j = 0; j < CP; ++j) at[j] = min(cb + j, nc - 1) * kProjRows;
      for (int i = part; i < rows; i += parts) {
        const T a = qs[i * ldq + q];
#pragma unroll
        for (int j = 0; j < CP; ++j) acc[j] += a * ys[at[j] + i];
      }
    };
    if (active) switch (cper) {
        case 1: dots(std::integral_constant<int, 1>{}); break;
        case 2: dots(std::integral_constant<int, 2>{}); break;
        case 3: dots(std::integral_constant<int, 3>{}); break;
        case 4: dots(std::integral_constant<int, 4>{}); break;
        default: dots(std::integral_constant<int, 6>{});
      }
  }
  if (parts > 1) {
    __syncthreads();
    T* sums = qs;  // part x column x rq (at most 256 values)
    if (active) sums[(part * nc + cb) * rq + q] = accv(acc[0]);
    __syncthreads();
    if (active && part == 0) {
      acc_t<T> tot = sums[cb * rq + q];
      for (int p = 1; p < parts; ++p) tot += sums[(p * nc + cb) * rq + q];
      VP[(leaf * k + c0 + cb) * r + q0 + q] = accv(tot);
    }
    return;
  }
  if (active)
#pragma unroll
    for (int j = 0; j < 6; ++j)
      if (cb + j < ce) VP[(leaf * k + c0 + cb + j) * r + q0 + q] = accv(acc[j]);
}

// y_c += sign * Q_leaf g_c for a chunk of up to CB columns and 128 rows: thread per leaf row, the
// chunk's coefficients g (CB x r) in shared memory, one accumulator per column; Q is read once
// per chunk.
constexpr int kExpRows = 128;

template <typename T, int CB>
__global__ void __launch_bounds__(kExpRows) k_leaf_qexpand(const T* __restrict__ Q, int r, DTree t,
                                                           const T* __restrict__ VG, T* __restrict__ Y, int64_t ldy,
                                                           int k, double sign) {
  extern __shared__ __align__(16) unsigned char smraw[];
  T* gs = reinterpret_cast<T*>(smraw);  // CB x r
  const int64_t leaf = blockIdx.x;
  const int m = d_leaf_size(t, leaf);
  const int64_t s = d_leaf_start(t, leaf);
  const int c0 = blockIdx.y * CB;
  const int nc = min(CB, k - c0);
  for (int e = threadIdx.x; e < nc * r; e += blockDim.x) gs[e] = VG[(leaf * k + c0) * r + e];
  __syncthreads();
  const T* Ql = Q + s * r;
  const bool add = sign > 0.0;
  const int i = blockIdx.z * kExpRows + threadIdx.x;
  if (i >= m) return;
  acc_t<T> acc[CB] = {};
  int q = 0;
  for (; q + 3 < r; q += 4) {  // four basis entries loaded ahead of their multiply-adds
    T a[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) a[u] = Ql[(int64_t)(q + u) * m + i];
#pragma unroll
    for (int c = 0; c < CB; ++c)
      if (c < nc) {
#pragma unroll
        for (int u = 0; u < 4; ++u) acc[c] += a[u] * gs[c * r + q + u];
      }
  }
  for (; q < r; ++q) {
    const T a = Ql[(int64_t)q * m + i];
#pragma unroll
    for (int c = 0; c < CB; ++c)
      if (c < nc) acc[c] += a * gs[c * r + q];
  }
#pragma unroll
  for (int c = 0; c < CB; ++c)
    if (c < nc) {
      T* y = Y + (int64_t)(c0 + c) * ldy + s + i;
      *y = add ? *y + accv(acc[c]) : *y - accv(acc[c]);
    }
}

// ---------------------------------------------------------------------------------------------
// FP64 leaf solves L x = b (op 0) and L' x = b (op 1) by 32-row blocks with the inverses of the
// diagonal blocks: x_q = X_q (b_q - L_{q,<q} x_{<q}).  A substitution inside a block is 32 steps of
// one useful lane each; with X_q it is a product whose rows a and 31 - a of two columns share a
// lane: 33 FP64 instructions for 2 columns instead of 128, and no chain.  X_q (strictly lower part)
// lives in the block's upper triangle of Lf, which nothing else uses.
// Measured: 128 leaves of 312 points, 32 right-hand sides 0.67 -> 0.54 ms; 2 leaves of 500, one right-hand
// side 270 -> 205 us.
//
// A product with X_q loses up to the block's condition number against the substitution (points closer to
// each other than the nugget hides, next to each other in a leaf), so a block whose X_q has an entry above
// kIllBlock times 1 / L[0][0] is solved by substitution.
// Blocks of a nugget of 1e-3 and more stay below 32.  Right-hand sides K x of a smooth x, 160 points with
// neighbours 1e-3 apart, error of x: nugget 1e-3 (entries to 25) 1.0e-12 both ways; 1e-5 (229) 8e-10 by products,
// 7e-11 by substitution.
// ---------------------------------------------------------------------------------------------

// X_q of every diagonal block: grid (nleaf, blocks), 4 warps, lane = column of X; warp i mod 4 keeps
// the rows i; row l is finished by its warp, then subtracted from the rows below.
__global__ void __launch_bounds__(128) k_leaf_diaginv(double* __restrict__ Lf, DTree t) {
  __shared__ double D[32 * 33], X[32 * 33], inv[32];
  const int64_t leaf = blockIdx.x;
  const int m = d_leaf_size(t, leaf), i0 = blockIdx.y * 32;
  if (i0 >= m) return;
  const int ib = min(32, m - i0), lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double* L = Lf + d_leaf_koff(t, leaf) + (int64_t)i0 * m + i0;
  for (int c = w; c < ib; c += 4)
    if (lane >= c && lane < ib) D[lane * 33 + c] = L[(int64_t)c * m + lane];
  for (int i = w; i < 32; i += 4) X[i * 33 + lane] = i == lane ? 1.0 : 0.0;
  if (w == 0 && lane < ib) inv[lane] = 1.0 / L[(int64_t)lane * m + lane];
  __syncthreads();
  for (int l = 0; l < ib; ++l) {
    if (w == (l & 3)) X[l * 33 + lane] *= inv[l];
    __syncthreads();
    const double x = X[l * 33 + lane];
    for (int i = l + 1 + ((w - l - 1) & 3); i < ib; i += 4) X[i * 33 + lane] -= D[i * 33 + l] * x;
  }
  __syncthreads();
  for (int i = w; i < ib; i += 4)  // X[i][l], l < i, at row l of column i
    if (lane < i) L[(int64_t)i * m + lane] = X[i * 33 + lane];
}

// The row updates of the backward solve read L along its columns, a row a lane.  With large leaves and several
// CTAs an SM these loads of 32 lines each bound it (128 leaves of 1025, 16 columns: 7.1 ms, the
// substitution 3.6), so that there a warp turns its entries round in shared memory (2.9 ms).  Up to 768 points
// or with a CTA an SM the direct loads are as fast or faster (128 of 700, 13 columns: 1.33 against 1.57 ms).
enum { kForward = 0, kDirect = 1, kTurned = 2 };
// CTAs an SM holds by their registers: 40 a thread forward with one or two columns, else 48; turned with more 64
__host__ __device__ constexpr int solve_ctas(int nc, int form) {
  return nc <= 2 ? (form == kForward ? 6 : 5) : form == kTurned ? 4 : 5;
}

// x of the 32-row block at row i0 of nc columns (column c at xs[c m]) by substitution: a warp per column, lane =
// row; D holds the block of L (row-major, leading dimension 33), the diagonal as reciprocals
template <int OP>
__device__ __noinline__ void block_subst(const double* D, double* xs, int m, int i0, int ib, int nc) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int c = w; c < nc; c += 8) {
    double v = lane < ib ? xs[c * m + i0 + lane] : 0.0;
    for (int u = 0; u < ib; ++u) {
      const int l = OP == 0 ? u : ib - 1 - u;
      if (lane == l) v *= D[l * 33 + l];
      const double x = __shfl_sync(0xffffffffu, v, l);
      if (OP == 0 ? (lane > l && lane < ib) : lane < l) v -= (OP == 0 ? D[lane * 33 + l] : D[l * 33 + lane]) * x;
    }
    if (lane < ib) xs[c * m + i0 + lane] = v;
  }
}

template <int NC, int FORM>
__global__ void __launch_bounds__(256, solve_ctas(NC, FORM)) k_leaf_solve(const double* __restrict__ Lf, DTree t,
                                                    double* __restrict__ Xg, int64_t ldx, int k) {
  constexpr int OP = FORM == kForward ? 0 : 1;
  extern __shared__ __align__(16) unsigned char smraw[];
  double* xs = reinterpret_cast<double*>(smraw);  // NC x m
  const int64_t leaf = blockIdx.x;
  const int m = d_leaf_size(t, leaf);
  const double* L = Lf + d_leaf_koff(t, leaf);
  double* D = xs + NC * m;                        // 32 x 33 (turned: 8 x 32 x 9 while rows are updated)
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int c0 = blockIdx.y * NC, nc = min(NC, k - c0);
  double* X = Xg + d_leaf_start(t, leaf) + (int64_t)c0 * ldx;
  for (int c = 0; c < nc; ++c)
    for (int i = tid; i < m; i += 256) xs[c * m + i] = X[(int64_t)c * ldx + i];
  const int nblk = (m + 31) / 32;
  const int ill = __double2hiint((double)(kIllBlock / (float)L[0]));
  for (int q = 0; q < nblk; ++q) {
    const int i0 = 32 * (OP == 0 ? q : nblk - 1 - q), ib = min(32, m - i0);
    bool above = false;
    __syncthreads();
    // op 0: D[a][l] = X_q[a][l], l <= a; op 1: D[a][l] = X_q[31 - l][31 - a], the transpose with rows
    // and columns reversed, again lower triangular (rows beyond the block are zero)
    for (int i = w; i < 32; i += 8) {
      double v = 0.0;
      if (i < ib && lane <= i) {
        const double e = L[(int64_t)(i0 + i) * m + i0 + lane];
        v = lane == i ? 1.0 / e : e;
        above |= (__double2hiint(v) & 0x7fffffff) > ill;
      }
      if (lane <= i) D[OP == 0 ? i * 33 + lane : (31 - lane) * 33 + 31 - i] = v;
    }
    if (__syncthreads_or(above)) {
      for (int l = w; l < ib; l += 8)
        if (lane >= l && lane < ib) {
          const double e = L[(int64_t)(i0 + l) * m + i0 + lane];
          D[lane * 33 + l] = lane == l ? 1.0 / e : e;
        }
      __syncthreads();
      block_subst<OP>(D, xs, m, i0, ib, nc);
    } else {
      for (int c = 2 * w; c < nc; c += 16) {
        double* b0 = xs + c * m + i0;
        double* b1 = c + 1 < nc ? b0 + m : b0;
        double first = 0.0, acc = 0.0;
        for (int u = 0; u <= 32; ++u) {
          const bool one = u <= lane;
          if (u == lane + 1) {
            first = acc;
            acc = 0.0;
          }
          const int row = one ? lane : 31 - lane, l = one ? u : u - lane - 1;
          const int i = OP == 0 ? l : 31 - l;
          const double b = i < ib ? (one ? b0 : b1)[i] : 0.0;
          acc += D[row * 33 + l] * b;
        }
        const double second = acc;
        __syncwarp();
        const int ra = OP == 0 ? lane : 31 - lane, rb = 31 - ra;
        if (ra < ib) b0[ra] = first;
        __syncwarp();
        if (c + 1 < nc && rb < ib) b1[rb] = second;
      }
    }
    __syncthreads();
    const int R = OP == 0 ? m - (i0 + ib) : i0, r0 = OP == 0 ? i0 + ib : 0;
    constexpr int CG = NC < 4 ? NC : 4;
    const int ng = (nc + CG - 1) / CG;
    if constexpr (FORM == kTurned) {
      // row i takes L[i0 + l, i], which runs along l in memory: a warp reads 8 entries of each of its 32 rows
      // (R is a multiple of 32), 4 rows a load, and turns them round in its part of shared memory
      double* ts = D + w * 32 * 9;
      const int nr = R / 32, lq = lane & 7;
      for (int e = w; e < nr * ng; e += 8) {
        const int g = e / nr, ib0 = 32 * (e - g * nr), cb = CG * g;
        const double* xc = xs + cb * m + i0;
        const double* a = L + (int64_t)(ib0 + (lane >> 3)) * m + i0 + lq;
        double acc[CG] = {}, pre[8];
        auto fetch = [&](int l) {
#pragma unroll
          for (int u = 0; u < 8; ++u) pre[u] = l + lq < ib ? a[(int64_t)4 * u * m + l] : 0.0;
        };
        fetch(0);
        for (int l = 0; l < ib; l += 8) {
          __syncwarp();
#pragma unroll
          for (int u = 0; u < 8; ++u) ts[(4 * u + (lane >> 3)) * 9 + lq] = pre[u];
          __syncwarp();
          if (l + 8 < ib) fetch(l + 8);
          const int n = min(8, ib - l);
#pragma unroll
          for (int u = 0; u < 8; ++u)
            if (u < n) {
              const double v = ts[lane * 9 + u];
#pragma unroll
              for (int j = 0; j < CG; ++j)
                if (cb + j < nc) acc[j] += v * xc[j * m + l + u];
            }
        }
#pragma unroll
        for (int j = 0; j < CG; ++j)
          if (cb + j < nc) xs[(cb + j) * m + ib0 + lane] -= acc[j];
      }
      continue;
    }
    for (int e = tid; e < R * ng; e += 256) {
      const int g = e / R, i = r0 + (e - g * R), cb = CG * g;
      const double* xc = xs + cb * m + i0;
      const double* a = OP == 0 ? L + (int64_t)i0 * m + i : L + (int64_t)i * m + i0;
      const int64_t sa = OP == 0 ? m : 1;
      double acc[CG] = {};
      int l = 0;
      for (; l + 7 < ib; l += 8) {  // eight entries loaded ahead of their multiply-adds
        double av[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) av[u] = a[(l + u) * sa];
#pragma unroll
        for (int u = 0; u < 8; ++u)
#pragma unroll
          for (int j = 0; j < CG; ++j)
            if (cb + j < nc) acc[j] += av[u] * xc[j * m + l + u];
      }
      for (; l < ib; ++l)
#pragma unroll
        for (int j = 0; j < CG; ++j)
          if (cb + j < nc) acc[j] += a[l * sa] * xc[j * m + l];
#pragma unroll
      for (int j = 0; j < CG; ++j)
        if (cb + j < nc) xs[(cb + j) * m + i] -= acc[j];
    }
  }
  __syncthreads();
  for (int c = 0; c < nc; ++c)
    for (int i = tid; i < m; i += 256) X[(int64_t)c * ldx + i] = xs[c * m + i];
}

// ---------------------------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------------------------
template <typename T, int NC>
static bool tri_launch(const T* Lf, const Tree& t, int op, LeafOperand B, LeafOperand X, int ncols,
                       cudaStream_t st) {
  const size_t sm = ((size_t)(op >= 2 ? 2 : 1) * NC * t.max_leaf + 32 * 33) * sizeof(T);
  if (sm > 200 * 1024) return false;
  smem_limit((const void*)k_leaf_tri<T, NC>, sm);
  dim3 grid((unsigned)t.nleaf, (unsigned)((ncols + NC - 1) / NC));
  k_leaf_tri<T, NC><<<grid, 256, sm, st>>>(Lf, dtree(t), op, B, X, ncols);
  return true;
}

template <typename T>
bool launch_leaf_tri(const T* Lf, const Tree& t, int op, T* Bptr, int64_t bmul, int64_t bld, int bld_is_m, T* Xptr,
                     int64_t xmul, int64_t xld, int xld_is_m, int ncols, cudaStream_t st) {
  LeafOperand B{reinterpret_cast<double*>(Bptr), bmul, bld, bld_is_m};
  LeafOperand X{reinterpret_cast<double*>(Xptr), xmul, xld, xld_is_m};
  // widest column chunk that still gives about four CTAs per SM (each CTA re-reads its leaf's
  // factor, which the L2 serves)
  auto ctas = [&](int nc) { return t.nleaf * (int64_t)((ncols + nc - 1) / nc); };
  const int64_t want = 4 * 152;
  if (ncols > 8 && ctas(16) >= want && tri_launch<T, 16>(Lf, t, op, B, X, ncols, st)) return true;
  if (ncols > 4 && ctas(8) >= want && tri_launch<T, 8>(Lf, t, op, B, X, ncols, st)) return true;
  if (ncols > 1 && tri_launch<T, 4>(Lf, t, op, B, X, ncols, st)) return true;
  return tri_launch<T, 1>(Lf, t, op, B, X, ncols, st);
}

template <int NC>
static bool tri_desc_launch(const double* Lf, const Tree& t, int op, const LeafDesc* descs, int n, int maxcols,
                            cudaStream_t st) {
  const size_t sm = ((size_t)(op >= 2 ? 2 : 1) * NC * t.max_leaf + 32 * 33) * sizeof(double);
  if (sm > 200 * 1024) return false;
  smem_limit((const void*)k_leaf_tri_desc<NC>, sm);
  dim3 grid((unsigned)n, (unsigned)((maxcols + NC - 1) / NC));
  k_leaf_tri_desc<NC><<<grid, 256, sm, st>>>(Lf, dtree(t), op, descs);
  return true;
}

bool launch_leaf_tri_desc(const double* Lf, const Tree& t, int op, const LeafDesc* descs, int n, int maxcols,
                          cudaStream_t st) {
  if (n <= 0) return true;
  if (tri_desc_launch<16>(Lf, t, op, descs, n, maxcols, st)) return true;
  if (tri_desc_launch<8>(Lf, t, op, descs, n, maxcols, st)) return true;
  if (tri_desc_launch<4>(Lf, t, op, descs, n, maxcols, st)) return true;
  return tri_desc_launch<1>(Lf, t, op, descs, n, maxcols, st);
}

template <typename T>
void launch_leaf_proj(const T* Q, const T*, int r, const Tree& t, const T* Y, int64_t ldy, T* VP, int k,
                      cudaStream_t st) {
  const unsigned chunks = (unsigned)((k + kProjCols - 1) / kProjCols);
  // basis columns of a CTA: halved while the CTAs do not fill the SMs twice (the right-hand sides
  // are then staged once per part)
  int parts = 1;
  while (t.nleaf * chunks * parts < 2 * 152 && r >= 16 * parts) parts *= 2;
  const int rq = (r + parts - 1) / parts;
  dim3 grid((unsigned)t.nleaf, chunks, (unsigned)((r + rq - 1) / rq));
  const size_t sm = std::max<size_t>((size_t)kProjRows * (rq + 1) + kProjCols * kProjRows, 256) * sizeof(T);
  smem_limit((const void*)k_leaf_qproj<T>, sm);
  k_leaf_qproj<T><<<grid, 256, sm, st>>>(Q, r, dtree(t), Y, ldy, VP, k, rq);
}

template <typename T, int CB>
static void expand_launch(const T* Q, int r, const Tree& t, const T* VG, T* Y, int64_t ldy, int k, double sign,
                          cudaStream_t st) {
  dim3 grid((unsigned)t.nleaf, (unsigned)((k + CB - 1) / CB), (unsigned)((t.max_leaf + kExpRows - 1) / kExpRows));
  k_leaf_qexpand<T, CB><<<grid, kExpRows, (size_t)CB * r * sizeof(T), st>>>(Q, r, dtree(t), VG, Y, ldy, k, sign);
}

template <typename T>
void launch_leaf_expand(const T* Q, const T*, int r, const Tree& t, const T* VG, T* Y, int64_t ldy, int k,
                        double sign, cudaStream_t st) {
  // 16 columns a CTA reads Q least often; 4 where 16 would leave SMs without a CTA
  const int64_t rows = (t.max_leaf + kExpRows - 1) / kExpRows;
  if (k <= 4 || t.nleaf * rows * ((k + 15) / 16) < 4 * 152)
    expand_launch<T, 4>(Q, r, t, VG, Y, ldy, k, sign, st);
  else
    expand_launch<T, 16>(Q, r, t, VG, Y, ldy, k, sign, st);
}

void launch_leaf_diaginv(double* Lf, const Tree& t, cudaStream_t st) {
  k_leaf_diaginv<<<dim3((unsigned)t.nleaf, (unsigned)((t.max_leaf + 31) / 32)), 128, 0, st>>>(Lf, dtree(t));
}

template <int NC, int FORM>
static bool solve_form(const double* Lf, const Tree& t, double* X, int64_t ldx, int k, size_t sm, cudaStream_t st) {
  smem_limit((const void*)k_leaf_solve<NC, FORM>, sm);
  k_leaf_solve<NC, FORM><<<dim3((unsigned)t.nleaf, (unsigned)((k + NC - 1) / NC)), 256, sm, st>>>(Lf, dtree(t), X, ldx, k);
  return true;
}

static int solve_form_of(const Tree& t, int op, int nc, int k) {
  return op == 0 ? kForward : t.max_leaf > 768 && t.nleaf * (int64_t)((k + nc - 1) / nc) > 152 ? kTurned : kDirect;
}
static size_t solve_smem(const Tree& t, int nc, int form) {
  return ((size_t)nc * t.max_leaf + (form == kTurned ? 8 * 32 * 9 : 32 * 33)) * sizeof(double);
}

template <int NC>
static bool solve_launch(const double* Lf, const Tree& t, int op, double* X, int64_t ldx, int k, cudaStream_t st) {
  const int form = solve_form_of(t, op, NC, k);
  const size_t sm = solve_smem(t, NC, form);
  if (sm > 200 * 1024) return false;
  return form == kForward  ? solve_form<NC, kForward>(Lf, t, X, ldx, k, sm, st)
         : form == kDirect ? solve_form<NC, kDirect>(Lf, t, X, ldx, k, sm, st)
                           : solve_form<NC, kTurned>(Lf, t, X, ldx, k, sm, st);
}

bool launch_leaf_solve_f64(const double* Lf, const Tree& t, int op, double* X, int64_t ldx, int k, cudaStream_t st) {
  // widest column chunk that still gives about four CTAs an SM (a CTA reads its leaf's factor once)
  auto ctas = [&](int nc) { return t.nleaf * (int64_t)((k + nc - 1) / nc); };
  const int64_t want = 4 * 152;
  if (k > 8 && ctas(16) >= want && solve_launch<16>(Lf, t, op, X, ldx, k, st)) return true;
  if (k > 4 && ctas(8) >= want && solve_launch<8>(Lf, t, op, X, ldx, k, st)) return true;
  // few CTAs: two columns each, or four where only those run all at once, by registers and shared memory
  // (32 leaves of 2800, 33 columns, backward: 12.0 ms in two waves, 10.0 in one)
  auto at_once = [&](int nc) {
    const int form = solve_form_of(t, op, nc, k);
    return ctas(nc) <= 152 * std::min<int64_t>(solve_ctas(nc, form), 227 * 1024 / (solve_smem(t, nc, form) + 1024));
  };
  if (k > 2 && (ctas(4) >= want || (!at_once(2) && at_once(4))) && solve_launch<4>(Lf, t, op, X, ldx, k, st)) return true;
  if (k > 1 && solve_launch<2>(Lf, t, op, X, ldx, k, st)) return true;
  return solve_launch<1>(Lf, t, op, X, ldx, k, st);
}

template bool launch_leaf_tri<double>(const double*, const Tree&, int, double*, int64_t, int64_t, int, double*,
                                      int64_t, int64_t, int, int, cudaStream_t);
template bool launch_leaf_tri<ff>(const ff*, const Tree&, int, ff*, int64_t, int64_t, int, ff*, int64_t, int64_t,
                                  int, int, cudaStream_t);
template void launch_leaf_proj<double>(const double*, const double*, int, const Tree&, const double*, int64_t,
                                       double*, int, cudaStream_t);
template void launch_leaf_proj<ff>(const ff*, const ff*, int, const Tree&, const ff*, int64_t, ff*, int,
                                   cudaStream_t);
template void launch_leaf_expand<double>(const double*, const double*, int, const Tree&, const double*, double*,
                                         int64_t, int, double, cudaStream_t);
template void launch_leaf_expand<ff>(const ff*, const ff*, int, const Tree&, const ff*, ff*, int64_t, int, double,
                                     cudaStream_t);

}  // namespace km
