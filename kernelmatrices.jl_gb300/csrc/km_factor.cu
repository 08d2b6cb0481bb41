// FP64 factorisation kernels of the nested Nystrom HODLR factorisation.
//
// The reference (src/HODLR/src/symfact.jl:6-49) factors K = W W' with
//   W = L_leaf * W_1 * ... * W_L,  W_N = I + M X M'  (src/HODLR/src/utils.jl:29-35),
// where every W_N is built from the Householder QR of the node's transformed off-diagonal
// panels.  With Nystrom blocks every panel is a row block of the single n x r matrix
// Phi = K(X, P) (or of Phi S^{-1}, S = K(P, P)), and left-multiplication by the earlier factors
// commutes with the right factor S^{-1}.  So after the leaf stage (A = L^{-1} Phi, A_leaf =
// Q_leaf R_leaf) every transformed panel of a node N lies in the span of its children's bases:
//   A[N] = blockdiag(Q_c1, Q_c2) G_N,   G_N = [R_c1 ; L22^{-1}(R_c2 - Ct' R_c1)]   (2r x r)
// with Ct = R_c1 S^{-1} R_c2' and L22 = chol(I - Ct' Ct), and the reference's
// X = chol([I C; C' I]) - I equals [[0,0],[C', L22 - I]] in those bases.  QR(G_N) = E_N R_N
// gives the node basis Q_N = blockdiag(Q_c1, Q_c2) E_N.  Only r x r work is left above the
// leaves; the factor is the reference's up to the rounding freedom of the QR of rank-deficient
// panels.  Orthogonal factors are kept in Householder (LAPACK dgeqrf-style) form.
#include <cooperative_groups.h>

#include <atomic>
#include <cstdlib>
#include <type_traits>

#include "km_cluster.cuh"
#include "km_kernels.h"

namespace km {

namespace cg = cooperative_groups;

// ---------------------------------------------------------------------------------------------
// Small dense Cholesky (r x r, lower, in place, column-major) for S = K(P, P).  One CTA.
// ---------------------------------------------------------------------------------------------
__global__ void k_chol_small(double* __restrict__ A, int n, int* __restrict__ info) {
  extern __shared__ double s[];  // n x (n+1)
  const int ld = n + 1;
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) s[(e % n) + (e / n) * ld] = A[e];
  __syncthreads();
  for (int j = 0; j < n; ++j) {
    const double d = s[j + j * ld];
    if (!(d > 0.0)) {
      if (threadIdx.x == 0 && info[0] == 0) info[0] = j + 1;
      __syncthreads();
      break;
    }
    const double sd = sqrt(d);
    __syncthreads();
    for (int i = j + 1 + threadIdx.x; i < n; i += blockDim.x) s[i + j * ld] /= sd;
    if (threadIdx.x == 0) s[j + j * ld] = sd;
    __syncthreads();
    // trailing lower triangle update
    const int w = n - j - 1;
    for (int e = threadIdx.x; e < w * w; e += blockDim.x) {
      const int i = j + 1 + e % w, c = j + 1 + e / w;
      if (i >= c) s[i + c * ld] -= s[i + j * ld] * s[c + j * ld];
    }
    __syncthreads();
  }
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
    const int i = e % n, c = e / n;
    A[e] = (i >= c) ? s[i + c * ld] : 0.0;
  }
}

// ---------------------------------------------------------------------------------------------
// Batched leaf Cholesky in float pairs: Lf_j = chol(K_j) (lower), blocked right-looking, one CTA
// per leaf (the FP64 form is in km_chol.cu).
// The current column panel (rows below the diagonal block) lives in shared memory.
// info[j] = first failing column (1-based) of leaf j, 0 if positive definite.
// ---------------------------------------------------------------------------------------------
template <typename T, int NB, int NT>
__global__ void __launch_bounds__(NT) k_leaf_chol(const double* __restrict__ K, T* __restrict__ Lf,
                                                  DTree t, int* __restrict__ info) {
  extern __shared__ __align__(16) unsigned char smraw[];
  T* sm = reinterpret_cast<T*>(smraw);
  const int64_t leaf = blockIdx.x;
  const int m = d_leaf_size(t, leaf);
  const int64_t off = d_leaf_koff(t, leaf);
  const double* A0 = K + off;
  T* A = Lf + off;
  constexpr int LDP = NB + 1;
  T* P = sm;                    // (m) x LDP, row-major panel rows
  T* D = sm + (size_t)m * LDP;  // NB x LDP
  const int tid = threadIdx.x, nth = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5, nwarp = nth >> 5;
  for (int64_t e = tid; e < (int64_t)m * m; e += nth) A[e] = from_double<T>(A0[e]);
  __syncthreads();
  int bad = 0;
  for (int k0 = 0; k0 < m; k0 += NB) {
    const int kb = min(NB, m - k0);
    // (1) diagonal block -> shared, unblocked Cholesky
    for (int e = tid; e < kb * kb; e += nth) {
      const int i = e % kb, c = e / kb;
      D[i * LDP + c] = A[(int64_t)(k0 + c) * m + k0 + i];
    }
    __syncthreads();
    for (int j = 0; j < kb; ++j) {
      const T d = D[j * LDP + j];
      const bool ok = d > 0.0;
      if (!ok && bad == 0) bad = k0 + j + 1;
      const T sd = ok ? sqrt(d) : T(1.0);
      __syncthreads();
      for (int i = j + 1 + tid; i < kb; i += nth) D[i * LDP + j] /= sd;
      if (tid == 0) D[j * LDP + j] = sd;
      __syncthreads();
      const int w = kb - j - 1;
      for (int e = tid; e < w * w; e += nth) {
        const int i = j + 1 + e % w, c = j + 1 + e / w;
        if (i >= c) D[i * LDP + c] -= D[i * LDP + j] * D[c * LDP + j];
      }
      __syncthreads();
    }
    for (int e = tid; e < kb * kb; e += nth) {
      const int i = e % kb, c = e / kb;
      if (i >= c) A[(int64_t)(k0 + c) * m + k0 + i] = D[i * LDP + c];
    }
    // (2) panel rows i >= k0+kb: x D' = a  (forward substitution per row)
    const int r0 = k0 + kb, mr = m - r0;
    for (int ii = tid; ii < mr; ii += nth) {
      const int i = r0 + ii;
      T x[NB];
#pragma unroll
      for (int c = 0; c < NB; ++c) {
        if (c < kb) {
          acc_t<T> v = A[(int64_t)(k0 + c) * m + i];
          for (int l = 0; l < c; ++l) v -= x[l] * D[c * LDP + l];
          x[c] = accv(v) / D[c * LDP + c];
        }
      }
#pragma unroll
      for (int c = 0; c < NB; ++c) {
        if (c < kb) {
          P[ii * LDP + c] = x[c];
          A[(int64_t)(k0 + c) * m + i] = x[c];
        }
      }
    }
    __syncthreads();
    // (3) trailing update of the lower triangle: A[i, c] -= sum_l P[i,l] P[c,l]
    for (int cc = warp; cc < mr; cc += nwarp) {
      T pc[NB];
#pragma unroll
      for (int l = 0; l < NB; ++l) pc[l] = (l < kb) ? P[cc * LDP + l] : T(0.0);
      T* col = A + (int64_t)(r0 + cc) * m + r0;
      for (int ii = cc + lane; ii < mr; ii += 32) {
        acc_t<T> acc{};
#pragma unroll
        for (int l = 0; l < NB; ++l) acc += P[ii * LDP + l] * pc[l];
        col[ii] -= accv(acc);
      }
    }
    __syncthreads();
  }
  if (tid == 0) info[leaf] = bad;
}

// ---------------------------------------------------------------------------------------------
// Batched Householder QR of the leaf panels A_j (m_j x r, column-major at start(j)*r), in place:
// reflector vectors below the diagonal (unit leading entry implicit), tau[j*r + c], and
// R_j (r x r column-major, zeros below the diagonal) written to Rout[j*r*r].
// Follows LAPACK dgeqr2/dlarfg: beta = -sign(alpha) ||(alpha, x)||, tau = (beta-alpha)/beta,
// v = x/(alpha-beta); a zero column x gives tau = 0 (H = I).  One CTA per leaf; the panel is
// copied to shared memory when it fits.
// ---------------------------------------------------------------------------------------------
// Householder QR of the leaf panels (m x r, in place: R above, the scaled reflectors below), a CTA per
// leaf, in dataflow order: of the NW warps warp w owns the columns w, w + NW, ...; reflector j + 1 is formed
// by the warp that owns its column as soon as it has applied reflector j to it, before its other columns,
// and published with a flag (the unscaled column; scale and tau in sc, ta).  The reflectors are scaled at
// the end.  Waits are bounded; one that runs out marks the leaf with info = -1 and the warp carries on.
// With two block barriers a column and one thread forming the reflector between them (same operations,
// same order) 256 panels of 256 x 72 took 636 us in float pairs and 1.64 ms in FP64, 512 of 488 x 72
// 2.35 ms in float pairs; now 527 us, 1.42 ms and 1.91 ms.  FP64 has
// half of the warps (64 panels of 469 x 72: 1.76, 1.07, 0.97, 0.95 ms with 4, 8, 12, 16).  grid nleaf, block 32 NW.
template <typename T>
constexpr int leaf_qr_warps() { return std::is_same<T, double>::value ? 16 : 32; }

template <typename T, bool SMEM>
__global__ void __launch_bounds__(32 * leaf_qr_warps<T>()) k_leaf_qr(T* __restrict__ Pan, int r, DTree t,
                                                                    T* __restrict__ tau, T* __restrict__ Rout,
                                                                    int* __restrict__ info, int wait_limit) {
  constexpr int NW = leaf_qr_warps<T>(), NT = 32 * NW;
  extern __shared__ __align__(16) unsigned char smraw[];
  T* sm = reinterpret_cast<T*>(smraw);
  __shared__ T red[32], sc[kMaxNysRank], ta[kMaxNysRank];
  __shared__ volatile int flag[kMaxNysRank];
  const int lim = wait_limit < 0 ? kWaitPolls : wait_limit;
  const int64_t leaf = blockIdx.x;
  const int m = d_leaf_size(t, leaf);
  T* G = Pan + d_leaf_start(t, leaf) * r;
  T* A = SMEM ? sm : G;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int kmax = min(m, r);
  for (int e = tid; e < r; e += NT) flag[e] = 0;
  if (SMEM)
    for (int e = tid; e < m * r; e += NT) sm[e] = G[e];
  __syncthreads();
  // reflector j from alpha = a[j][j] and sig, the squared norm below it (all lanes alike): one division
  // forms tau = (beta - alpha) / beta in lane 1 and scale = 1 / (alpha - beta) in the others
  auto reflect = [&](int j, T sig) {
    T* aj = A + (int64_t)j * m;
    const T alpha = aj[j];
    T tj = T(0.0), beta = alpha, scal = T(0.0);
    if (sig != 0.0) {
      const T nrm = sqrt(alpha * alpha + sig);
      beta = alpha >= 0.0 ? -nrm : nrm;
      const T num = lane == 1 ? beta - alpha : T(1.0), den = lane == 1 ? beta : alpha - beta;
      const T q = num / den;
      tj = shfl_idx(q, 1);
      scal = shfl_idx(q, 0);
    }
    __syncwarp();
    if (lane == 0) {
      aj[j] = beta;
      sc[j] = scal;
      ta[j] = tj;
      tau[leaf * r + j] = tj;
    }
    __threadfence_block();
    __syncwarp();
    if (lane == 0) flag[j] = 1;
  };
  {  // norm of column 0 below its first row
    T part = T(0.0);
    // (in FP64 the sums of 8 warps, also with 16: the order of the additions fixes the factor's bits)
    constexpr int NS = std::is_same<T, double>::value ? 8 : NW;
    if (w < NS)
      for (int i = 1 + tid; i < m; i += 32 * NS) part += A[i] * A[i];
    part = warp_sum_t(part);
    if (lane == 0) red[w] = part;
    __syncthreads();
    if (w == 0) reflect(0, warp_sum_t(lane < NS ? red[lane] : T(0.0)));
  }
  bool timed_out = false;
  const int last = w < r ? w + (r - 1 - w) / NW * NW : -1;
  for (int j = 0; j < min(kmax, last); ++j) {
    if (!timed_out) {
      int spins = 0;
      // the warp of the next reflector polls; the others leave it the issue slots
      const unsigned nap = (j + 1) % NW == w ? 0 : (j + 2) % NW == w ? 32 : 256;
      while (wait_limit == 0 || flag[j] == 0) {
        if (++spins > lim) {
          if (lane == 0) info[leaf] = -1;
          timed_out = true;
          break;
        }
        if (nap) __nanosleep(nap);
      }
    }
    __threadfence_block();
    const T scal = sc[j], tj = ta[j];
    const T* aj = A + (int64_t)j * m;
    int c = j < w ? w : w + ((j - w) / NW + 1) * NW;  // own columns > j
    if (c == j + 1) {
      T* ac = A + (int64_t)c * m;
      T nrm = T(0.0);
      if (tj != 0.0) {
        T acc = T(0.0);
        for (int i = j + 1 + lane; i < m; i += 32) acc += aj[i] * ac[i];
        acc = (warp_sum_t(acc) * scal + ac[j]) * tj;
        __syncwarp();
        if (lane == 0) ac[j] -= acc;
        const T f = acc * scal;
        for (int i = j + 1 + lane; i < m; i += 32) {
          const T v = ac[i] - f * aj[i];
          ac[i] = v;
          if (i > j + 1) nrm += v * v;
        }
        __syncwarp();
      } else {
        for (int i = j + 2 + lane; i < m; i += 32) nrm += ac[i] * ac[i];
      }
      if (c < kmax) reflect(c, warp_sum_t(nrm));
      c += NW;
    }
    if (tj == 0.0) continue;
    // float pairs: two columns at a time, two independent dot products and updates in flight
    constexpr int NC = std::is_same<T, ff>::value ? 2 : 1;
    for (; c <= last; c += NC * NW) {
      const bool two = NC == 2 && c + NW <= last;
      T* ac = A + (int64_t)c * m;
      T* ac2 = two ? ac + (int64_t)NW * m : ac;
      T acc = T(0.0), acc2 = T(0.0);
      for (int i = j + 1 + lane; i < m; i += 32) {
        const T x = aj[i];
        acc += x * ac[i];
        if (two) acc2 += x * ac2[i];
      }
      acc = (warp_sum_t(acc) * scal + ac[j]) * tj;
      if (two) acc2 = (warp_sum_t(acc2) * scal + ac2[j]) * tj;
      __syncwarp();
      if (lane == 0) {
        ac[j] -= acc;
        if (two) ac2[j] -= acc2;
      }
      const T f = acc * scal, f2 = acc2 * scal;
      for (int i = j + 1 + lane; i < m; i += 32) {
        const T x = aj[i];
        ac[i] -= f * x;
        if (two) ac2[i] -= f2 * x;
      }
    }
  }
  __syncthreads();
  for (int j = w; j < kmax; j += NW) {
    T* aj = A + (int64_t)j * m;
    const T scal = sc[j];
    for (int i = j + 1 + lane; i < m; i += 32) aj[i] *= scal;
  }
  __syncthreads();
  for (int j = kmax + tid; j < r; j += NT) tau[leaf * r + j] = T(0.0);
  for (int e = tid; e < r * r; e += NT) {
    const int i = e % r, c = e / r;
    Rout[leaf * (int64_t)r * r + e] = (i <= c && i < m) ? A[(int64_t)c * m + i] : T(0.0);
  }
  if (SMEM)
    for (int e = tid; e < m * r; e += NT) G[e] = sm[e];
}

// Explicit leaf basis Q = H_0 ... H_{r-1} [I; 0] in place of the reflectors (LAPACK dorg2r).
// Runs on the side stream, overlapped with the node levels (only the solves need Q).
template <typename T, bool SMEM>
__global__ void __launch_bounds__(32 * leaf_qr_warps<T>()) k_leaf_formq(T* __restrict__ Pan, const T* __restrict__ tau,
                                                                     int r, DTree t) {
  extern __shared__ __align__(16) unsigned char smraw[];
  T* sm = reinterpret_cast<T*>(smraw);
  const int64_t leaf = blockIdx.x;
  const int m = d_leaf_size(t, leaf);
  const int64_t s = d_leaf_start(t, leaf);
  T* G = Pan + s * r;
  T* A = SMEM ? sm : G;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  if (SMEM) {
    for (int64_t e = tid; e < (int64_t)m * r; e += blockDim.x) sm[e] = G[e];
  }
  const int kmax = min(m, r);
  __syncthreads();
  // explicit Q = H_0 ... H_{r-1} [I; 0] in place (LAPACK dorg2r)
  for (int j = kmax - 1; j >= 0; --j) {
    T* aj = A + (int64_t)j * m;
    const T tj = tau[leaf * r + j];
    if (j < r - 1) {
      if (tid == 0) aj[j] = T(1.0);
      __syncthreads();
      for (int c = j + 1 + w; c < r; c += (int)(blockDim.x >> 5)) {
        T* ac = A + (int64_t)c * m;
        T acc = T(0.0);
        for (int i = j + lane; i < m; i += 32) acc += aj[i] * ac[i];
        acc = warp_sum_t(acc) * tj;
        for (int i = j + lane; i < m; i += 32) ac[i] -= acc * aj[i];
      }
      __syncthreads();
    }
    for (int i = j + 1 + tid; i < m; i += blockDim.x) aj[i] = -(tj * aj[i]);
    for (int i = tid; i < j; i += blockDim.x) aj[i] = T(0.0);
    if (tid == 0) aj[j] = T(1.0) - tj;
    __syncthreads();
  }
  if (SMEM) {
    __syncthreads();
    for (int64_t e = tid; e < (int64_t)m * r; e += blockDim.x) G[e] = sm[e];
  }
}

// ---------------------------------------------------------------------------------------------
// Node factorisation in float pairs (the FP64 form is in km_node64.cu), one CTA or a cluster of 2, 4 or 8
// CTAs per node of level l.  Given the children's R factors (slots c1, c2) and Sc = chol(S) (lower):
//   T1 = R1 Sc^{-T}, T2 = R2 Sc^{-T}   (upper triangular)
//   Ct = T1 T2'                        (= R1 S^{-1} R2')
//   L22 = chol(I - Ct' Ct)
//   if l < L:  G = [R1 ; L22^{-1}(R2 - Ct' R1)],  Householder QR  G = E R_N  (structured:
//              reflector j is e_j on top plus a dense bottom part, kept in Eref[:, j])
// Outputs per node: Ct, L22 (lower), Eref (r x r), Etau (r), R_N into slot N.
//
// Products: (column, 32-row chunk) or entry items over the threads, sums in the Dot2 accumulator
// (km_ff.cuh).  In a cluster every CTA loads the inputs and takes the columns rank, rank + csize, ... of
// T1 and Ct, which go into every CTA's shared memory, and the rows of T2 that it needs itself; H goes to
// CTA 0, the columns of B to the others.  Cluster barriers separate the phases (they also make sure that
// every CTA has started before the first remote store and that no CTA exits while others write to it).
// Cholesky: one warp factors panels of 4 columns in registers, other warps apply them; a panel's chain of
// square roots and reciprocals (about 450 cycles a column) bounds it, so that its warp has its quarter of
// the SM to itself.  L22^{-1} B follows one panel behind, in the same CTA or in the other CTAs of the
// cluster, which get every panel in one bulk copy; CTA 0 collects the result.
// QR (CTA 0): a dataflow pipeline in which each warp owns four columns and forms their reflectors itself.
// Rank 72, cycles of a node: 265 k with one CTA (was 425 k with a warp per Cholesky column, flags between
// them, and the solve after it), 134 k with 8 (was 245 k).
// Shared memory: four r x 82 matrices, three r-vectors, barriers, flags and the list of H's entries.
// ---------------------------------------------------------------------------------------------

// v into the same shared-memory location as p in every CTA of the cluster (locally if csize = 1)
template <typename T>
__device__ __forceinline__ void put_all(T* p, T v, int csize) {
  if (csize == 1) {
    *p = v;
    return;
  }
  cg::cluster_group cl = cg::this_cluster();
  for (int d = 0; d < csize; ++d) *cl.map_shared_rank(p, (unsigned)d) = v;
}

// v into the same shared-memory location as p in CTA 0 of the cluster (locally if csize = 1)
template <typename T>
__device__ __forceinline__ void put_rank0(T* p, T v, int csize) {
  if (csize == 1) {
    *p = v;
    return;
  }
  *cg::this_cluster().map_shared_rank(p, 0u) = v;
}

// barrier over the cluster (release/acquire for the remote stores), or over the CTA if csize = 1
__device__ __forceinline__ void node_barrier(int csize) {
  if (csize == 1) __syncthreads();
  else cg::this_cluster().sync();
}

// up to 96 registers a thread (with 1024 threads some values went to local memory); warps for 80 QR columns
constexpr int kNodeThreads = 640;
constexpr int kPanel = 4;    // columns of L22 factored at a time
// columns of the shared-memory matrices lie this far apart: above the largest rank (80), a constant, so
// that addresses are immediates, and 16 bytes times an odd number, so that two neighbours of a column
// are one load and the lanes' loads from 8 columns hit different banks
constexpr int kNodeLd = 82;

constexpr int kPivotRow = 81;  // (row 81 of a column is free)

struct __align__(16) ffpair {
  ff a, b;
};
// elements l and l + 1 (l even) of a column
__device__ __forceinline__ ffpair two(const ff* p) { return *reinterpret_cast<const ffpair*>(p); }

// The kPanel = 4 columns c0 .. c0 + 3 of L22 by one warp, element (i, c) at X[i + c kNodeLd]: the rows
// from the chunk of c0 down in its lanes, NC chunks of 32.  The columns hold their accumulators, all
// earlier panels applied.  The reciprocal pivot of column c goes to X[kPivotRow + c kNodeLd], into bad
// the first column (from 1) whose pivot is not positive.
template <int NC>
__device__ __forceinline__ void chol_panel(ff* X, int r, int c0, int lane, int& bad) {
  constexpr int ld = kNodeLd;
  const int i0 = (c0 & ~31) + lane;
  ffacc v[4][NC];
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int s = 0; s < NC; ++s) {
      const int i = i0 + 32 * s, c = c0 + j;
      v[j][s] = (i >= c && i < r && c < r) ? X[i + c * ld] : ff(0.f, 0.f);
    }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int c = c0 + j;
    if (c >= r) break;
    const ff d = shfl_idx(accv(v[j][0]), c & 31);
    if (!(d > 0.0) && bad == 0) bad = c + 1;
    const ff sd = d > 0.0 ? sqrt(d) : ff(1.0);
    const ff inv = ff_recip(sd);
    ff x[NC];
#pragma unroll
    for (int s = 0; s < NC; ++s) {
      const int i = i0 + 32 * s;
      x[s] = accv(v[j][s]) * inv;
      if (i == c) x[s] = sd;
      if (i >= c && i < r) X[i + c * ld] = x[s];
    }
    if (lane == 0) X[kPivotRow + c * ld] = inv;
#pragma unroll
    for (int q = j + 1; q < 4; ++q) {
      const ff m = shfl_idx(x[0], (c0 + q) & 31);
#pragma unroll
      for (int s = 0; s < NC; ++s) v[q][s] -= x[s] * m;
    }
  }
}

// Entry (i, c), i >= c, number e of a lower triangle of order r: columns p and r - 1 - p together hold
// r + 1 entries, so consecutive threads take consecutive entries of such a pair, and every part of the
// numbering has early and late columns.  False for the second half of the middle column of an odd r.
__device__ __forceinline__ bool lower_entry(int e, int r, int& i, int& c) {
  const int p = e / (r + 1), u = e - p * (r + 1);
  if (u >= r - p && 2 * p == r - 1) return false;
  c = u < r - p ? p : r - 1 - p;
  i = u < r - p ? p + u : r - 1 - p + (u - (r - p));
  return true;
}

template <typename T>
__global__ void __launch_bounds__(kNodeThreads) k_node_factor(T* __restrict__ R, const T* __restrict__ SinvT,
                                                     int r, int level, int L, int64_t nleaf,
                                                     int64_t cbase, int64_t nbase, T* __restrict__ Ct_out,
                                                     T* __restrict__ L22_out, T* __restrict__ Eref,
                                                     T* __restrict__ Etau, int* __restrict__ info,
                                                     int csize, int wait_limit) {
  extern __shared__ __align__(16) unsigned char smraw[];
  T* sm = reinterpret_cast<T*>(smraw);
  constexpr int ld = kNodeLd;
  // polls of a flag before a wait gives up; wait_limit 0: every wait gives up at its first poll,
  // as if its flag were never set (the test of the timeout path)
  const int lim = wait_limit < 0 ? kWaitPolls : wait_limit;
  T* X0 = sm;
  T* X1 = X0 + r * ld;
  T* X2 = X1 + r * ld;
  T* X3 = X2 + r * ld;
  T* va = X3 + r * ld;  // r values: the reflector betas
  T* vb = va + r;       // r values: the reflector scales
  T* vc = vb + r;       // r values: the reflector taus
  const int np = (r + kPanel - 1) / kPanel;  // panels of L22
  unsigned long long* pbar = reinterpret_cast<unsigned long long*>(vc + r);  // np: a panel of L22 has arrived
  int* flags = reinterpret_cast<int*>(pbar + np);  // r ints: reflector published
  unsigned short* tab = reinterpret_cast<unsigned short*>(flags + r);  // entries of H by columns: row | column << 8
  const int64_t k = blockIdx.x / csize;
  const int rank = (int)(blockIdx.x % csize);  // rank in the node's cluster (1-D clusters)
  const int64_t node = nbase + k;  // node index within all nodes (level-major)
  const T* R1 = R + (cbase + 2 * k) * (int64_t)r * r;
  const T* R2 = R + (cbase + 2 * k + 1) * (int64_t)r * r;
  const int tid = threadIdx.x, nth = blockDim.x, lane = tid & 31, w = tid >> 5, nw = nth >> 5;
  const int nch = (r + 31) >> 5;   // 32-row chunks per column (r <= 96)
  const bool solve = level < L;
  // own columns of T1 and Ct (rows of T2) c = rank + csize lc, in items (lc, 32-row chunk s)
  const int nitems = (r - rank + csize - 1) / csize * nch;
  // own columns of B: c = cfirst + cstep lc; in a cluster CTA 0 has none, it factors H
  const int cstep = csize > 1 ? csize - 1 : 1, cfirst = csize > 1 ? rank - 1 : 0;
  const int nown = cfirst < 0 ? 0 : (r - cfirst + cstep - 1) / cstep;
  // upper triangle of an r x r matrix, zero below, with all loads of a warp in flight
  auto load = [&](T* X, const T* G, bool own) {
    constexpr int kC = (80 + kNodeThreads / 32 - 1) / (kNodeThreads / 32);
    T t[kC][3];
#pragma unroll
    for (int a = 0; a < kC; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        const int c = w + nw * a, i = lane + 32 * b;
        t[a][b] = (i <= c && c < r && (!own || c % cstep == cfirst)) ? G[i + c * r] : T(0.0);
      }
#pragma unroll
    for (int a = 0; a < kC; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        const int c = w + nw * a, i = lane + 32 * b;
        if (i < r && c < r) X[i + c * ld] = t[a][b];
      }
  };
  for (int e = tid; e < r; e += nth) flags[e] = 0;
  if (rank == 0)
    for (int c = w; c < r; c += nw)
      for (int i = c + lane; i < r; i += 32) tab[c * r - c * (c - 1) / 2 + i - c] = (unsigned short)(i | c << 8);
  if (csize > 1 && solve)
    for (int e = tid; e < np; e += nth) {
      const unsigned b = smem_u32(pbar + e), n = min(kPanel, r - kPanel * e) * ld * sizeof(T);
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"(n) : "memory");
    }
  // X0 = Sc^{-T}, X1 = R1, X2 = R2, all upper triangular   (element (i,c) at i + c*ld)
  load(X0, SinvT, false);
  load(X1, R1, false);
  load(X2, R2, false);
  node_barrier(csize);
  // T1 = R1 Sc^{-T} -> X3 of every CTA: T1[i][c] = sum_{l = i..c} R1[i][l] Sinv[l][c]
  // (in all products a0 takes the first, third, ... term, a1 the second, fourth, ...)
  auto upper = [&](const T* A, int s, int c) {
    const T *a = A + min(32 * s + lane, r - 1), *x = X0 + c * ld;
    acc_t<T> a0{}, a1{};
    int l = 32 * s;
#pragma unroll 2
    for (; l + 1 <= c; l += 2) {
      const ffpair v = two(x + l);
      a0 += a[l * ld] * v.a;
      a1 += a[(l + 1) * ld] * v.b;
    }
    if (l <= c) a0 += a[l * ld] * x[l];
    return accv(a0) + accv(a1);
  };
  for (int q = w; q < nitems; q += nw) {
    const int lc = q / nch, s = q - lc * nch, c = rank + csize * lc, i = 32 * s + lane;
    if (32 * s > c) continue;
    const T v = upper(X1, s, c);
    if (i < r) put_all(X3 + i + c * ld, v, csize);
  }
  __syncthreads();
  // T2' = (R2 Sc^{-T})' -> X1 (T2[i][c] at c + i ld), own rows only: the other CTAs need no part of them
  for (int q = w; q < nitems; q += nw) {
    const int lc = q / nch, s = q - lc * nch;
    if (csize == 1) {  // a column of all rows: even work for the lanes
      const int c = lc, i = 32 * s + lane;
      if (32 * s > c) continue;
      const T v = upper(X2, s, c);
      if (i < r) X1[c + i * ld] = v;
    } else {
      const int i = rank + csize * lc, c = 32 * s + lane;
      if (c < i || c >= r) continue;
      const T *a = X2 + i, *x = X0 + c * ld;
      acc_t<T> a0{}, a1{};
      int l = i & ~1;
#pragma unroll 2
      for (; l + 1 <= c; l += 2) {
        const ffpair v = two(x + l);
        a0 += a[l * ld] * v.a;
        a1 += a[(l + 1) * ld] * v.b;
      }
      if (l <= c) a0 += a[l * ld] * x[l];
      X1[c + i * ld] = accv(a0) + accv(a1);
    }
  }
  node_barrier(csize);
  // Ct = T1 T2' -> X0 of every CTA: Ct[i][c] = sum_{l >= max(i, c)} T1[i][l] T2[c][l]
  for (int q = w; q < nitems; q += nw) {
    const int lc = q / nch, s = q - lc * nch, c = rank + csize * lc, i = 32 * s + lane;
    const T *a = X3 + min(i, r - 1), *x = X1 + c * ld;
    acc_t<T> a0{}, a1{};
    int l = max(32 * s, c);
    const bool odd = l & 1;
    if (odd) {
      a1 += a[l * ld] * x[l];  // (the two sums change places)
      ++l;
    }
#pragma unroll 2
    for (; l + 1 < r; l += 2) {
      const ffpair v = two(x + l);
      a0 += a[l * ld] * v.a;
      a1 += a[(l + 1) * ld] * v.b;
    }
    if (l < r) a0 += a[l * ld] * x[l];
    const T u = odd ? accv(a1) : accv(a0), v = odd ? accv(a0) : accv(a1);
    if (i < r) put_all(X0 + i + c * ld, u + v, csize);
  }
  node_barrier(csize);
  // R1 into X1 again: the own columns for B, all of them in CTA 0 for the QR
  if (solve) load(X1, R1, rank != 0);
  // H = I - Ct' Ct -> X3 of CTA 0, lower triangle; B costs as much as H, and CTA 0 has no part of B
  const int nh = (r + 1) / 2 * (r + 1), h0 = solve ? min(nh, (2 * nh + csize - 1) / csize) : (nh + csize - 1) / csize;
  const int hs = csize > 1 ? (nh - h0 + csize - 2) / (csize - 1) : 0;
  const int hbeg = rank ? h0 + (rank - 1) * hs : 0, hend = min(nh, hbeg + (rank ? hs : h0));
  for (int e = hbeg + tid; e < hend; e += nth) {
    int i, c;
    if (!lower_entry(e, r, i, c)) continue;
    const T *x = X0 + i * ld, *y = X0 + c * ld;
    acc_t<T> a0{}, a1{};
    int l = 0;
#pragma unroll 2
    for (; l + 1 < r; l += 2) {
      const ffpair u = two(x + l), v = two(y + l);
      a0 += u.a * v.a;
      a1 += u.b * v.b;
    }
    if (l < r) a0 += x[l] * y[l];
    put_rank0(X3 + i + c * ld, (i == c ? T(1.0) : T(0.0)) - (accv(a0) + accv(a1)), csize);
  }
  // B = R2 - Ct' R1 -> X2, own columns (column c of R1 has entries l <= c), from the last thread down:
  // the upper threads of a cluster's CTA have no entry of H
  if (solve) {
    __syncthreads();
    for (int e = nth - 1 - tid; e < nown * r; e += nth) {
      const int lc = e / r, i = e - lc * r, c = cfirst + cstep * lc;
      const T *x = X0 + i * ld, *y = X1 + c * ld;
      acc_t<T> a0{}, a1{};
      int l = 0;
#pragma unroll 2
      for (; l + 1 <= c; l += 2) {
        const ffpair u = two(x + l), v = two(y + l);
        a0 += u.a * v.a;
        a1 += u.b * v.b;
      }
      if (l <= c) a0 += x[l] * y[l];
      X2[i + c * ld] = X2[i + c * ld] - (accv(a0) + accv(a1));
    }
  }
  node_barrier(csize);
  if (rank != 0 && !solve) return;  // (no CTA touches another's memory from here on)
  // L22 = chol(H) in CTA 0 by panels of 4 columns and B' = L22^{-1} B by the CTAs that own its columns
  // (element (i, c) at X2[i + c * ld]), one panel behind.  In step p
  //   in CTA 0 four other warps on the SM quarter of warp 0 apply panel p - 1 to panel p, a column each,
  //   then warp 0 factors it and copies it to the other CTAs;
  //   warps 1 to 3, a thread per own column, take panel p - 2 in the rows of panel p - 1, solve these
  //   and hand them to CTA 0;
  //   the other warps apply panel p - 1 to the entries of H behind panel p and panel p - 2 to the rows
  //   of B from panel p on; (Next to seven busy warps warp 0 would take 7500 cycles for a panel, alone
  //   it takes 1400 to 2000.)
  // An unfinished entry of H or B is its accumulator.  Rows of B are renormalised when all rows before
  // their block of 8 are in.
  {
    const int wid = w < 4 ? -1 : rank ? w - 4 : (w & 3) ? 3 * (w >> 2) + (w & 3) - 4 : -1;
    const int nwk = rank ? nw - 4 : 3 * (nw / 4 - 1), id = 32 * wid + lane, nid = 32 * nwk;
    int bad = 0;
    bool dead = false;
    for (int p = rank ? 1 : 0; p < np + (solve ? 1 : 0); ++p) {
      const int c0 = kPanel * p, k0 = c0 - kPanel, q0 = k0 - kPanel;  // panels p, p - 1, p - 2
      if (rank && !dead && !bar_wait(smem_u32(pbar + p - 1), wait_limit, csize)) {
        if (lane == 0) info[node] = -1;
        dead = true;
      }
      if (rank == 0 && p > 0 && p < np && !(w & 3) && w <= 4 * kPanel) {
        const int c = c0 + (w >> 2) - 1;
        if (w > 0 && c < r) {
          const T *a = X3 + k0 * ld, *b = a + c;
          T *col = X3 + c * ld, m[kPanel];
#pragma unroll
          for (int q = 0; q < kPanel; ++q) m[q] = b[q * ld];
          acc_t<T> v[3];
#pragma unroll
          for (int s = 0; s < 3; ++s) {
            const int i = min(32 * s + lane, r - 1);
            v[s] = col[i];
            if (32 * s + 31 < c) continue;
#pragma unroll
            for (int q = 0; q < kPanel; ++q) v[s] -= a[i + q * ld] * m[q];
          }
#pragma unroll
          for (int s = 0; s < 3; ++s)
            if (32 * s + lane >= c && 32 * s + lane < r) col[32 * s + lane] = T(v[s].s, v[s].c);
        }
        asm volatile("bar.sync 1, 160;" ::: "memory");  // (warps 0, 4, 8, 12, 16)
      }
      if (w == 0) {
        if (rank == 0 && p < np) switch (nch - (c0 >> 5)) {
            case 1: chol_panel<1>(X3, r, c0, lane, bad); break;
            case 2: chol_panel<2>(X3, r, c0, lane, bad); break;
            default: chol_panel<3>(X3, r, c0, lane, bad);
          }
        if (rank == 0 && p < np && csize > 1 && solve) {
          // the panel with its reciprocal pivots to the other CTAs, a copy each
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane > 0 && lane < csize) {
            const unsigned src = smem_u32(X3 + c0 * ld), n = min(kPanel, r - c0) * ld * sizeof(T);
            copy_to_rank(at_rank(src, lane), src, n, at_rank(smem_u32(pbar + p), lane));
          }
        }
      } else if (w < 4) {
        if (solve && p > 0 && tid - 32 < nown) {
          T* b = X2 + (cfirst + cstep * (tid - 32)) * ld;
          const T* l = X3 + k0;
          T y[kPanel];
          acc_t<T> acc[kPanel];
#pragma unroll
          for (int j = 0; j < kPanel; ++j) acc[j] = b[min(k0 + j, r - 1)];
          if (p >= 2) {
#pragma unroll
            for (int q = 0; q < kPanel; ++q) y[q] = b[q0 + q];
#pragma unroll
            for (int j = 0; j < kPanel; ++j) {
              if ((k0 & 7) && k0 > kPanel) acc[j] = accv(acc[j]);
#pragma unroll
              for (int q = 0; q < kPanel; ++q) acc[j] -= l[j + (q0 + q) * ld] * y[q];
              if (!(k0 & 7)) acc[j] = accv(acc[j]);
            }
          }
#pragma unroll
          for (int j = 0; j < kPanel; ++j) {
            if (k0 + j >= r) break;
#pragma unroll
            for (int q = 0; q < j; ++q) acc[j] -= l[j + (k0 + q) * ld] * y[q];
            y[j] = accv(acc[j]) * l[kPivotRow - k0 + (k0 + j) * ld];
          }
#pragma unroll
          for (int j = 0; j < kPanel; ++j)
            if (k0 + j < r) {
              b[k0 + j] = y[j];
              if (csize > 1) put_rank0(b + k0 + j, y[j], csize);
            }
        }
      } else if (wid >= 0) {
        const int cc = c0 + kPanel;
        if (rank == 0 && p > 0 && cc < r) {
          for (int e = cc * r - cc * (cc - 1) / 2 + id; e < r * (r + 1) / 2; e += nid) {
            const int i = tab[e] & 255, c = tab[e] >> 8;
            const T *a = X3 + i + k0 * ld, *b = X3 + c + k0 * ld;
            acc_t<T> v = X3[i + c * ld];
#pragma unroll
            for (int q = 0; q < kPanel; ++q) v -= a[q * ld] * b[q * ld];
            X3[i + c * ld] = T(v.s, v.c);
          }
        }
        if (nown > 0 && solve && p >= 2 && c0 < r) {
          // two columns at a time, which share the loads of L22
          const int m = r - c0, dl = nid / m, di = nid - dl * m;
          int lc = id / m, i = id - lc * m;
          while (2 * lc < nown) {
            T* b0 = X2 + (cfirst + cstep * 2 * lc) * ld + q0;
            T* b1 = 2 * lc + 1 < nown ? b0 + cstep * ld : b0;
            const T* l = X3 + c0 + i + q0 * ld;
            acc_t<T> u = b0[2 * kPanel + i], v = b1[2 * kPanel + i];
#pragma unroll
            for (int q = 0; q < kPanel; q += 2) {
              const ffpair x = two(b0 + q), y = two(b1 + q);
              const T l0 = l[q * ld], l1 = l[(q + 1) * ld];
              u -= l0 * x.a;
              v -= l0 * y.a;
              u -= l1 * x.b;
              v -= l1 * y.b;
            }
            b0[2 * kPanel + i] = T(u.s, u.c);
            if (b1 != b0) b1[2 * kPanel + i] = T(v.s, v.c);
            i += di;
            lc += dl;
            if (i >= m) {
              i -= m;
              ++lc;
            }
          }
        }
      }
      __syncthreads();
    }
    if (tid == 0 && bad && info[node] == 0) info[node] = bad;
    if (csize > 1 && solve) {
      // after a wait that gave up: all panels have arrived (all are sent), so that nothing is on its way
      // to this CTA when it leaves
      if (dead)
        for (int p = 0; p < np; ++p) bar_wait(smem_u32(pbar + p), -1, csize);
      node_barrier(csize);
      if (rank != 0) return;
    }
  }
  // store Ct and L22
  for (int c = w; c < r; c += nw)
    for (int i = lane; i < r; i += 32) {
      const int64_t e = node * (int64_t)r * r + i + (int64_t)c * r;
      Ct_out[e] = X0[i + c * ld];
      L22_out[e] = (i >= c) ? X3[i + c * ld] : T(0.0);
    }
  if (level >= L) return;
  // structured Householder QR of [X1 (upper r x r) ; X2 (r x r)]: reflector j acts on row j of
  // the top and all r rows of the bottom.  Dataflow over columns: column c belongs to the group
  // of 8 lanes c & 3 of warp c >> 2 (lane q of the group holds bottom rows q, q+8, ..., so a dot
  // product is a 3-level shuffle reduction) and stays in registers.  A warp applies reflectors
  // 0, 1, ... to its four columns as they are published; when the next reflector is formed from
  // one of its own columns it forms it at once and publishes it (the unscaled vector into
  // X2[:, j], beta, scale and tau into va, vb, vc, then flag[j]).  No block barrier inside the
  // loop; three of four handoffs stay inside a warp.  The betas and the scaling of the reflector
  // columns are applied in the output loop.
  const int gq = lane & 7, grp = lane >> 3;
  const int rpl = (r + 7) >> 3;  // rows per lane (<= 10 for r <= 80)
  auto gsum = [&](T x) {
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) x = x + shfl_xor(x, o);
    return x;
  };
  if (w < ((r + 3) >> 2)) {
    volatile int* vflag = flags;
    const int c0 = 4 * w, cmine = c0 + grp;  // this group's column (may be >= r on the last warp)
    const int clast = min(c0 + 3, r - 1);
    T x[10];
#pragma unroll
    for (int t = 0; t < 10; ++t) {
      const int i = gq + 8 * t;
      x[t] = (t < rpl && i < r && cmine < r) ? X2[i + cmine * ld] : T(0.0);
    }
    bool timed_out = false;
    for (int j = 0; j <= clast; ++j) {
      if (j >= c0) {
        // reflector j from this warp's column j (group j - c0); every group computes its own
        // column's norm alike, the owning group publishes
        acc_t<T> part{};
#pragma unroll
        for (int t = 0; t < 10; ++t) part += x[t] * x[t];
        const T sig = gsum(accv(part));
        const T alpha = X1[j + j * ld];
        T tj = T(0.0), beta = alpha, scal = T(0.0);
        if (sig != 0.0) {
          const T nrm = sqrt(alpha * alpha + sig);
          beta = alpha >= 0.0 ? -nrm : nrm;
          tj = (beta - alpha) * ff_recip(beta);
          scal = ff_recip(alpha - beta);
        }
        if (cmine == j) {
#pragma unroll
          for (int t = 0; t < 10; ++t) {
            const int i = gq + 8 * t;
            if (t < rpl && i < r) X2[i + j * ld] = x[t];
          }
          if (gq == 0) {
            va[j] = beta;
            vb[j] = scal;
            vc[j] = tj;
            Etau[node * (int64_t)r + j] = tj;
          }
        }
        __threadfence_block();
        __syncwarp();
        if (lane == 0) vflag[j] = 1;
      } else if (!timed_out) {
        int spins = 0;
        // only the warp that owns column j + 1 forms the next reflector; the others nap between
        // polls so that their polls do not take issue slots from it
        const bool nap = j + 1 < c0;
        while (wait_limit == 0 || vflag[j] == 0) {
          if (++spins > lim) {
            if (lane == 0) info[node] = -1;
            timed_out = true;
            break;
          }
          if (nap) __nanosleep(32);
        }
        __threadfence_block();
      }
      // apply reflector j to this warp's columns c > j
      if (j < clast) {
        const T tj = vc[j];
        if (tj != 0.0) {
          const T scal = vb[j];
          T v[10];
#pragma unroll
          for (int t = 0; t < 10; ++t) {
            const int i = gq + 8 * t;
            v[t] = (t < rpl && i < r) ? X2[i + j * ld] : T(0.0);
          }
          acc_t<T> dacc{};
#pragma unroll
          for (int t = 0; t < 10; ++t) dacc += v[t] * x[t];
          const bool live = cmine > j && cmine < r;
          const T top = live ? X1[j + cmine * ld] : T(0.0);
          const T acc = (gsum(accv(dacc)) * scal + top) * tj;
          if (live) {
            if (gq == 0) X1[j + cmine * ld] = top - acc;
            const T f = acc * scal;
#pragma unroll
            for (int t = 0; t < 10; ++t) x[t] -= f * v[t];
          }
        }
      }
    }
  }
  __syncthreads();
  T* Rn = R + (nleaf + node) * (int64_t)r * r;
  for (int c = w; c < r; c += nw)
    for (int i = lane; i < r; i += 32) {
      const int64_t e = i + (int64_t)c * r;
      Rn[e] = (i < c) ? X1[i + c * ld] : (i == c ? va[c] : T(0.0));
      Eref[node * (int64_t)r * r + e] = X2[i + c * ld] * vb[c];
    }
}

// Sc^{-T} (upper triangular) from the landmark Cholesky factor Sc (lower): X = Sc^{-1} by forward
// substitution on all r columns at once, one CTA with Sc and the right-hand sides in shared
// memory.  At step l the columns j <= l take x[l][j] = b[l][j] / Sc[l][l], then the rows i > l of
// those columns take b[i][j] -= Sc[i][l] x[l][j].  Every x[i][j] sees the operations of the
// row-by-row substitution of its column in the same order (b = e_j; l = j, ..., i - 1; one
// division), two barriers a row instead of a serial chain of r^2 / 2 steps per thread.
__global__ void k_tri_inv_t(const double* __restrict__ Sc, int r, double* __restrict__ SinvT) {
  extern __shared__ double s[];
  const int ld = r + 1;
  double* L = s;           // Sc, element (i, c) at i + c * ld
  double* B = s + r * ld;  // right-hand sides, then X
  const int tid = threadIdx.x, nth = blockDim.x;
  for (int e = tid; e < r * r; e += nth) {
    const int i = e % r, c = e / r;
    L[i + c * ld] = Sc[e];
    B[i + c * ld] = (i == c) ? 1.0 : 0.0;
  }
  __syncthreads();
  for (int l = 0; l < r; ++l) {
    for (int j = tid; j <= l; j += nth) B[l + j * ld] = B[l + j * ld] / L[l + l * ld];
    __syncthreads();
    const int w = r - 1 - l;
    for (int e = tid; e < w * (l + 1); e += nth) {
      const int i = l + 1 + e % w, j = e / w;
      B[i + j * ld] -= L[i + l * ld] * B[l + j * ld];
    }
    __syncthreads();
  }
  for (int e = tid; e < r * r; e += nth) {
    const int j = e % r, i = e / r;  // SinvT[j + i r] = X[i][j] for i >= j
    SinvT[e] = (i >= j) ? B[i + j * ld] : 0.0;
  }
}

// ---------------------------------------------------------------------------------------------
// log det: 2 sum log diag(L_leaf) + 2 sum log |diag(L22)|, deterministic two-pass reduction.
// ---------------------------------------------------------------------------------------------
template <typename T>
__global__ void k_logdet_partial(const T* __restrict__ Lf, DTree t, const T* __restrict__ L22,
                                 int r, int64_t nnode, double* __restrict__ partial) {
  __shared__ double red[8];
  const int64_t nleafdiag = t.n;
  const int64_t tot = nleafdiag + nnode * r;
  double acc = 0.0;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < tot;
       e += (int64_t)gridDim.x * blockDim.x) {
    T d;
    if (e < nleafdiag) {
      // leaf containing row e
      const int64_t big = t.rem * (t.m0 + 1);
      const int64_t j = e < big ? e / (t.m0 + 1) : t.rem + (e - big) / t.m0;
      const int64_t i = e - d_leaf_start(t, j);
      const int m = d_leaf_size(t, j);
      d = Lf[d_leaf_koff(t, j) + i * m + i];
    } else {
      const int64_t q = e - nleafdiag;
      const int64_t node = q / r, i = q % r;
      d = L22[node * (int64_t)r * r + i * r + i];
    }
    acc += 2.0 * log(fabs(to_double(d)));
  }
  acc = warp_sum(acc);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) s += red[q];
    partial[blockIdx.x] = s;
  }
}

__global__ void k_sum_partials(const double* __restrict__ partial, int np, double* __restrict__ out) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    double s = 0.0;
    for (int q = 0; q < np; ++q) s += partial[q];
    out[0] = s;
  }
}

void launch_sum_partials(const double* partial, int np, double* out, cudaStream_t st) {
  k_sum_partials<<<1, 32, 0, st>>>(partial, np, out);
}

// ---------------------------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------------------------
bool launch_chol_small(double* A, int n, int* info, cudaStream_t st) {
  const size_t sm = (size_t)n * (n + 1) * sizeof(double);
  if (sm > 200 * 1024) return false;
  smem_limit((const void*)k_chol_small, sm);
  k_chol_small<<<1, 256, sm, st>>>(A, n, info);
  return true;
}

template <typename T, int NB>
static void leaf_chol_launch(const double* K, T* Lf, const Tree& t, int* info, cudaStream_t st) {
  constexpr int NT = 256;
  const size_t sm = (size_t)(t.max_leaf + NB) * (NB + 1) * sizeof(T);
  smem_limit((const void*)k_leaf_chol<T, NB, NT>, sm);
  k_leaf_chol<T, NB, NT><<<(unsigned)t.nleaf, NT, sm, st>>>(K, Lf, dtree(t), info);
}

template <typename T>
bool launch_leaf_chol(const double* K, T* Lf, const Tree& t, int* info, cudaStream_t st) {
  const int64_t m = t.max_leaf;
  auto fits = [&](int nb) { return (size_t)(m + nb) * (nb + 1) * sizeof(T) <= 200 * 1024; };
  // (float pairs need twice the registers per value: the widest panel is 16 columns)
  if (fits(16)) {
    leaf_chol_launch<T, 16>(K, Lf, t, info, st);
  } else if (fits(8)) {
    leaf_chol_launch<T, 8>(K, Lf, t, info, st);
  } else {
    return false;
  }
  return true;
}

template <typename T>
void launch_leaf_qr(T* Pan, int r, const Tree& t, T* tau, T* Rout, int* info, int wait_limit, cudaStream_t st) {
  const unsigned nth = 32 * leaf_qr_warps<T>();
  const size_t sm = (size_t)t.max_leaf * r * sizeof(T);
  if (sm <= 200 * 1024) {
    smem_limit((const void*)k_leaf_qr<T, true>, sm);
    k_leaf_qr<T, true><<<(unsigned)t.nleaf, nth, sm, st>>>(Pan, r, dtree(t), tau, Rout, info, wait_limit);
  } else {
    k_leaf_qr<T, false><<<(unsigned)t.nleaf, nth, 0, st>>>(Pan, r, dtree(t), tau, Rout, info, wait_limit);
  }
}

void launch_tri_inv_t(const double* Sc, int r, double* SinvT, cudaStream_t st) {
  const size_t sm = (size_t)2 * r * (r + 1) * sizeof(double);
  smem_limit((const void*)k_tri_inv_t, sm);
  k_tri_inv_t<<<1, 512, sm, st>>>(Sc, r, SinvT);
}

// SM count of the current device (cached per device)
static int sm_count() {
  constexpr int kDevMax = 64;
  static std::atomic<int> nsm_of[kDevMax];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevMax) return 1;
  int v = nsm_of[dev].load();
  if (v == 0) {
    int nsm = 0;
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    v = nsm > 0 ? nsm : 1;
    nsm_of[dev].store(v);
  }
  return v;
}

// CTAs per node of the node kernels (form 0: FP64, 1: float pairs): the largest of 8, 4, 2 with
// nodes x csize <= the SM count and as many such clusters schedulable at once (asked once per form,
// device, size and number of CTAs that an SM's shared memory holds: clusters do not straddle the groups
// that SMs come in, so 16 of 8 may not fit 152 SMs), else 1.  max_cs (the handle's setting) and KM_NODE_CLUSTER=1, 2, 4 or 8 cap it
// (1 gives the one-CTA form).
static int node_cluster_size(int form, const void* fn, int64_t nodes, int threads, size_t smem, int max_cs) {
  static const int cap = [] {
    const char* e = std::getenv("KM_NODE_CLUSTER");
    const int v = e ? std::atoi(e) : 8;
    return v >= 8 ? 8 : v >= 4 ? 4 : v >= 2 ? 2 : 1;
  }();
  constexpr int kDevMax = 64;
  // per form, device, size 1, 2, 4, 8 and CTAs an SM by shared memory (1, 2, 3, 4 and more): clusters at
  // once, 0 unknown, -1 none (handles on several host threads may ask at once; a repeated query gives the
  // same answer)
  static std::atomic<int> room[2][kDevMax][4][4];
  const int per_sm = (int)std::min<size_t>(std::max<size_t>(228 * 1024 / (smem + 1024), 1), 4);
  const int nsm = sm_count();
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevMax) return 1;
  const int top = std::min(cap, max_cs);
  for (int cs = top, lg = top >= 8 ? 3 : top == 4 ? 2 : top == 2 ? 1 : 0; cs > 1; cs >>= 1, --lg) {
    if (nodes * cs > nsm) continue;
    std::atomic<int>& n = room[form][dev][lg][per_sm - 1];
    if (n.load() == 0) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3((unsigned)cs);
      cfg.blockDim = dim3((unsigned)threads);
      cfg.dynamicSmemBytes = smem;
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = (unsigned)cs;
      at[0].val.clusterDim.y = 1;
      at[0].val.clusterDim.z = 1;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      int nclusters = 0;
      const cudaError_t e = cudaOccupancyMaxActiveClusters(&nclusters, fn, &cfg);
      if (e != cudaSuccess) cudaGetLastError();  // clear the query's error; the size is not used
      n.store((e == cudaSuccess && nclusters > 0) ? nclusters : -1);
    }
    if (n.load() >= nodes) return cs;
  }
  return 1;
}

template <typename T>
void launch_node_factor(T* R, const T* SinvT, int r, int level, const Tree& t, T* Ct, T* L22, T* Eref,
                        T* Etau, int* info, cudaStream_t st, int max_cluster, int wait_limit) {
  if constexpr (std::is_same<T, double>::value) {
    const size_t sm = node_f64_smem(r);
    smem_limit(node_f64_kernel(), sm);
    const int64_t nodes = t.nodes_at(level);
    const int cs = node_cluster_size(0, node_f64_kernel(), nodes, 256, sm, max_cluster);
    if (cs > 1) {
      const cudaError_t prior = cudaPeekAtLastError();
      if (launch_node_f64(R, SinvT, r, level, t, Ct, L22, Eref, Etau, info, cs, wait_limit, st) == cudaSuccess) return;
      // the cluster launch was refused (nothing ran): one CTA per node instead; an error from
      // before this launch stays for the caller
      if (prior == cudaSuccess) cudaGetLastError();
    }
    launch_node_f64(R, SinvT, r, level, t, Ct, L22, Eref, Etau, info, 1, wait_limit, st);
  } else {
    const int64_t cbase = (level == 1) ? 0 : t.nleaf + t.node_off[level - 1];
    const int64_t nbase = t.node_off[level];
    const size_t sm = ((size_t)4 * r * kNodeLd + 3 * r + (r + kPanel - 1) / kPanel) * sizeof(T) + (size_t)r * sizeof(int) +
                      (size_t)r * (r + 1) / 2 * sizeof(unsigned short);
    smem_limit((const void*)k_node_factor<T>, sm);
    const int64_t nodes = t.nodes_at(level);
    const int cs = node_cluster_size(1, (const void*)k_node_factor<T>, nodes, kNodeThreads, sm, max_cluster);
    if (cs > 1) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3((unsigned)(nodes * cs));
      cfg.blockDim = dim3(kNodeThreads);
      cfg.dynamicSmemBytes = sm;
      cfg.stream = st;
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = (unsigned)cs;
      at[0].val.clusterDim.y = 1;
      at[0].val.clusterDim.z = 1;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      const cudaError_t prior = cudaPeekAtLastError();
      if (cudaLaunchKernelEx(&cfg, k_node_factor<T>, R, SinvT, r, level, t.L, t.nleaf, cbase, nbase, Ct, L22, Eref,
                             Etau, info, cs, wait_limit) == cudaSuccess)
        return;
      // the cluster launch was refused (nothing ran): one CTA per node instead; an error from
      // before this launch stays for the caller
      if (prior == cudaSuccess) cudaGetLastError();
    }
    {
      k_node_factor<T><<<(unsigned)nodes, kNodeThreads, sm, st>>>(R, SinvT, r, level, t.L, t.nleaf, cbase, nbase, Ct, L22,
                                                          Eref, Etau, info, 1, wait_limit);
    }
  }
}

template <typename T>
void launch_logdet(const T* Lf, const Tree& t, const T* L22, int r, double* partial, int np, double* out,
                   cudaStream_t st) {
  k_logdet_partial<T><<<np, 256, 0, st>>>(Lf, dtree(t), L22, r, t.nnode, partial);
  k_sum_partials<<<1, 32, 0, st>>>(partial, np, out);
}

// double -> float pair conversion of n values (in place allowed: same 8-byte slots)
__global__ void k_to_ff(const double* __restrict__ in, ff* __restrict__ out, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = ff(in[i]);
}
__global__ void k_from_ff(const ff* __restrict__ in, double* __restrict__ out, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = (double)in[i];
}
void launch_to_ff(const double* in, ff* out, int64_t n, cudaStream_t st) {
  k_to_ff<<<(unsigned)std::min<int64_t>((n + 255) / 256, 4096), 256, 0, st>>>(in, out, n);
}
void launch_from_ff(const ff* in, double* out, int64_t n, cudaStream_t st) {
  k_from_ff<<<(unsigned)std::min<int64_t>((n + 255) / 256, 4096), 256, 0, st>>>(in, out, n);
}


// Solve operators of the nodes of one level, formed off the critical path (side stream):
// L22^{-1} (lower) and the explicit transfer E = H_0 ... H_{r-1} [I; 0] (2r x r) from the
// reflectors of QR(G_N).  One CTA per node; columns are independent.
// Per node of one level: L22^{-1} (lower) and, below the root, the explicit 2r x r factor E
// of G = E R_N from the structured reflectors.  One warp per column; the column lives in
// registers (row i in lane i % 32, slot i / 32, r <= 96), so the dependent chains need no
// block barriers.  Column c's two chains take r - c and c + 1 steps, r + 1 together, so every
// column costs the same; gridDim.y CTAs share a node's columns (warp w of CTA y takes columns
// y * nw + w, stepping gridDim.y * nw), enough on levels with few nodes for one column per warp.
// Runs on the side stream, overlapped with the next level's node kernel.
template <typename T>
__device__ __forceinline__ T slot_get(const T (&x)[3], int s) {
  return s == 0 ? x[0] : (s == 1 ? x[1] : x[2]);
}

template <typename T>
__global__ void __launch_bounds__(512) k_node_finalize(const T* __restrict__ L22, const T* __restrict__ Ct,
                                                       const T* __restrict__ Eref, const T* __restrict__ Etau, int r,
                                                       int64_t nbase, int with_e, T* __restrict__ L22i,
                                                       T* __restrict__ Eexp, T* __restrict__ CtT,
                                                       T* __restrict__ L22T, T* __restrict__ L22iT,
                                                       T* __restrict__ ET) {
  extern __shared__ __align__(16) unsigned char smraw[];
  T* sm = reinterpret_cast<T*>(smraw);
  const int ld = r + 1;
  T* Ls = sm;               // L22
  T* Vs = Ls + r * ld;      // reflector bottoms
  T* Cs = Vs + r * ld;      // Ct
  T* ts = Cs + r * ld;      // tau
  const int64_t node = nbase + blockIdx.x;
  const int64_t off = node * (int64_t)r * r;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nw = blockDim.x >> 5;
  const int c0 = (int)blockIdx.y * nw + w, cstep = (int)gridDim.y * nw;  // this warp's columns
  for (int e = tid; e < r * r; e += blockDim.x) {
    const int i = e % r, c = e / r;
    Ls[i + c * ld] = L22[off + e];
    Cs[i + c * ld] = Ct[off + e];
    if (with_e) Vs[i + c * ld] = Eref[off + e];
  }
  if (with_e)
    for (int e = tid; e < r; e += blockDim.x) ts[e] = Etau[node * (int64_t)r + e];
  __syncthreads();
  // transposes of Ct and L22 for the sweeps (entries split over the node's CTAs)
  for (int e = (int)blockIdx.y * blockDim.x + tid; e < r * r; e += (int)gridDim.y * blockDim.x) {
    const int i = e % r, c = e / r;
    CtT[off + e] = Cs[c + i * ld];
    L22T[off + e] = Ls[c + i * ld];
  }
  // L22^{-1} e_c by forward substitution in column (axpy) order: row i accumulates
  // -L[i,p] x_p for p = c .. i-1 and is then divided by L[i,i]
  for (int c = c0; c < r; c += cstep) {
    T x[3];
#pragma unroll
    for (int s = 0; s < 3; ++s) x[s] = (lane + 32 * s) == c ? T(1.0) : T(0.0);
    for (int p = c; p < r; ++p) {
      const T xp = shfl_idx(slot_get(x, p >> 5), p & 31) / Ls[p + p * ld];
#pragma unroll
      for (int s = 0; s < 3; ++s) {
        const int i = lane + 32 * s;
        if (i == p) x[s] = xp;
        else if (i > p && i < r) x[s] -= Ls[i + p * ld] * xp;
      }
    }
    T* out = L22i + off + (int64_t)c * r;
#pragma unroll
    for (int s = 0; s < 3; ++s) {
      const int i = lane + 32 * s;
      if (i < r) {
        out[i] = x[s];
        L22iT[off + c + (int64_t)i * r] = x[s];
      }
    }
  }
  if (!with_e) return;
  // column c of E: H_c ... H_0 applied in turn (j = c down to 0) to [e_c ; 0]; H_j acts on
  // top row j and the whole bottom, so top row j is final once H_j has acted
  T* Eo = Eexp + node * (int64_t)2 * r * r;
  T* Et = ET + node * (int64_t)2 * r * r;  // r x 2r: element (c, l) at c + l*r
  for (int c = c0; c < r; c += cstep) {
    T* top = Eo + (int64_t)c * 2 * r;
    T* bot = top + r;
    T b[3] = {T(0.0), T(0.0), T(0.0)};
    for (int i = c + 1 + lane; i < r; i += 32) {
      top[i] = T(0.0);
      Et[c + (int64_t)i * r] = T(0.0);
    }
    for (int j = c; j >= 0; --j) {
      const T tj = ts[j];
      const T tjtop = j == c ? T(1.0) : T(0.0);
      if (tj == 0.0) {
        if (lane == 0) {
          top[j] = tjtop;
          Et[c + (int64_t)j * r] = tjtop;
        }
        continue;
      }
      T part = T(0.0);
#pragma unroll
      for (int s = 0; s < 3; ++s) {
        const int i = lane + 32 * s;
        if (i < r) part += Vs[i + j * ld] * b[s];
      }
      const T acc = (tjtop + warp_sum_t(part)) * tj;
      if (lane == 0) {
        top[j] = tjtop - acc;
        Et[c + (int64_t)j * r] = tjtop - acc;
      }
#pragma unroll
      for (int s = 0; s < 3; ++s) {
        const int i = lane + 32 * s;
        if (i < r) b[s] -= acc * Vs[i + j * ld];
      }
    }
#pragma unroll
    for (int s = 0; s < 3; ++s) {
      const int i = lane + 32 * s;
      if (i < r) {
        bot[i] = b[s];
        Et[c + (int64_t)(r + i) * r] = b[s];
      }
    }
  }
}

// Explicit Q of a leaf panel in float pairs, m >= r.  Column c of Q = H_0 ... H_{r-1} [I; 0] is
// H_0 ... H_c e_c: a warp keeps NC columns in registers (RPL rows a lane) and applies the reflectors to
// them from the last to the first, without a barrier.  The columns go in groups of W NC from the
// right, each written over its reflectors once all warps have read these (the columns to the left need
// none of them).  In place in memory, with two barriers a reflector (k_leaf_formq), 512 panels of
// 488 x 72 took 3.0 ms, 256 of 256 x 72 0.50 ms; now 1.04 and 0.30 ms.  grid nleaf, block 32 W.
template <int RPL, int NC, int W>
__global__ void __launch_bounds__(32 * W) k_leaf_formq_reg(ff* __restrict__ Pan, const ff* __restrict__ tau, int r, DTree t) {
  const int64_t leaf = blockIdx.x;
  const int m = d_leaf_size(t, leaf);
  ff* G = Pan + d_leaf_start(t, leaf) * r;
  const ff* tl = tau + leaf * r;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int c1 = r; c1 > 0; c1 -= W * NC) {
    const int hi = c1 - 1 - NC * w;  // columns hi, hi - 1, ..
    ff x[NC][RPL];
#pragma unroll
    for (int u = 0; u < NC; ++u)
#pragma unroll
      for (int q = 0; q < RPL; ++q) x[u][q] = ff(lane + 32 * q == hi - u ? 1.f : 0.f, 0.f);
    for (int j = hi; j >= 0; --j) {
      const ff tj = tl[j];
      const ff* vj = G + (int64_t)j * m;
      ff v[RPL];
#pragma unroll
      for (int q = 0; q < RPL; ++q) {
        const int i = lane + 32 * q;
        v[q] = i > j && i < m ? vj[i] : ff(i == j ? 1.f : 0.f, 0.f);
      }
      ff a[NC];
#pragma unroll
      for (int u = 0; u < NC; ++u) {
        acc_t<ff> acc{};
#pragma unroll
        for (int q = 0; q < RPL; ++q) acc += v[q] * x[u][q];
        a[u] = accv(acc);
      }
      // sums over the lanes: while more than one column is left a lane passes on half of them
      int o = 16;
#pragma unroll
      for (int h = NC / 2; h > 0; h >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int u = 0; u < h; ++u) {
          const ff keep = up ? a[u + h] : a[u], pass = up ? a[u] : a[u + h];
          a[u] = keep + shfl_xor(pass, o);
        }
      }
      ff sum = a[0];
      for (; o > 0; o >>= 1) sum = sum + shfl_xor(sum, o);
      sum = sum * tj;
#pragma unroll
      for (int u = 0; u < NC; ++u) {
        const ff f = shfl_idx(sum, NC == 4 ? (u >> 1) * 16 + (u & 1) * 8 : NC == 2 ? 16 * u : 0);
#pragma unroll
        for (int q = 0; q < RPL; ++q) x[u][q] -= f * v[q];
      }
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < NC; ++u)
      if (hi - u >= 0)
#pragma unroll
        for (int q = 0; q < RPL; ++q)
          if (lane + 32 * q < m) G[(int64_t)(hi - u) * m + lane + 32 * q] = x[u][q];
  }
}

template <typename T>
void launch_leaf_formq(T* Pan, const T* tau, int r, const Tree& t, cudaStream_t st) {
  if constexpr (std::is_same<T, ff>::value) {
    if (t.max_leaf > r && t.max_leaf <= 1024) {  // (leaf sizes differ by one at most)
      const unsigned nl = (unsigned)t.nleaf;
      if (t.max_leaf <= 256) k_leaf_formq_reg<8, 4, 16><<<nl, 512, 0, st>>>(Pan, tau, r, dtree(t));
      else if (t.max_leaf <= 512) k_leaf_formq_reg<16, 2, 16><<<nl, 512, 0, st>>>(Pan, tau, r, dtree(t));
      else k_leaf_formq_reg<32, 1, 8><<<nl, 256, 0, st>>>(Pan, tau, r, dtree(t));
      return;
    }
  }
  const size_t sm = (size_t)t.max_leaf * r * sizeof(T);
  if (sm <= 200 * 1024) {
    smem_limit((const void*)k_leaf_formq<T, true>, sm);
    k_leaf_formq<T, true><<<(unsigned)t.nleaf, 32 * leaf_qr_warps<T>(), sm, st>>>(Pan, tau, r, dtree(t));
  } else {
    k_leaf_formq<T, false><<<(unsigned)t.nleaf, 32 * leaf_qr_warps<T>(), 0, st>>>(Pan, tau, r, dtree(t));
  }
}

template <typename T>
void launch_node_finalize(const T* L22, const T* Ct, const T* Eref, const T* Etau, int r, int level, const Tree& t,
                          T* L22i, T* Eexp, T* CtT, T* L22T, T* L22iT, T* ET, cudaStream_t st) {
  const size_t sm = ((size_t)3 * r * (r + 1) + r) * sizeof(T);
  smem_limit((const void*)k_node_finalize<T>, sm);
  // CTAs per node: enough for one column per warp (16 warps per CTA) while nodes x CTAs stays
  // within the SM count; one per node on the wide levels
  const int64_t nodes = t.nodes_at(level);
  const int nsm = sm_count();
  const int per_node = (int)std::max<int64_t>(1, std::min<int64_t>((r + 15) / 16, nsm / std::max<int64_t>(nodes, 1)));
  k_node_finalize<T><<<dim3((unsigned)nodes, (unsigned)per_node), 512, sm, st>>>(
      L22, Ct, Eref, Etau, r, t.node_off[level], level < t.L ? 1 : 0, L22i, Eexp, CtT, L22T, L22iT, ET);
}

template void launch_leaf_formq<double>(double*, const double*, int, const Tree&, cudaStream_t);
template void launch_leaf_formq<ff>(ff*, const ff*, int, const Tree&, cudaStream_t);
template void launch_node_finalize<double>(const double*, const double*, const double*, const double*, int, int,
                                           const Tree&, double*, double*, double*, double*, double*, double*,
                                           cudaStream_t);
template void launch_node_finalize<ff>(const ff*, const ff*, const ff*, const ff*, int, int, const Tree&, ff*, ff*,
                                       ff*, ff*, ff*, ff*, cudaStream_t);

template bool launch_leaf_chol<ff>(const double*, ff*, const Tree&, int*, cudaStream_t);
template void launch_leaf_qr<double>(double*, int, const Tree&, double*, double*, int*, int, cudaStream_t);
template void launch_leaf_qr<ff>(ff*, int, const Tree&, ff*, ff*, int*, int, cudaStream_t);
template void launch_node_factor<double>(double*, const double*, int, int, const Tree&, double*, double*, double*,
                                         double*, int*, cudaStream_t, int, int);
template void launch_node_factor<ff>(ff*, const ff*, int, int, const Tree&, ff*, ff*, ff*, ff*, int*, cudaStream_t,
                                     int, int);
template void launch_logdet<double>(const double*, const Tree&, const double*, int, double*, int, double*, cudaStream_t);
template void launch_logdet<ff>(const ff*, const Tree&, const ff*, int, double*, int, double*, cudaStream_t);

}  // namespace km
