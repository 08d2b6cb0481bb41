// Householder QR with explicit Q of batches of panels (m x k, FP64), used on the U and V panels of
// the general factorisation (lrsymfact's qr calls, src/HODLR/src/utils.jl:29-35).
//
// Reflector blocks of 32 columns (LAPACK dgeqrf / dorgqr structure, compact-WY).  Per block:
//   k_pqr_factor  one cluster per panel: the block's rows are spread over the CTAs' shared memory,
//                 one cluster barrier per column; its T factor and the product T V_top'
//   k_pqr_vtc     partial products V' C of the trailing columns, over (tile, row chunk) CTAs
//   k_pqr_apply   C -= V (op(T) V' C), over (row chunk, tile) CTAs
// and for Q, from the last block to the first, k_pqr_vtc and k_pqr_apply on the columns formed
// already and k_pqr_form on the block's own, Q = E - V (T V_top') without a column recurrence.
//
// Two multiply-adds a clock and SM bound the updates, the column chain (a reduction, a square root
// and two divisions, 580 cycles each) the factor step.  With 8-column blocks factored by one CTA
// from global memory and 8-column update tiles, the panels of a 2^14 matrix (2 x 8192 x 350 at the
// top) took 191 ms, now 37 ms.
#include <cooperative_groups.h>

#include <algorithm>

#include "km_kernels.h"

namespace km {

namespace cg = cooperative_groups;

namespace {

constexpr int kPB = 32;          // columns of a reflector block
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kRowsMax = 768;    // rows of a block that one CTA holds (32 x 769 doubles)
constexpr int kVtcRows = 512;    // most rows of one V' C partial product
constexpr int kApplyRows = 256;  // most rows of one update CTA

// Sums v[0..4) over the warp; lanes 8 b (b = 0..3) return the sum of v[2 b1 + b0] with b1, b0 the
// lane's bits 4 and 3.
__device__ __forceinline__ double reduce4(double (&v)[4], int lane) {
#pragma unroll
  for (int h = 2, o = 16; h > 0; h >>= 1, o >>= 1) {
#pragma unroll
    for (int k = 0; k < h; ++k) {
      const bool up = (lane & o) != 0;
      const double keep = up ? v[k + h] : v[k], send = up ? v[k] : v[k + h];
      v[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  double s = v[0];
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// Block of columns j0 .. j0+jb-1, rows j0 .. m-1: CTA q of the panel's cluster holds rows
// [q rs, (q+1) rs) of it in shared memory (column c at P + c ldp).  At column j every CTA forms the
// dots of its rows below j of column j with all 32 columns (the norm, the products with the later
// columns for the update and with the earlier vectors for T) and, if it owns row j, that row;
// after the cluster barrier all CTAs add the parts in CTA order and form the same reflector
// (dlarfg: beta = -sign(alpha) ||.||).  The parts alternate between two buffers, so one barrier a
// column is enough.
__global__ void __launch_bounds__(kThreads) k_pqr_factor(const PanelDesc* __restrict__ descs, int j0,
                                                         double* __restrict__ Ts, int nblk, int rs, int CS) {
  extern __shared__ double P[];
  __shared__ double part[2][kPB], top[2][kPB], tot[kPB], trow[kPB], T[kPB * kPB], G[kPB], refl[3];
  // (a panel of one CTA is a plain launch: no cluster operations)
  const int g = (int)(blockIdx.x % CS);
  auto team_sync = [&]() {
    if (CS == 1) __syncthreads();
    else cg::this_cluster().sync();
  };
  auto at = [&](double* p, int q) { return CS == 1 ? p : cg::this_cluster().map_shared_rank(p, q); };
  const PanelDesc D = descs[blockIdx.x / CS];
  if (D.big || j0 >= D.k) return;  // the whole cluster leaves
  const int jb = min(kPB, D.k - j0), M = (int)D.m - j0;
  const int lo = min(M, g * rs), n = min(M, lo + rs) - lo, ldp = rs | 1;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  double* A = D.A + (int64_t)j0 * D.lda + j0 + lo;
  for (int c = w; c < jb; c += kWarps)
    for (int i = lane; i < n; i += 32) P[c * ldp + i] = A[(int64_t)c * D.lda + i];
  for (int e = tid; e < kPB * kPB; e += kThreads) T[e] = 0.0;
  __syncthreads();
  for (int j = 0; j < jb; ++j) {
    double* pt = part[j & 1];
    double* tp = top[j & 1];
    const double* pj = P + j * ldp;
    const int i0 = max(j + 1 - lo, 0);  // first local row below row j
    {
      // warp w: columns w, w + 8, w + 16, w + 24
      double v[4] = {};
      if (i0 < n) {
        for (int i = i0 + lane; i < n; i += 32) {
          const double x = pj[i];
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (w + 8 * u < jb) v[u] += x * P[(w + 8 * u) * ldp + i];
        }
      }
      const double s = reduce4(v, lane);
      const int c = w + 8 * (2 * ((lane >> 4) & 1) + ((lane >> 3) & 1));
      if ((lane & 7) == 0 && c < jb) pt[c] = s;
    }
    const bool own = j >= lo && j < lo + n;
    if (own && tid < jb) tp[tid] = P[tid * ldp + j - lo];
    team_sync();
    {
      // 8 lanes per column add the CTAs' parts
      const int c = tid >> 3, p = tid & 7;
      double s = 0.0;
      if (c < jb)
        for (int q = p; q < CS; q += 8) s += at(pt, q)[c];
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (p == 0 && c < jb) {
        tot[c] = s;
        trow[c] = at(tp, j / rs)[c];
      }
    }
    __syncthreads();
    if (w < 2) {  // two warps share the divisions
      const double sig = tot[j], alpha = trow[j];
      double beta = alpha, x = 0.0;
      if (sig != 0.0) {
        const double nrm = sqrt(alpha * alpha + sig);
        beta = alpha >= 0.0 ? -nrm : nrm;
        x = w == 0 ? (beta - alpha) / beta : 1.0 / (alpha - beta);
      }
      if (lane == 0) {
        refl[w] = x;
        if (w == 0) refl[2] = beta;
      }
    }
    __syncthreads();
    const double tau = refl[0], scal = refl[1];
    // H_j on the later columns: c -= tau (v . c) v with v = (1, scal x)
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int c = w + 8 * u;
      if (c > j && c < jb) {
        const double f = tau * (scal * tot[c] + trow[c]), fs = f * scal;
        if (own && lane == 0) P[c * ldp + j - lo] -= f;
        for (int i = i0 + lane; i < n; i += 32) P[c * ldp + i] -= fs * pj[i];
      }
    }
    if (g == 0 && w == 0) {  // T[:, j] = -tau T (V' v_j); entry j: tau
      if (lane < j) G[lane] = scal * tot[lane] + trow[lane];
      __syncwarp();
      double z = 0.0;
      if (lane < j)
        for (int l = lane; l < j; ++l) z += T[lane + l * kPB] * G[l];
      if (lane < j) T[lane + j * kPB] = -tau * z;
      if (lane == j) T[j + j * kPB] = tau;
      __syncwarp();
    }
    __syncthreads();
    if (own && tid == 0) P[j * ldp + j - lo] = refl[2];
    for (int i = i0 + tid; i < n; i += kThreads) P[j * ldp + i] *= scal;
    __syncthreads();
  }
  for (int c = w; c < jb; c += kWarps)
    for (int i = lane; i < n; i += 32) A[(int64_t)c * D.lda + i] = P[c * ldp + i];
  if (g == 0) {
    // T and T V_top' (V_top: the block's own rows of V, all in this CTA: rs >= 32 or M <= rs)
    double* out = Ts + ((int64_t)(blockIdx.x / CS) * nblk + j0 / kPB) * 2 * kPB * kPB;
    for (int e = tid; e < kPB * kPB; e += kThreads) {
      const int p = e % kPB, c = e / kPB;
      double z = 0.0;
      // V_top[c, q]: 1 at q = c, stored vectors at q < c
      for (int q = p; q <= c && q < jb; ++q) z += T[p + q * kPB] * (q == c ? 1.0 : (c < n ? P[q * ldp + c] : 0.0));
      out[e] = T[e];
      out[kPB * kPB + e] = z;
    }
  }
  team_sync();  // no CTA leaves while another may still read its parts
}

// Entry (i, p) of the block's V, rows counted from j0
__device__ __forceinline__ double v_entry(const double* A, int64_t lda, int i, int p, int M, int jb) {
  if (i >= M || p >= jb || i < p) return 0.0;
  return i == p ? 1.0 : A[(int64_t)p * lda + i];
}

// Wp[panel][chunk][c][p] = sum over the chunk's rows of V[i, p] C[i, c], c counted from the first
// trailing column j1: grid (panel, column tile of 32, row chunk).
__global__ void __launch_bounds__(kThreads) k_pqr_vtc(const PanelDesc* __restrict__ descs, int j0, double* __restrict__ Wp,
                                                      int kmax, int nchunk, int rows) {
  __shared__ double Vs[32 * 33], Cs[32 * 33];
  const PanelDesc D = descs[blockIdx.x];
  const int j1 = j0 + kPB, nt = D.k - j1, c0 = blockIdx.y * 32, M = (int)D.m - j0;
  const int r0 = blockIdx.z * rows, r1 = min(M, r0 + rows);
  if (D.big || c0 >= nt || r0 >= M) return;
  const double* V = D.A + (int64_t)j0 * D.lda + j0;
  const double* C = D.A + (int64_t)(j1 + c0) * D.lda + j0;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double acc[4] = {};  // p = lane, c = w + 8 q
  for (int i0 = r0; i0 < r1; i0 += 32) {
    __syncthreads();
    const int i = i0 + lane;
    for (int u = w; u < 32; u += kWarps) {
      Vs[lane * 33 + u] = v_entry(V, D.lda, i, u, r1, kPB);
      Cs[lane * 33 + u] = (i < r1 && c0 + u < nt) ? C[(int64_t)u * D.lda + i] : 0.0;
    }
    __syncthreads();
#pragma unroll 8
    for (int l = 0; l < 32; ++l) {
      const double x = Vs[l * 33 + lane];
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[q] += x * Cs[l * 33 + w + 8 * q];
    }
  }
  double* out = Wp + (((int64_t)blockIdx.x * nchunk + blockIdx.z) * kmax + c0) * kPB;
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (c0 + w + 8 * q < nt) out[(w + 8 * q) * kPB + lane] = acc[q];
}

// C -= V (op(T) W), W the sum of the partial products: grid (panel, column tile of 32, row chunk);
// transT = 1 while factoring (op(T) = T'), 0 while forming Q.
__global__ void __launch_bounds__(kThreads) k_pqr_apply(const PanelDesc* __restrict__ descs, int j0,
                                                        const double* __restrict__ Wp, const double* __restrict__ Ts,
                                                        int nblk, int kmax, int nchunk, int vrows, int rows,
                                                        int transT) {
  __shared__ double Vs[32 * 33], W[32 * 33], W2[32 * 33], Tm[32 * 33];
  const PanelDesc D = descs[blockIdx.x];
  const int j1 = j0 + kPB, nt = D.k - j1, c0 = blockIdx.y * 32, M = (int)D.m - j0;
  const int r0 = blockIdx.z * rows, r1 = min(M, r0 + rows);
  if (D.big || c0 >= nt || r0 >= M) return;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int nch = (M + vrows - 1) / vrows;
  const double* Tin = Ts + ((int64_t)blockIdx.x * nblk + j0 / kPB) * 2 * kPB * kPB;
  for (int u = w; u < 32; u += kWarps) {
    double s = 0.0;
    if (c0 + u < nt) {
      const double* in = Wp + ((int64_t)blockIdx.x * nchunk * kmax + c0 + u) * kPB + lane;
      for (int q = 0; q < nch; ++q) s += in[(int64_t)q * kmax * kPB];
    }
    W[lane * 33 + u] = s;  // (p, c)
    Tm[lane * 33 + u] = transT ? Tin[u + lane * kPB] : Tin[lane + u * kPB];  // op(T)(lane, u)
  }
  __syncthreads();
  {
    double acc[4] = {};
#pragma unroll 8
    for (int l = 0; l < 32; ++l) {
      const double x = Tm[lane * 33 + l];
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[q] += x * W[l * 33 + w + 8 * q];
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) W2[lane * 33 + w + 8 * q] = acc[q];
  }
  const double* V = D.A + (int64_t)j0 * D.lda + j0;
  double* C = D.A + (int64_t)(j1 + c0) * D.lda + j0;
  for (int i0 = r0; i0 < r1; i0 += 32) {
    const int i = i0 + lane;
    __syncthreads();
    for (int u = w; u < 32; u += kWarps) Vs[lane * 33 + u] = v_entry(V, D.lda, i, u, r1, kPB);
    __syncthreads();
    double acc[4] = {};
#pragma unroll 8
    for (int l = 0; l < 32; ++l) {
      const double x = Vs[lane * 33 + l];
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[q] += x * W2[l * 33 + w + 8 * q];
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int c = w + 8 * q;
      if (i < r1 && c0 + c < nt) C[(int64_t)c * D.lda + i] -= acc[q];
    }
  }
}

// R out of the factored panels (big: the panels of that kind)
__global__ void k_pqr_rout(const PanelDesc* __restrict__ descs, int big) {
  const PanelDesc D = descs[blockIdx.x];
  if ((D.big != 0) != (big != 0)) return;
  const int k = D.k;
  for (int e = blockIdx.y * blockDim.x + threadIdx.x; e < k * k; e += gridDim.y * blockDim.x) {
    const int i = e % k, c = e / k;
    D.R[e] = (i <= c) ? D.A[(int64_t)c * D.lda + i] : 0.0;
  }
}

// The block's own columns of Q: zeros above row j0, E - V (T V_top') below; grid (panel, row
// chunk), rows counted from the top of the panel.  A CTA reads V in its own rows only.
__global__ void __launch_bounds__(kThreads) k_pqr_form(const PanelDesc* __restrict__ descs, int j0,
                                                       const double* __restrict__ Ts, int nblk, int rows) {
  __shared__ double Vs[32 * 33], W2[32 * 33];
  const PanelDesc D = descs[blockIdx.x];
  const int m = (int)D.m, M = m - j0;
  const int r0 = blockIdx.y * rows, r1 = min(m, r0 + rows);
  if (D.big || j0 >= D.k || r0 >= m) return;
  const int jb = min(kPB, D.k - j0);
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const double* M2 = Ts + (((int64_t)blockIdx.x * nblk + j0 / kPB) * 2 + 1) * kPB * kPB;
  for (int u = w; u < 32; u += kWarps) W2[lane * 33 + u] = M2[lane + u * kPB];
  double* A = D.A + (int64_t)j0 * D.lda;
  for (int i0 = r0; i0 < r1; i0 += 32) {
    const int i = i0 + lane;  // panel row; block row i - j0
    __syncthreads();
    for (int u = w; u < 32; u += kWarps)
      Vs[lane * 33 + u] = (i < r1 && i >= j0) ? v_entry(A + j0, D.lda, i - j0, u, M, jb) : 0.0;
    __syncthreads();
    double acc[4] = {};
#pragma unroll 8
    for (int l = 0; l < 32; ++l) {
      const double x = Vs[lane * 33 + l];
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[q] += x * W2[l * 33 + w + 8 * q];
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int c = w + 8 * q;
      if (i < r1 && c < jb) A[(int64_t)c * D.lda + i] = i < j0 ? 0.0 : (i - j0 == c ? 1.0 : 0.0) - acc[q];
    }
  }
}

}  // namespace

static int pqr_cluster_limit() {
  return cluster_limit((const void*)k_pqr_factor, kThreads, (size_t)kPB * (kRowsMax | 1) * sizeof(double));
}

int64_t panel_rows_max() { return (int64_t)kRowsMax * pqr_cluster_limit(); }

// rows of a CTA when `others` CTAs share a row range of mmax: the most that still give four CTAs an
// SM, at least 64 (an update CTA repeats the 32 x 32 x 32 product with T)
static int pqr_rows(int64_t others, int64_t mmax, int most) {
  const int64_t chunks = std::max<int64_t>(1, (4 * 152 + others - 1) / others);
  const int64_t rows = ((mmax + chunks - 1) / chunks + 31) / 32 * 32;
  return (int)std::min<int64_t>(std::max<int64_t>(rows, 64), most);
}

// T factors (two kPB x kPB values per block) and the partial products of one block (most chunks: one
// column tile left)
int64_t panel_qr_scratch(int n, int kmax, int64_t mmax) {
  if (n <= 0 || kmax <= 0) return 0;
  const int64_t rows = pqr_rows(n, mmax, kVtcRows);
  const int64_t nblk = (kmax + kPB - 1) / kPB, nchunk = (mmax + rows - 1) / rows;
  return n * nblk * 2 * kPB * kPB + n * nchunk * std::max(kmax, 1) * kPB;
}

void launch_panel_rout(const PanelDesc* descs, int n, int kmax, int big, cudaStream_t st) {
  k_pqr_rout<<<dim3((unsigned)n, (unsigned)std::max(1, kmax * kmax / 4096)), 256, 0, st>>>(descs, big);
}

int launch_panel_qr(const PanelDesc* descs, int n, int kmax, int64_t mmax, double* scratch, cudaStream_t st) {
  if (n <= 0 || kmax <= 0) return 0;
  const int nblk = (kmax + kPB - 1) / kPB;
  auto chunks = [&](int rows) { return (unsigned)((mmax + rows - 1) / rows); };
  double* Ts = scratch;
  double* Wp = Ts + (int64_t)n * nblk * 2 * kPB * kPB;
  // CTAs per panel: enough for the rows to fit, then as many as keep a CTA per SM and 128 rows or
  // more each (a column's work shrinks with the rows, its barrier does not)
  int cs = 1;
  const int most = pqr_cluster_limit();
  while (cs < most && mmax > (int64_t)cs * kRowsMax) cs <<= 1;
  while (cs < most && n * cs * 2 <= 152 && mmax > (int64_t)cs * 128) cs <<= 1;
  int launches = 0;
  const int frows = pqr_rows(n, mmax, kApplyRows);
  auto apply = [&](int j0, int nt, int transT) {
    const unsigned tiles = (unsigned)((nt + 31) / 32);
    const int vrows = pqr_rows((int64_t)n * tiles, mmax, kVtcRows), arows = pqr_rows((int64_t)n * tiles, mmax, kApplyRows);
    const int nchunk = (int)chunks(vrows);
    k_pqr_vtc<<<dim3((unsigned)n, tiles, (unsigned)nchunk), kThreads, 0, st>>>(descs, j0, Wp, kmax, nchunk, vrows);
    k_pqr_apply<<<dim3((unsigned)n, tiles, chunks(arows)), kThreads, 0, st>>>(descs, j0, Wp, Ts, nblk, kmax, nchunk,
                                                                              vrows, arows, transT);
    launches += 2;
  };
  for (int b = 0; b < nblk; ++b) {
    const int j0 = b * kPB;
    const int M = (int)mmax - j0;
    const int rs = std::max((M + cs - 1) / cs, kPB);
    const size_t sm = (size_t)kPB * (rs | 1) * sizeof(double);
    smem_limit((const void*)k_pqr_factor, sm);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(n * cs));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = sm;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim = {(unsigned)cs, 1, 1};
    cfg.attrs = at;
    cfg.numAttrs = cs > 1 ? 1 : 0;
    cudaLaunchKernelEx(&cfg, k_pqr_factor, descs, j0, Ts, nblk, rs, cs);
    ++launches;
    const int nt = kmax - j0 - kPB;
    if (nt > 0) apply(j0, nt, 1);
  }
  launch_panel_rout(descs, n, kmax, 0, st);
  for (int b = nblk - 1; b >= 0; --b) {
    const int j0 = b * kPB, nt = kmax - j0 - kPB;
    if (nt > 0) apply(j0, nt, 0);
    k_pqr_form<<<dim3((unsigned)n, chunks(frows)), kThreads, 0, st>>>(descs, j0, Ts, nblk, frows);
    ++launches;
  }
  return launches + 1;
}

}  // namespace km
