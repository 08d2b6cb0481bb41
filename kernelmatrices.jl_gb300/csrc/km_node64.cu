// FP64 node factorisation of the nested Nystrom HODLR (lrsymfact of a node, src/HODLR/src/utils.jl:
// 29-35, in the bases described in km_factor.cu).  Given the children's R factors and Sc^{-T}:
//   T1 = R1 Sc^{-T}, T2 = R2 Sc^{-T}, Ct = T1 T2', L22 = chol(I - Ct' Ct)
//   G = [R1 ; L22^{-1}(R2 - Ct' R1)],  structured Householder QR  G = E R_N
// (reflector j is e_j on top plus a dense bottom part).  Outputs: Ct, L22, the scaled reflector
// bottoms, the taus and R_N.
//
// An FP64 instruction occupies a quarter of an SM for 65 cycles per warp, with one active lane or
// 32, and a square root or a division takes nine of them in a row.  A node of rank 72 needs about
// 65 k such instructions, so one CTA per node took 1.05 ms whatever the level, and the levels
// with fewer nodes than SMs left the others idle.  Here a node is a cluster of up to 8 CTAs:
//   products       (column, 32-row chunk) items over all warps of the cluster; T1, T2 and Ct are
//                  stored into every CTA's shared memory; column c of H = I - Ct'Ct (lower half
//                  only) and of B = R2 - Ct'R1 belongs to CTA c mod CTAs
//   Cholesky       by columns in dataflow order, (column, chunk) items: a chunk takes the earlier
//                  columns as they arrive, the chunk with the pivot publishes its square root, and
//                  every chunk divides by it and goes to all CTAs with asynchronous stores that
//                  complete a barrier there (no fence, no cluster barrier)
//   L22^{-1} B     every CTA on its own columns, a step per row
//   QR             a warp owns its columns; the warp of column j + 1 applies reflector j to that
//                  column first, forms reflector j + 1 and sends it in the same way, then applies
//                  reflector j to its other columns, four at a time so that their dot products
//                  share the additions over the lanes.  One warp per quarter of the SM where the
//                  column chain bounds it (several CTAs a node), two where the FP64 pipe does.
// Rank 72, time per level: 1.05 ms -> 0.34 ms with 8 CTAs a node, 0.75 ms with one.  (Cholesky in CTA 0
// alone, where its chunks compete for four quarters, took 286 k cycles against 168 k.)
//
// Every number is formed by the operations of the one-CTA kernel in the same order (dot products by
// row chunks of 32 and a butterfly over the lanes, updates one fused multiply-add at a time), so the
// factor's bits do not depend on the cluster size.
#include <cooperative_groups.h>

#include "km_cluster.cuh"
#include "km_kernels.h"

namespace km {

namespace cg = cooperative_groups;

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;

// v into the same location of every CTA (local store if the cluster is one CTA)
__device__ __forceinline__ void put_all(double* p, double v, int cs) {
  if (cs == 1) {
    *p = v;
    return;
  }
  cg::cluster_group cl = cg::this_cluster();
  for (int d = 0; d < cs; ++d) *cl.map_shared_rank(p, (unsigned)d) = v;
}

__device__ __forceinline__ void cluster_barrier(int cs) {
  if (cs == 1) __syncthreads();
  else cg::this_cluster().sync();
}

// Sums v[0..4) over the warp by the additions of the butterfly v + shfl_xor(v, 16, 8, 4, 2, 1);
// a lane returns the sum of v[2 b4 + b3] (b4, b3: its bits 4 and 3).
__device__ __forceinline__ double reduce4(double (&v)[4], int lane) {
#pragma unroll
  for (int h = 2, o = 16; h > 0; h >>= 1, o >>= 1) {
#pragma unroll
    for (int k = 0; k < h; ++k) {
      const bool up = (lane & o) != 0;
      const double keep = up ? v[k + h] : v[k], send = up ? v[k] : v[k + h];
      v[k] = __dadd_rn(keep, __shfl_xor_sync(0xffffffffu, send, o));
    }
  }
  double s = v[0];
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) s = __dadd_rn(s, __shfl_xor_sync(0xffffffffu, s, o));
  return s;
}

// d > 0, d != 0 on the bits: an FP64 comparison would take the FP64 pipe for 65 cycles
__device__ __forceinline__ bool positive(double d) {
  const long long b = __double_as_longlong(d);
  return b > 0 && b <= 0x7ff0000000000000ll;
}
__device__ __forceinline__ bool nonzero(double d) { return (__double_as_longlong(d) << 1) != 0; }

__device__ __forceinline__ double butterfly(double s) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s = __dadd_rn(s, __shfl_xor_sync(0xffffffffu, s, o));
  return s;
}

}  // namespace

__global__ void __launch_bounds__(kThreads, 1) k_node_factor_f64(double* __restrict__ R, const double* __restrict__ SinvT,
                                                              int r, int level, int L, int64_t nleaf, int64_t cbase,
                                                              int64_t nbase, double* __restrict__ Ct_out,
                                                              double* __restrict__ L22_out, double* __restrict__ Eref,
                                                              double* __restrict__ Etau, int* __restrict__ info, int cs,
                                                              int wait_limit) {
  extern __shared__ __align__(16) double sm[];
  const int ld = r + 1;
  double* X0 = sm;            // Sc^{-T}, then Ct; then G: L22^{-1} B, the updated columns, the reflectors
  double* X1 = X0 + r * ld;   // R1, then T2, then the own columns of R1 (of R_N in the end)
  double* X2 = X1 + r * ld;   // R2, then the own columns of B
  double* X3 = X2 + r * ld;   // T1, then the own columns of H, then L22
  double* va = X3 + r * ld;   // pivots of L22, then the betas
  double* vb = va + r;        // reflector scales
  double* vc = vb + r;        // reflector taus
  double* vi = vc + r;        // 1 / L22[j][j] (not va: another CTA's betas may arrive during the solve)
  unsigned long long* bars = reinterpret_cast<unsigned long long*>(vi + r);  // reflector j has arrived
  unsigned long long* cols = bars + r;  // 3 r: chunk s of column c of L22 (entry 3 c + s) has arrived
  volatile int* fd = reinterpret_cast<volatile int*>(cols + 3 * r);  // r: pivot of an own column is known
  __shared__ int sh_bad[8];   // of CTA 0: first non-positive pivot found by each CTA
  __shared__ int my_bad;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int rank = (int)(blockIdx.x % cs);
  const int64_t k = blockIdx.x / cs, node = nbase + k;
  const double* R1 = R + (cbase + 2 * k) * (int64_t)r * r;
  const double* R2 = R + (cbase + 2 * k + 1) * (int64_t)r * r;
  const int nch = (r + 31) >> 5, gw = rank * kWarps + w, ngw = cs * kWarps;
  // a wait_limit of 0 makes every wait give up at its first poll, as if its flag were never set
  const int lim = wait_limit < 0 ? kWaitPolls : wait_limit;
  for (int c = w; c < r; c += kWarps)
    for (int i = lane; i < r; i += 32) {
      const int e = i + c * r;
      X0[i + c * ld] = SinvT[e];
      X1[i + c * ld] = R1[e];
      X2[i + c * ld] = R2[e];
    }
  for (int e = tid; e < r; e += kThreads) fd[e] = 0;
  if (tid == 0) my_bad = r + 1;
  // one CTA: a barrier completes by the arrival of the warp that formed the reflector or chunk;
  // several: by the bytes it sends (entry 4 j: reflector j, 4 j + 1 + s: chunk s of column j)
  for (int e = tid; e < 4 * r; e += kThreads) {
    const int j = e >> 2, s = (e & 3) - 1;
    const int n = s < 0 ? r + 3 : min(r, 32 * s + 32) - max(j, 32 * s);  // values
    if (n <= 0) continue;
    const unsigned b = smem_u32(s < 0 ? bars + j : cols + 3 * j + s);
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b) : "memory");
    if (cs == 1) continue;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"(n * 8) : "memory");
  }
  cluster_barrier(cs);
  // T1 = R1 Sc^{-T} -> X3, T2 = R2 Sc^{-T} -> X1 (upper triangular), Ct = T1 T2' -> X0
  for (int half = 0; half < 2; ++half) {
    const double* A = half == 0 ? X1 : X2;
    double* T = half == 0 ? X3 : X1;
    for (int q = gw; q < r * nch; q += ngw) {
      const int c = q / nch, s = q - c * nch, i = 32 * s + lane;
      double acc = 0.0;
      if (i < r)
        for (int l = 32 * s; l <= c; ++l)
          if (l >= i) acc = __fma_rn(A[i + l * ld], X0[l + c * ld], acc);
      if (i < r) put_all(T + i + c * ld, acc, cs);
    }
    cluster_barrier(cs);
  }
  for (int q = gw; q < r * nch; q += ngw) {
    const int c = q / nch, s = q - c * nch, i = 32 * s + lane;
    double acc = 0.0;
    if (i < r) {
      const int l0 = max(32 * s, c);
      for (int l = l0; l < r; ++l)
        if (l >= i) acc = __fma_rn(X3[i + l * ld], X1[c + l * ld], acc);
      put_all(X0 + i + c * ld, acc, cs);
    }
  }
  cluster_barrier(cs);
  // H = I - Ct' Ct -> X3 of the column's CTA, lower triangle: columns p and r - 1 - p together hold r + 1
  // entries, so consecutive lanes take consecutive entries of such a pair
  {
    const int npair = (r + 1) / 2;
    for (int e = rank * kThreads + tid; e < npair * (r + 1); e += cs * kThreads) {
      const int p = e / (r + 1), u = e - p * (r + 1);
      if (u >= r - p && 2 * p == r - 1) continue;  // the middle column of an odd r, already taken
      const int c = u < r - p ? p : r - 1 - p, i = u < r - p ? p + u : r - 1 - p + (u - (r - p));
      double acc = 0.0;
      for (int l = 0; l < r; ++l) acc = __fma_rn(X0[l + i * ld], X0[l + c * ld], acc);
      double* H = cs == 1 ? X3 : cg::this_cluster().map_shared_rank(X3, (unsigned)(c % cs));
      H[i + c * ld] = __dsub_rn(i == c ? 1.0 : 0.0, acc);
    }
  }
  const int nown = (r - rank + cs - 1) / cs;  // own columns c = rank + cs lc
  if (level < L) {
    for (int lc = w; lc < nown; lc += kWarps) {
      const int c = rank + cs * lc;
      for (int i = lane; i < r; i += 32) X1[i + c * ld] = R1[i + c * r];
    }
    __syncthreads();
    // B = R2 - Ct' R1 -> X2, own columns (column c of R1 has entries l <= c)
    for (int q = w; q < nown * nch; q += kWarps) {
      const int lc = q / nch, s = q - lc * nch, c = rank + cs * lc, i = 32 * s + lane;
      if (i < r) {
        double acc = 0.0;
        for (int l = 0; l <= c; ++l) acc = __fma_rn(X0[l + i * ld], X1[l + c * ld], acc);
        X2[i + c * ld] = __dsub_rn(X2[i + c * ld], acc);
      }
    }
  }
  cluster_barrier(cs);
  // L22 = chol(H): chunks s of the own columns in column order, round robin over the warps.  A wait
  // that gives up marks the node with info = -1; the warp then stops waiting and carries on, so
  // that everything is sent.
  bool dead = false;
  auto give_up = [&]() {
    if (lane == 0) info[node] = -1;
    dead = true;
  };
  {
    int at = 0;
    for (int c = rank; c < r; c += cs) {
      const int pc = c >> 5;
      for (int s = pc; s < nch; ++s, ++at) {
        if (at % kWarps != w) continue;
        const int i = 32 * s + lane;
        const bool live = i >= c && i < r;
        double v = live ? X3[i + c * ld] : 0.0;
        int k0 = 0;
        while (k0 < c) {
          // chunk s of the column, and chunk pc for the multiplier L22[c][k]
          if (!dead && !bar_wait(smem_u32(cols + 3 * k0 + pc), wait_limit, cs)) give_up();
          if (s != pc && !dead && !bar_wait(smem_u32(cols + 3 * k0 + s), wait_limit, cs)) give_up();
          int k1 = k0 + 1;
          while (k1 < c && (dead || (bar_try(smem_u32(cols + 3 * k1 + pc), cs) &&
                                     (s == pc || bar_try(smem_u32(cols + 3 * k1 + s), cs)))))
            ++k1;
          if (live)
            for (int kk = k0; kk < k1; ++kk) v = __fma_rn(-X3[i + kk * ld], X3[c + kk * ld], v);
          k0 = k1;
        }
        double sd;
        if (s == pc) {
          const double d = __shfl_sync(0xffffffffu, v, c & 31);
          const bool ok = positive(d);
          if (!ok && lane == 0) atomicMin(&my_bad, c + 1);
          sd = ok ? sqrt(d) : 1.0;
          if (s + 1 < nch) {
            if (lane == 0) va[c] = sd;
            __threadfence_block();
            __syncwarp();
            if (lane == 0) fd[c] = 1;
          }
        } else {
          int spins = 0;
          while (!dead && (wait_limit == 0 || fd[c] == 0))
            if (++spins > lim) give_up();
          __threadfence_block();
          sd = va[c];
        }
        // (a zero numerator in an idle lane would send the warp through the slow division)
        const double x = i == c ? sd : (live ? v : 1.0) / sd;
        if (cs == 1) {
          if (live) X3[i + c * ld] = x;
          __threadfence_block();
          __syncwarp();
          if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(cols + 3 * c + s)) : "memory");
        } else if (live) {
          // the CTA of the next column first
          const unsigned to = smem_u32(X3 + i + c * ld), bar = smem_u32(cols + 3 * c + s);
          for (int u = 1, d = rank; u <= cs; ++u) {
            d = d + 1 == cs ? 0 : d + 1;
            st_async(at_rank(to, d), x, at_rank(bar, d));
          }
        }
      }
    }
  }
  // all of L22 has arrived (also after a wait that gave up: everything is sent)
  for (int c = w; c < r; c += kWarps)
    for (int q = c >> 5; q < nch; ++q)
      if (!bar_wait(smem_u32(cols + 3 * c + q), -1, cs) && lane == 0) info[node] = -1;
  __syncthreads();
  if (tid == 0) {
    int* to = cs == 1 ? sh_bad : cg::this_cluster().map_shared_rank(sh_bad, 0u);
    to[rank] = my_bad;
  }
  cluster_barrier(cs);
  if (rank == 0 && tid == 0) {
    int bad = r + 1;
    for (int d = 0; d < cs; ++d) bad = min(bad, sh_bad[d]);
    if (bad <= r && info[node] == 0) info[node] = bad;
  }
  for (int q = w; q < nown; q += kWarps) {
    const int c = rank + cs * q;
    for (int i = lane; i < r; i += 32) {
      const int64_t e = node * (int64_t)r * r + i + (int64_t)c * r;
      Ct_out[e] = X0[i + c * ld];
      L22_out[e] = i >= c ? X3[i + c * ld] : 0.0;
    }
  }
  if (level >= L) return;  // (no CTA touches another's memory from here on)
  // G = L22^{-1} B -> X0 (own columns), row by row: a thread keeps to one column and every
  // 256 / nown-th row, scales the row's entry for itself, and the first of them stores it
  for (int i = tid; i < r; i += kThreads) vi[i] = 1.0 / X3[i + i * ld];
  __syncthreads();
  if (nown > 0) {  // (a CTA of a rank below the cluster size may own no column)
    const int per = kThreads / nown, off = tid / nown, c = rank + cs * (tid - off * nown);
    double* b = X2 + c * ld;
    for (int i = 0; i < r; ++i) {
      if (off < per) {
        const double x = __dmul_rn(b[i], vi[i]);
        if (off == 0) X0[i + c * ld] = x;
        for (int ii = i + 1 + off; ii < r; ii += per) b[ii] = __fma_rn(-X3[ii + i * ld], x, b[ii]);
      }
      __syncthreads();
    }
  }
  // Householder QR of [X1 (upper) ; X0] by columns: warp w < qw of CTA `rank` owns the columns
  // c = rank + cs (w + qw t)
  const int qw = cs == 1 ? kWarps : 4;
  const int mine = rank + cs * w, step = cs * qw;
  const int last = w >= qw || mine >= r ? -1 : mine + (r - 1 - mine) / step * step;  // largest own column
  auto rows3 = [&](const double* col, double (&x)[3]) {
#pragma unroll
    for (int s = 0; s < 3; ++s) x[s] = 32 * s + lane < r ? col[32 * s + lane] : 0.0;
  };
  // reflector c from its column (all earlier reflectors applied): to every CTA
  auto reflect = [&](int c, const double (&x)[3]) {
    double p[4] = {__dmul_rn(x[0], x[0]), __dmul_rn(x[1], x[1]), __dmul_rn(x[2], x[2]), 0.0};
    const double t = reduce4(p, lane);
    const double s0 = __shfl_sync(0xffffffffu, t, 0), s1 = __shfl_sync(0xffffffffu, t, 8),
                 s2 = __shfl_sync(0xffffffffu, t, 16);
    const double sig = __dadd_rn(__dadd_rn(s0, s1), s2), alpha = X1[c + c * ld];
    double beta = alpha, q = 0.0;
    if (nonzero(sig)) {
      const double nrm = sqrt(__fma_rn(alpha, alpha, sig));
      beta = __double_as_longlong(alpha) >= 0 || !nonzero(alpha) ? -nrm : nrm;  // alpha >= 0
      // lane 1: tau = (beta - alpha) / beta; the others: scale = 1 / (alpha - beta)
      const double d = __dsub_rn(lane == 1 ? beta : alpha, lane == 1 ? alpha : beta);
      q = __ddiv_rn(lane == 1 ? d : 1.0, lane == 1 ? beta : d);
    }
    const unsigned bar = smem_u32(bars + c), col = smem_u32(X0 + c * ld);
    const double mineq = lane == 2 ? beta : q;  // lane 0 scale, 1 tau, 2 beta
    double* mineto = (lane == 0 ? vb : lane == 1 ? vc : va) + c;
    const unsigned slot = smem_u32(mineto);
    if (cs == 1) {
#pragma unroll
      for (int s = 0; s < 3; ++s)
        if (32 * s + lane < r) X0[32 * s + lane + c * ld] = x[s];
      if (lane < 3) *mineto = mineq;
      __threadfence_block();
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
    }
    for (int u = 1, d = rank; u <= cs && cs > 1; ++u) {  // the CTA of the next column first
      d = d + 1 == cs ? 0 : d + 1;
      const unsigned rb = at_rank(bar, d), rc = at_rank(col, d);
#pragma unroll
      for (int s = 0; s < 3; ++s)
        if (32 * s + lane < r) st_async(rc + 8 * (32 * s + lane), x[s], rb);
      if (lane < 3) st_async(at_rank(slot, d), mineq, rb);
    }
    if (lane == 1) Etau[node * (int64_t)r + c] = q;
  };
  if (mine == 0 && w < qw) {
    double x[3];
    rows3(X0, x);
    reflect(0, x);
  }
  for (int j = 0; j < last; ++j) {
    if (!dead && !bar_wait(smem_u32(bars + j), wait_limit, cs)) give_up();
    const double tau = vc[j], scal = vb[j];
    double v[3];
    rows3(X0 + j * ld, v);
    const int first = j < mine ? mine : mine + ((j - mine) / step + 1) * step;  // own columns > j
    int c0 = first;
    if (first == j + 1) {  // the next reflector's column
      double x[3];
      rows3(X0 + first * ld, x);
      if (nonzero(tau)) {
        double a = __fma_rn(v[0], x[0], 0.0);
        a = __fma_rn(v[1], x[1], a);
        a = __fma_rn(v[2], x[2], a);
        const double x1 = X1[j + first * ld];
        a = __dmul_rn(__fma_rn(butterfly(a), scal, x1), tau);
        const double f = __dmul_rn(a, scal);
#pragma unroll
        for (int s = 0; s < 3; ++s) x[s] = __fma_rn(-f, v[s], x[s]);
        if (lane == 0) X1[j + first * ld] = __dsub_rn(x1, a);
      }
      reflect(first, x);
      c0 += step;
    }
    if (!nonzero(tau)) continue;
    for (; c0 < r; c0 += 4 * step) {
      double x[4][3], a[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int c = min(c0 + u * step, last);
        rows3(X0 + c * ld, x[u]);
      }
      const int nu = (last - c0) / step + 1;  // columns of this group (4 or fewer)
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        a[u] = 0.0;
        if (u < nu) {
          a[u] = __fma_rn(v[0], x[u][0], 0.0);
          a[u] = __fma_rn(v[1], x[u][1], a[u]);
          a[u] = __fma_rn(v[2], x[u][2], a[u]);
        }
      }
      const int mu = 2 * ((lane >> 4) & 1) + ((lane >> 3) & 1);
      const int cm = min(c0 + mu * step, last);
      const double x1 = X1[j + cm * ld];
      const double acc = __dmul_rn(__fma_rn(reduce4(a, lane), scal, x1), tau);
      const double f = __dmul_rn(acc, scal);
      __syncwarp();
      if ((lane & 7) == 0 && mu < nu) X1[j + cm * ld] = __dsub_rn(x1, acc);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const double fu = __shfl_sync(0xffffffffu, f, (u >> 1) * 16 + (u & 1) * 8);
        if (u < nu) {
          double* col = X0 + (c0 + u * step) * ld;
#pragma unroll
          for (int s = 0; s < 3; ++s)
            if (32 * s + lane < r) col[32 * s + lane] = __fma_rn(-fu, v[s], x[u][s]);
        }
      }
      __syncwarp();
    }
  }
  // every reflector has arrived (also after a wait that gave up: all are sent), so that nothing is
  // on its way to this CTA when it leaves; then R_N and the scaled bottoms of the own columns
  for (int c = w; c < r; c += kWarps) {
    if (!bar_wait(smem_u32(bars + c), -1, cs) && lane == 0) info[node] = -1;
  }
  __syncthreads();
  double* Rn = R + (nleaf + node) * (int64_t)r * r;
  for (int c = mine; c <= last; c += step) {
    const double scal = vb[c], beta = va[c];
    for (int i = lane; i < r; i += 32) {
      const int64_t e = i + (int64_t)c * r;
      Rn[e] = i < c ? X1[i + c * ld] : (i == c ? beta : 0.0);
      Eref[node * (int64_t)r * r + e] = __dmul_rn(X0[i + c * ld], scal);
    }
  }
}

size_t node_f64_smem(int r) {
  return ((size_t)4 * r * (r + 1) + 8 * r) * sizeof(double) + (size_t)r * sizeof(int);
}

cudaError_t launch_node_f64(double* R, const double* SinvT, int r, int level, const Tree& t, double* Ct, double* L22,
                            double* Eref, double* Etau, int* info, int cs, int wait_limit, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(t.nodes_at(level) * cs));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = node_f64_smem(r);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim = {(unsigned)cs, 1, 1};
  cfg.attrs = at;
  cfg.numAttrs = cs > 1 ? 1 : 0;
  const int64_t cbase = (level == 1) ? 0 : t.nleaf + t.node_off[level - 1];
  return cudaLaunchKernelEx(&cfg, k_node_factor_f64, R, SinvT, r, level, t.L, t.nleaf, cbase, t.node_off[level], Ct, L22,
                            Eref, Etau, info, cs, wait_limit);
}

const void* node_f64_kernel() { return (const void*)k_node_factor_f64; }

}  // namespace km
