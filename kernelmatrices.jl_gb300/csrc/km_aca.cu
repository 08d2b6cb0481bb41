// ACA assembly and the general (per-block basis) HODLR factorisation used for ACA blocks.
//
// ACA: one cluster of CTAs per off-diagonal block (16, for many small blocks 4 or 2) runs the partially pivoted adaptive cross approximation of
// the reference (src/factorizations.jl:9-84) step for step: the start-row search, the pivot
// rule of restrictedmaxabs (src/utils.jl:2-15: first strict maximum of |x| outside the used set,
// the first unused index when nothing is non-zero), residual updates as a multiply followed by a
// subtract (Julia's `tmprow .-= U[j][mi]*V[j]` is not fused), the Frobenius-norm estimate update
// and the stopping rule norm(row)*norm(col) > rtol*sqrt(znorm2).  Kernel rows and columns are
// evaluated on the fly; U and V are written into per-block panels (column-major).
//
// General factorisation (src/HODLR/src/symfact.jl:6-49 without the Nystrom nesting): leaf
// Cholesky, leaf triangular solves of every panel, then per level the Householder QR of the
// node's V (rows c1) and U (rows c2) panels with explicit Q, C = R1 R2', L22 = chol(I - C'C),
// and the application of W_N^{-1} to the coarser panels.  In the QR bases W_N^{-1} only changes
// the c2 rows:  y_c2 -= Q2 (z2 - L22^{-1}(z2 - C' z1)),  z1 = Q1' y_c1, z2 = Q2' y_c2.
#include <cooperative_groups.h>

#include <algorithm>
#include <climits>

#include "km_kernels.h"

namespace km {

namespace cg = cooperative_groups;

// ---------------------------------------------------------------------------------------------
// CTA-wide reductions (deterministic order)
// ---------------------------------------------------------------------------------------------
__device__ double cta_sum(double v, double* sred) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  v = warp_sum(v);
  if (lane == 0) sred[w] = v;
  __syncthreads();
  if (w == 0) {
    double t = (lane < nw) ? sred[lane] : 0.0;
    t = warp_sum(t);
    if (lane == 0) sred[32] = t;
  }
  __syncthreads();
  const double t = sred[32];
  __syncthreads();
  return t;
}

// ---------------------------------------------------------------------------------------------
// Grid barrier of a cooperative launch.  It spins a bounded number of times; one that runs out sets
// an error word that every CTA sees at its next barrier, so the launch ends early as a whole.
// ---------------------------------------------------------------------------------------------
constexpr long long kGridSpinLimit = 1ll << 20;  // L2 polls per barrier wait (~0.3 s)

struct GridBar {
  unsigned* count;
  volatile unsigned* gen;
  volatile int* err;
  long long limit;  // polls before a wait gives up (< 0: kGridSpinLimit; 0: at the first poll, as
                    // if the other CTAs never arrived: the test of the timeout path)
};

// Returns true when every CTA has arrived and no barrier of this launch has run out; the answer
// is the same for all threads of the CTA (thread 0's view, passed through shared memory), so the
// CTA leaves its loop as a whole.
__device__ bool grid_barrier(GridBar gb) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    const long long lim = gb.limit < 0 ? kGridSpinLimit : gb.limit;
    const unsigned g = *gb.gen;
    __threadfence();
    if (atomicAdd(gb.count, 1u) == gridDim.x - 1) {
      *gb.count = 0;
      __threadfence();
      atomicExch((unsigned*)gb.gen, g + 1);
    } else {
      long long spins = 0;
      while ((gb.limit == 0 || *gb.gen == g) && *gb.err == 0) {
        if (++spins > lim) {
          atomicExch((int*)gb.err, 1);
          break;
        }
      }
    }
    __threadfence();
    s_ok = *gb.err == 0;
  }
  __syncthreads();
  return s_ok != 0;
}

// ---------------------------------------------------------------------------------------------
// ACA of one block by a team of CTAs: a thread-block cluster (k_aca) or, for blocks of 8192 points
// and more, every SM (k_aca_grid, a cooperative launch).  status: 0 ok, 1 "Incompatible maxrank or
// matrix dimensions." (factorizations.jl:30), 2 rank capacity of the panel reached before
// convergence, 3 a grid barrier ran out.
//
// Each CTA owns a slice of the rows and a slice of the columns.  A step takes three team barriers
// (0.2 us in a cluster, about 1.5 us over the grid): the CTAs' candidates for the column pivot; those
// for the next row pivot with the squared norms and the dots with the earlier columns; the shares
// of the norm update.  Candidates are compared by |x| (as integers) with ties to the smaller
// index, so every CTA takes the pivots of a scan over the whole row.
//
// A residual entry is a chain of one multiply and one subtract per earlier column, in the
// reference's order, and a warp's FP64 instruction takes 65 cycles of its quarter of the SM however
// few lanes are active: the chains bound the kernel.  One CTA per block ran a 512 x 512 block of
// rank 496 (the README example: unsorted points, tolerance 1e-12) in 147 ms.  Split over 16 SMs a
// slice holds 32 entries, and where a slice has at most 64 the multiplies, which do not wait for
// one another, go to the quarters that the subtractions leave idle.  The slices of the first columns
// stay in shared memory (L2 latency had doubled the chains' time): 20.6 ms.  The 4096-point blocks
// of a 2^14 matrix went from 191 to 21.4 ms, its 8192-point block (every SM in both forms; before
// with seven barriers a step, searches by one thread and unbatched loads) from 74 to 21.8 ms.
// ---------------------------------------------------------------------------------------------
namespace {

constexpr int kAcaThreads = 256;
constexpr int kAcaChunk = 32;   // earlier columns per stage of the split residual
constexpr int kAcaSplit = 64;   // widest slice whose multiplies and subtractions go to different warps

struct AcaRec {                 // one CTA's part of a search and of the sums
  unsigned long long key;       // bits of the largest |x| outside the used set (0: none is non-zero)
  long long idx, first;         // its index; the first unused index
  double val;                   // x[idx]
  double z;                     // share of the norm update
};

struct AcaShared {
  AcaRec rec[3];                // column search, row search, norm update: the barriers of a step apart
  AcaRec win;                   // combined search of this step (same in every CTA)
  AcaRec part[kAcaThreads / 32];
  double sums[2];               // squared norms of the new row and column
  double zpart[kAcaThreads / 32];
  int stop;
};

__device__ __forceinline__ bool aca_better(unsigned long long k, long long i, const AcaRec& r) {
  return k > r.key || (k == r.key && i < r.idx);
}

__device__ __forceinline__ void aca_warp_best(AcaRec& r) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long k = __shfl_xor_sync(0xffffffffu, r.key, o);
    const long long i = __shfl_xor_sync(0xffffffffu, r.idx, o), f = __shfl_xor_sync(0xffffffffu, r.first, o);
    const double v = __shfl_xor_sync(0xffffffffu, r.val, o);
    if (aca_better(k, i, r)) {
      r.key = k;
      r.idx = i;
      r.val = v;
    }
    r.first = min(r.first, f);
  }
}

// Entry x of index i offered to a thread's candidate; a NaN is never the largest.
__device__ __forceinline__ void aca_offer(AcaRec& r, double x, long long i, bool used) {
  if (used) return;
  if (r.first == LLONG_MAX) r.first = i;
  const unsigned long long k = (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
  if (k <= 0x7ff0000000000000ull && k > r.key) {
    r.key = k;
    r.idx = i;
    r.val = x;
  }
}

// The CTAs of a cluster exchange records and partial dots through distributed shared memory.
struct ClusterTeam {
  static constexpr int kLanes = 4;  // lanes that sum one column's partial dots over the CTAs
  AcaShared* S;
  double* d;                        // 2 x (cap + 1): partial dots of U_j . col, then of V_j . row
  int cap1;
  __device__ int size() const { return (int)cg::this_cluster().num_blocks(); }
  __device__ int rank() const { return (int)cg::this_cluster().block_rank(); }
  __device__ bool barrier() const {
    cg::this_cluster().sync();
    return true;
  }
  __device__ AcaRec* mine(int s) const { return S->rec + s; }
  __device__ double* dots(int side) const { return d + side * cap1; }
  __device__ AcaRec get(int s, int q) const { return cg::this_cluster().map_shared_rank(S, q)->rec[s]; }
  __device__ double get_z(int q) const { return cg::this_cluster().map_shared_rank(S, q)->rec[2].z; }
  __device__ double dot(int side, int q, int j) const {
    return *cg::this_cluster().map_shared_rank(d + side * cap1 + j, q);
  }
};

// The CTAs of a cooperative launch exchange them through L2.
struct GridTeam {
  static constexpr int kLanes = 32;
  GridBar gb;
  AcaRec* recs;   // 3 x CTAs
  double* d;      // CTAs x 2 x (cap + 1)
  int cap1;
  __device__ int size() const { return (int)gridDim.x; }
  __device__ int rank() const { return (int)blockIdx.x; }
  __device__ bool barrier() const { return grid_barrier(gb); }
  __device__ AcaRec* mine(int s) const { return recs + s * gridDim.x + blockIdx.x; }
  __device__ double* dots(int side) const { return d + (2 * (int64_t)blockIdx.x + side) * cap1; }
  __device__ AcaRec get(int s, int q) const {
    const AcaRec* r = recs + s * gridDim.x + q;
    return AcaRec{__ldcg(&r->key), __ldcg(&r->idx), __ldcg(&r->first), __ldcg(&r->val), 0.0};
  }
  __device__ double get_z(int q) const { return __ldcg(&recs[2 * gridDim.x + q].z); }
  __device__ double dot(int side, int q, int j) const { return __ldcg(d + (2 * (int64_t)q + side) * cap1 + j); }
};

// The team's winner of record slot s, the same in every CTA; ends with a CTA barrier.
template <typename Team>
__device__ void aca_combine(const Team& team, AcaShared& S, int s, int64_t n) {
  if (threadIdx.x < 32) {
    AcaRec r{0, LLONG_MAX, LLONG_MAX, 0.0, 0.0};
    for (int q = threadIdx.x; q < team.size(); q += 32) {
      const AcaRec o = team.get(s, q);
      if (aca_better(o.key, o.idx, r)) {
        r.key = o.key;
        r.idx = o.idx;
        r.val = o.val;
      }
      r.first = min(r.first, o.first);
    }
    aca_warp_best(r);
    if (threadIdx.x == 0) {
      if (r.key == 0) {  // nothing non-zero is left: the first unused index
        r.val = 0.0;
        r.idx = r.first == LLONG_MAX ? n - 1 : r.first;
      }
      S.win = r;
    }
  }
  __syncthreads();
}

// This CTA's candidate into its record of slot s (a team barrier follows).
__device__ void aca_publish(AcaShared& S, AcaRec* out, AcaRec r) {
  aca_warp_best(r);
  if ((threadIdx.x & 31) == 0) S.part[threadIdx.x >> 5] = r;
  __syncthreads();
  if (threadIdx.x == 0) {
    r = S.part[0];
    for (int q = 1; q < kAcaThreads / 32; ++q) {
      if (aca_better(S.part[q].key, S.part[q].idx, r)) {
        r.key = S.part[q].key;
        r.idx = S.part[q].idx;
        r.val = S.part[q].val;
      }
      r.first = min(r.first, S.part[q].first);
    }
    out->key = r.key;
    out->idx = r.idx;
    out->first = r.first;
    out->val = r.val;
  }
}

// A CTA's slices of the earlier columns of U or V: the first `kept` columns in shared memory
// (column j at s + j n), every column in global memory (entry e at g + e + j ld, lo <= e < lo + n).
struct AcaSlice {
  double* s;
  int kept, n;
  const double* g;
  int64_t ld, lo;
};

// Residual entries of the slice of a row or column: out[e] = k(e) - sum_j coef[j] M[e, j], one
// multiply and one subtract per j in order; returns the thread's candidate among those not in
// `used`.  keep: where to put a copy (entry e - lo) or null.  role: this warp's number, rotated between the clusters so that the subtraction warps
// of co-resident CTAs fall on different quarters of the SM.
template <typename Eval>
__device__ AcaRec aca_residual(Eval&& eval, const AcaSlice& M, double* out, double* keep, const uint8_t* used,
                               const double* coef, int nj, double* prod, int role) {
  AcaRec r{0, LLONG_MAX, LLONG_MAX, 0.0, 0.0};
  const int lane = threadIdx.x & 31;
  if (M.n > kAcaSplit) {
    for (int e = role * 32 + lane; e < M.n; e += kAcaThreads) {
      double v = eval(M.lo + e);
      const int js = min(nj, M.kept);
      int j = 0;
#pragma unroll 8
      for (; j < js; ++j) v = __dsub_rn(v, __dmul_rn(coef[j], M.s[j * M.n + e]));
      const double* g = M.g + M.lo + e;
      for (; j + 8 <= nj; j += 8) {
        double m[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) m[q] = g[(int64_t)(j + q) * M.ld];
#pragma unroll
        for (int q = 0; q < 8; ++q) v = __dsub_rn(v, __dmul_rn(coef[j + q], m[q]));
      }
      for (; j < nj; ++j) v = __dsub_rn(v, __dmul_rn(coef[j], g[(int64_t)j * M.ld]));
      out[M.lo + e] = v;
      if (keep) keep[e] = v;
      aca_offer(r, v, M.lo + e, used[M.lo + e]);
    }
    return r;
  }
  const int nc = M.n > 32 ? 2 : 1;                 // subtraction warps: roles 0 .. nc-1
  const int np = (kAcaThreads / 128) * (4 - nc);   // multiply warps: roles with role % 4 >= nc
  const int e = role * 32 + lane;
  const bool mine = role < nc && e < M.n;
  double v = mine ? eval(M.lo + e) : 0.0;
  const int nchunk = (nj + kAcaChunk - 1) / kAcaChunk;
  for (int t = 0; t <= nchunk; ++t) {
    if ((role & 3) >= nc) {
      if (t < nchunk) {
        double* buf = prod + (t & 1) * kAcaChunk * kAcaSplit;
        const int j0 = t * kAcaChunk, jn = min(kAcaChunk, nj - j0);
        const int pw = (role >> 2) * (4 - nc) + (role & 3) - nc;
        if (j0 + jn <= M.kept) {
          for (int it = pw; it < jn * nc; it += np) {
            const int jj = it / nc, ee = (it - jj * nc) * 32 + lane;
            if (ee < M.n) buf[jj * kAcaSplit + ee] = __dmul_rn(coef[j0 + jj], M.s[(j0 + jj) * M.n + ee]);
          }
        } else {
#pragma unroll 8
          for (int it = pw; it < jn * nc; it += np) {
            const int jj = it / nc, ee = (it - jj * nc) * 32 + lane;
            if (ee < M.n) buf[jj * kAcaSplit + ee] = __dmul_rn(coef[j0 + jj], M.g[M.lo + ee + (j0 + jj) * M.ld]);
          }
        }
      }
    } else if (mine && t > 0) {
      const double* buf = prod + ((t - 1) & 1) * kAcaChunk * kAcaSplit + e;
      const int jn = min(kAcaChunk, nj - (t - 1) * kAcaChunk);
#pragma unroll 8
      for (int jj = 0; jj < jn; ++jj) v = __dsub_rn(v, buf[jj * kAcaSplit]);
    }
    __syncthreads();
  }
  if (mine) {
    out[M.lo + e] = v;
    if (keep) keep[e] = v;
    aca_offer(r, v, M.lo + e, used[M.lo + e]);
  }
  return r;
}

// 4 lanes' parts of sum_e M[e, j] x[e] over the slice
__device__ __forceinline__ double aca_dot(const AcaSlice& M, int j, const double* x, int p) {
  double a = 0.0;
  if (j < M.kept) {
    const double* m = M.s + j * M.n;
#pragma unroll 8
    for (int e = p; e < M.n; e += 4) a += m[e] * x[e];
  } else {
    const double* m = M.g + M.lo + (int64_t)j * M.ld;
#pragma unroll 8
    for (int e = p; e < M.n; e += 4) a += m[e] * x[e];
  }
  return a;
}

// store: shared memory of `room` doubles for the slices of the first columns.
// The whole approximation; false if a barrier ran out (every CTA of the team then leaves).
template <typename Team>
__device__ bool aca_run(const Team& team, AcaShared& S, double* dsm, double* store, int64_t room, int turn, const double* __restrict__ pts,
                        const KParams& kp, const AcaBlock& B, double* P, uint8_t* F, int* __restrict__ piv,
                        double rtol, int* __restrict__ rank_out, int* __restrict__ status) {
  const int G = team.size(), g = team.rank();
  const int64_t nro = B.nro, ncl = B.ncl;
  const int cap = B.cap;
  double* coef = dsm;              // cap: U[ri, j] or V[cj, j] of the earlier columns
  double* prod = coef + cap;       // 2 x kAcaChunk x kAcaSplit
  double* da = team.dots(0);       // cap + 1: this CTA's part of U_j . col; entry frnk: |col|^2
  double* db = team.dots(1);       // cap + 1: V_j . row; |row|^2
  double* U = P + B.offU;
  double* V = P + B.offV;
  uint8_t* urow = F + B.offFlag;   // a CTA reads and sets the flags of its own slices only
  uint8_t* ucol = urow + nro;
  int* prow = piv + 2 * B.offPiv;
  int* pcol = prow + cap;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  constexpr int nw = kAcaThreads / 32;
  const int role = (w + turn) & (nw - 1);
  const int64_t rs = (nro + G - 1) / G, cs = (ncl + G - 1) / G;
  const int64_t r_lo = min(nro, g * rs), r_hi = min(nro, r_lo + rs);
  const int64_t c_lo = min(ncl, g * cs), c_hi = min(ncl, c_lo + cs);
  const int rn = (int)(r_hi - r_lo), cn = (int)(c_hi - c_lo);
  const int kept = (int)min((int64_t)cap, room / (rs + cs));
  const AcaSlice Us{store, kept, rn, U, nro, r_lo}, Vs{store + (int64_t)kept * rs, kept, cn, V, ncl, c_lo};
  const double* xr = pts + 2 * B.row0;
  const double* xc = pts + 2 * B.col0;
  for (int64_t i = r_lo + tid; i < r_hi; i += kAcaThreads) urow[i] = 0;
  for (int64_t c = c_lo + tid; c < c_hi; c += kAcaThreads) ucol[c] = 0;
  __syncthreads();
  const int maxsz = B.maxsz;
  auto row_of = [&](int64_t i) {
    const double px = xr[2 * i], py = xr[2 * i + 1];
    return [=](int64_t c) { return kernel_value(kp, px, py, xc[2 * c], xc[2 * c + 1]); };
  };
  auto col_of = [&](int64_t j) {
    const double px = xc[2 * j], py = xc[2 * j + 1];
    return [=](int64_t i) { return kernel_value(kp, xr[2 * i], xr[2 * i + 1], px, py); };
  };
  int st = 0, frnk = 0;
  double znorm2 = 0.0;
  // first row not all zero (factorizations.jl:24-30)
  int64_t ri = 0;
  for (;;) {
    aca_publish(S, team.mine(0), aca_residual(row_of(ri), Vs, V, nullptr, ucol, coef, 0, prod, role));
    if (!team.barrier()) return false;
    aca_combine(team, S, 0, ncl);
    if (S.win.key != 0 || ri + 1 >= maxsz) break;
    ++ri;
    if (!team.barrier()) return false;  // the records have been read
  }
  if (ri + 1 == maxsz) {
    st = 1;
  } else {
    for (;;) {
      // S.win: the column pivot; row `frnk` of V holds the unscaled residual row of row pivot ri
      const double cv = S.win.val;
      const int64_t cj = S.win.idx;
      if (frnk > 0 && cv == 0.0) break;
      double* row = V + (int64_t)frnk * ncl;
      double* col = U + (int64_t)frnk * nro;
      if (tid == 0) {
        if (ri >= r_lo && ri < r_hi) urow[ri] = 1;
        if (cj >= c_lo && cj < c_hi) ucol[cj] = 1;
        if (g == 0) {
          prow[frnk] = (int)ri;
          pcol[frnk] = (int)cj;
        }
      }
      for (int j = tid; j < frnk; j += kAcaThreads) coef[j] = __ldcg(V + cj + (int64_t)j * ncl);
      double* rkeep = frnk < kept ? Vs.s + frnk * cn : nullptr;
      double* ckeep = frnk < kept ? Us.s + frnk * rn : nullptr;
      for (int c = tid; c < cn; c += kAcaThreads) {
        const double v = __ddiv_rn(row[c_lo + c], cv);
        row[c_lo + c] = v;
        if (rkeep) rkeep[c] = v;
      }
      __syncthreads();
      const AcaRec rr = aca_residual(col_of(cj), Us, col, ckeep, urow, coef, frnk, prod, role);
      __syncthreads();
      // this CTA's parts of the dots with the earlier columns and (entry frnk) of the squared
      // norms: 4 lanes per column, so that a warp reduces 8 columns by two shuffle steps
      for (int j0 = 0; j0 <= frnk; j0 += kAcaThreads / 4) {
        const int j = j0 + (tid >> 2), p = tid & 3;
        double a = 0.0, b = 0.0;
        if (j <= frnk) {
          a = aca_dot(Us, j, ckeep ? ckeep : col + r_lo, p);
          b = aca_dot(Vs, j, rkeep ? rkeep : row + c_lo, p);
        }
        if (j0 + (w << 3) <= frnk) {
          a += __shfl_xor_sync(0xffffffffu, a, 1);
          b += __shfl_xor_sync(0xffffffffu, b, 1);
          a += __shfl_xor_sync(0xffffffffu, a, 2);
          b += __shfl_xor_sync(0xffffffffu, b, 2);
          if (p == 0 && j <= frnk) {
            da[j] = a;
            db[j] = b;
          }
        }
      }
      aca_publish(S, team.mine(1), rr);
      if (!team.barrier()) return false;
      aca_combine(team, S, 1, nro);
      ri = S.win.idx;
      // sums over the CTAs: CTA g takes the columns j = g, g + G, ...; every CTA the norms
      {
        constexpr int kL = Team::kLanes, kPer = 32 / kL;  // columns per warp
        const int p = lane % kL, nmine = g < frnk ? (frnk - g + G - 1) / G : 0;
        double z = 0.0;
        for (int t0 = w * kPer; t0 <= nmine; t0 += nw * kPer) {
          const int t = t0 + lane / kL, j = t < nmine ? g + t * G : frnk;
          double a = 0.0, b = 0.0;
          if (t <= nmine)
            for (int q = p; q < G; q += kL) {
              a += team.dot(0, q, j);
              b += team.dot(1, q, j);
            }
#pragma unroll
          for (int o = 1; o < kL; o <<= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, o);
            b += __shfl_xor_sync(0xffffffffu, b, o);
          }
          if (t < nmine && p == 0) z += __dmul_rn(__dmul_rn(2.0, fabs(a)), fabs(b));
          if (t == nmine && p == 0) {
            S.sums[0] = b;
            S.sums[1] = a;
          }
        }
        if (w * kPer <= nmine) {  // (warps without a column hold zero)
#pragma unroll
          for (int o = kL; o < 32; o <<= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
        }
        if (lane == 0) S.zpart[w] = z;
      }
      __syncthreads();
      if (tid == 0) {
        double z = S.zpart[0];
        const int used_w = min(nw, (g < frnk ? (frnk - g + G - 1) / G : 0) * Team::kLanes / 32 + 1);
        for (int q = 1; q < used_w; ++q) z += S.zpart[q];
        team.mine(2)->z = z;
      }
      if (!team.barrier()) return false;
      if (w == 0) {
        double z = 0.0;
        for (int q = lane; q < G; q += 32) z += team.get_z(q);
        z = warp_sum(z);
        const double sr = S.sums[0], sc = S.sums[1];
        znorm2 = __dadd_rn(__dadd_rn(znorm2, z), __dmul_rn(sr, sc));
        const bool go = __dmul_rn(sqrt(sr), sqrt(sc)) > __dmul_rn(rtol, sqrt(znorm2)) && frnk + 1 < maxsz;
        if (lane == 0) S.stop = !go;
      }
      __syncthreads();
      ++frnk;
      if (S.stop) break;
      if (frnk >= cap) {
        st = 2;
        break;
      }
      // residual row of the next row pivot, and its largest entry outside the used columns
      for (int j = tid; j < frnk; j += kAcaThreads) coef[j] = __ldcg(U + ri + (int64_t)j * nro);
      __syncthreads();
      if (tid == 0 && ri >= r_lo && ri < r_hi) urow[ri] = 1;
      aca_publish(S, team.mine(0), aca_residual(row_of(ri), Vs, V + (int64_t)frnk * ncl, nullptr, ucol, coef, frnk, prod, role));
      if (!team.barrier()) return false;
      aca_combine(team, S, 0, ncl);
    }
  }
  if (g == 0 && tid == 0) {
    *rank_out = frnk;
    *status = st;
  }
  return team.barrier();  // no CTA leaves while another may still read its shared memory
}

// ---------------------------------------------------------------------------------------------
// Householder QR with explicit Q of tall panels (more rows than a cluster's shared memory holds,
// see km_pqr.cu for the others), blocked (LAPACK dgeqrf / dorgqr structure): reflectors of kQB
// columns are formed by the unblocked dgeqr2 / dlarfg rules and applied to the rest of the panel as
// one compact-WY block reflector I - V T V'.
// ---------------------------------------------------------------------------------------------
constexpr int kQB = 8;

// T (kQB x kQB, upper, column-major) of the block reflector of columns j0 .. j0+jb-1:
//   T[q][q] = tau_q,  T[0:q, q] = -tau_q T[0:q, 0:q] (V[:, 0:q]' v_q)
// with v_p = e_p + A[p+1:, p] (zero above row p).  G holds the dots v_p . v_q.
__device__ void panel_block_T(const double* A, int64_t m, int64_t lda, int j0, int jb, const double* tau,
                              double* G, double* Tm) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int pq = w; pq < jb * jb; pq += nw) {
    const int p = pq % jb, q = pq / jb;
    if (p >= q) continue;
    const double* vp = A + (int64_t)(j0 + p) * lda;
    const double* vq = A + (int64_t)(j0 + q) * lda;
    // v_p[j0+q] * 1 + sum_{i > j0+q} v_p[i] v_q[i]
    double acc = 0.0;
    for (int64_t i = j0 + q + 1 + lane; i < m; i += 32) acc += vp[i] * vq[i];
    acc = warp_sum(acc);
    if (lane == 0) G[p + q * kQB] = acc + vp[j0 + q];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int q = 0; q < jb; ++q) {
      const double tq = tau[j0 + q];
      for (int p = 0; p < q; ++p) {
        double z = 0.0;
        for (int l = p; l < q; ++l) z += Tm[p + l * kQB] * G[l + q * kQB];
        Tm[p + q * kQB] = -tq * z;
      }
      Tm[q + q * kQB] = tq;
      for (int p = q + 1; p < kQB; ++p) Tm[p + q * kQB] = 0.0;
    }
  }
  __syncthreads();
}

// One CTA's factor and form steps of a block, used where the cooperative launch of all SMs is
// refused: k_pq_factor is dgeqr2 on the block's kQB columns and its T, k_pq_form dorg2r on the
// block's own columns (the columns to its right are already formed).
__global__ void __launch_bounds__(512) k_pq_factor(const PanelDesc* __restrict__ descs, int j0,
                                                   double* __restrict__ taus, int ldtau, double* __restrict__ Ts,
                                                   int nblk) {
  __shared__ double red[40];
  __shared__ double sh[2];
  __shared__ double G[kQB * kQB], Tm[kQB * kQB];
  const PanelDesc D = descs[blockIdx.x];
  const int k = D.k;
  if (j0 >= k) return;
  double* A = D.A;
  const int64_t m = D.m, lda = D.lda;
  double* tau = taus + (int64_t)blockIdx.x * ldtau;
  const int jb = min(kQB, k - j0);
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nw = blockDim.x >> 5;
  for (int j = j0; j < j0 + jb; ++j) {  // dgeqr2 / dlarfg: beta = -sign(alpha) ||.||
    double* aj = A + (int64_t)j * lda;
    double part = 0.0;
    for (int64_t i = j + 1 + tid; i < m; i += blockDim.x) part += aj[i] * aj[i];
    const double sig = cta_sum(part, red);
    if (tid == 0) {
      const double alpha = aj[j];
      double tj = 0.0, beta = alpha, scal = 0.0;
      if (sig != 0.0) {
        const double nrm = sqrt(alpha * alpha + sig);
        beta = alpha >= 0.0 ? -nrm : nrm;
        tj = (beta - alpha) / beta;
        scal = 1.0 / (alpha - beta);
      }
      aj[j] = beta;
      sh[0] = scal;
      sh[1] = tj;
      tau[j] = tj;
    }
    __syncthreads();
    const double scal = sh[0], tj = sh[1];
    for (int64_t i = j + 1 + tid; i < m; i += blockDim.x) aj[i] *= scal;
    __syncthreads();
    if (tj != 0.0) {
      for (int c = j + 1 + w; c < j0 + jb; c += nw) {
        double* ac = A + (int64_t)c * lda;
        double acc = (lane == 0) ? ac[j] : 0.0;
        for (int64_t i = j + 1 + lane; i < m; i += 32) acc += aj[i] * ac[i];
        acc = warp_sum(acc) * tj;
        if (lane == 0) ac[j] -= acc;
        for (int64_t i = j + 1 + lane; i < m; i += 32) ac[i] -= acc * aj[i];
      }
    }
    __syncthreads();
  }
  if (j0 + jb < k) {
    panel_block_T(A, m, lda, j0, jb, tau, G, Tm);
    double* Tout = Ts + ((int64_t)blockIdx.x * nblk + j0 / kQB) * kQB * kQB;
    for (int e = tid; e < kQB * kQB; e += blockDim.x) Tout[e] = Tm[e];
  }
}

// dorg2r on the block's own columns j0 .. j1-1 (the columns to its right are already formed).
__global__ void __launch_bounds__(512) k_pq_form(const PanelDesc* __restrict__ descs, int j0,
                                                 const double* __restrict__ taus, int ldtau) {
  const PanelDesc D = descs[blockIdx.x];
  const int k = D.k;
  if (j0 >= k) return;
  double* A = D.A;
  const int64_t m = D.m, lda = D.lda;
  const double* tau = taus + (int64_t)blockIdx.x * ldtau;
  const int j1 = min(j0 + kQB, k);
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nw = blockDim.x >> 5;
  for (int j = j1 - 1; j >= j0; --j) {
    double* aj = A + (int64_t)j * lda;
    const double tj = tau[j];
    if (j < j1 - 1) {
      if (tid == 0) aj[j] = 1.0;
      __syncthreads();
      for (int c = j + 1 + w; c < j1; c += nw) {
        double* ac = A + (int64_t)c * lda;
        double acc = 0.0;
        for (int64_t i = j + lane; i < m; i += 32) acc += aj[i] * ac[i];
        acc = warp_sum(acc) * tj;
        for (int64_t i = j + lane; i < m; i += 32) ac[i] -= acc * aj[i];
      }
      __syncthreads();
    }
    for (int64_t i = j + 1 + tid; i < m; i += blockDim.x) aj[i] *= -tj;
    for (int64_t i = tid; i < j; i += blockDim.x) aj[i] = 0.0;
    if (tid == 0) aj[j] = 1.0 - tj;
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------------------
// Application of node factors to column blocks:
//   mode 0 (W^{-1}):  y2 -= Q2 (z2 - L22^{-1}(z2 - C' z1))
//   mode 1 (W^{-T}):  t = L22^{-T} z2;  y1 -= Q1 C t;  y2 -= Q2 (z2 - t)
//   mode 2 (W):       y2 += Q2 (C' z1 + L22 z2 - z2)
//   mode 3 (W'):      y1 += Q1 C z2;  y2 += Q2 (L22' z2 - z2)
//   mode 4 (pre-factor product): y1 += V (U' y2_in), y2 += U (V' y1_in) with Q1 = V, Q2 = U
//          reading x (in) and accumulating into y (out)
// with z1 = Q1' y1, z2 = Q2' y2.  One CTA per (item, CB columns), grid = (items, chunks).
//
// The FP64 pipe bounds it (two multiply-adds a clock and SM): a projection entry is a dot product
// over the rows by one warp, eight at a time so that the sums over the lanes take 9 additions for
// 8 entries instead of 40; an expansion takes a thread per row.  One warp per column, as before,
// left most of the SM idle and walked the r x r solve serially: 7.2 ms for one column at r = 496
// with 512-row panels, now 0.65 ms.  CB = 8 reads each Q once per 8 columns; a single right-hand
// side takes CB = 1, a rank whose vectors do not fit in shared memory 8 at a time 4, 2 or 1.
// ---------------------------------------------------------------------------------------------
namespace {

constexpr int kGaThreads = 256;
constexpr int kGaWarps = kGaThreads / 32;
constexpr int kGaStage = 512;   // rows of x staged per pass of a projection

// Sums v[0..8) over the warp's lanes; lane 4 b (b = 0..7) returns the sum of v[perm(b)] with
// perm(b) = 4 b2 + 2 b1 + b0 of lane bits 4, 3, 2.
__device__ __forceinline__ double reduce8(double (&v)[8], int lane) {
#pragma unroll
  for (int h = 4, o = 16; h > 0; h >>= 1, o >>= 1) {
#pragma unroll
    for (int k = 0; k < h; ++k) {
      const bool up = (lane & o) != 0;
      const double keep = up ? v[k + h] : v[k], send = up ? v[k] : v[k + h];
      v[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  double s = v[0];
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  return s;
}

// Z[c * ldz + q] += sign * sum_{i < n} A[i + q lda] x(i, c) for q < nq, c < CB; x staged in shared
// memory at xs[c * ldx + i].  Warps take 8 / CB entries q at a time.
template <int CB>
__device__ void ga_proj(const double* A, int64_t lda, int nq, int n, const double* xs, int ldx, double* Z, int ldz,
                        double sign) {
  constexpr int QB = 8 / CB;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int q0 = w * QB; q0 < nq; q0 += kGaWarps * QB) {
    double v[8] = {};
    const double* a[QB];
#pragma unroll
    for (int u = 0; u < QB; ++u) a[u] = A + (int64_t)min(q0 + u, nq - 1) * lda;
#pragma unroll 2
    for (int i = lane; i < n; i += 32) {
      double x[CB];
#pragma unroll
      for (int c = 0; c < CB; ++c) x[c] = xs[c * ldx + i];
#pragma unroll
      for (int u = 0; u < QB; ++u) {
        const double e = a[u][i];
#pragma unroll
        for (int c = 0; c < CB; ++c) v[u * CB + c] += e * x[c];
      }
    }
    const double s = reduce8(v, lane);
    const int k = ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
    const int q = q0 + k / CB;
    if ((lane & 3) == 0 && q < nq) Z[(k % CB) * ldz + q] += sign > 0.0 ? s : -s;
  }
}

// The same with x in global memory (column c at x + c ldx, nc of them): staged kGaStage rows at a
// time.  Zeroes Z first; ends with a barrier.
template <int CB>
__device__ void ga_proj_rows(const double* Q, int64_t s, int r, const double* x, int64_t ldx, int nc, double* xs,
                             double* Z) {
  for (int e = threadIdx.x; e < CB * r; e += kGaThreads) Z[e] = 0.0;
  for (int64_t i0 = 0; i0 < s; i0 += kGaStage) {
    const int n = (int)min((int64_t)kGaStage, s - i0);
    __syncthreads();
    for (int c = 0; c < CB; ++c)
      for (int i = threadIdx.x; i < n; i += kGaThreads) xs[c * kGaStage + i] = c < nc ? x[c * ldx + i0 + i] : 0.0;
    __syncthreads();
    ga_proj<CB>(Q + i0, s, r, n, xs, kGaStage, Z, r, 1.0);
  }
  __syncthreads();
}

// out(i, c) = sum_{l0 <= l < l1(i)} A[i + l lda] G[c * ldg + l] for a thread's row i
template <int CB>
__device__ __forceinline__ void ga_row(const double* A, int64_t lda, int64_t i, int l0, int l1, const double* G,
                                       int ldg, double (&acc)[CB]) {
#pragma unroll
  for (int c = 0; c < CB; ++c) acc[c] = 0.0;
  int l = l0;
  for (; l + 4 <= l1; l += 4) {
    double a[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) a[u] = A[i + (int64_t)(l + u) * lda];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int c = 0; c < CB; ++c) acc[c] += a[u] * G[c * ldg + l + u];
  }
  for (; l < l1; ++l) {
    const double a = A[i + (int64_t)l * lda];
#pragma unroll
    for (int c = 0; c < CB; ++c) acc[c] += a * G[c * ldg + l];
  }
}

// y(i, c) += sign Q G over the s rows of Q
template <int CB>
__device__ void ga_expand(const double* Q, int64_t s, int r, const double* G, double* y, int64_t ldy, int nc,
                          double sign) {
  for (int64_t i = threadIdx.x; i < s; i += kGaThreads) {
    double acc[CB];
    ga_row<CB>(Q, s, i, 0, r, G, r, acc);
#pragma unroll
    for (int c = 0; c < CB; ++c)
      if (c < nc) y[c * ldy + i] += sign > 0.0 ? acc[c] : -acc[c];
  }
}

// T <- L^{-1} T (trans = 0) or L^{-T} T for the lower triangular r x r L, CB columns of T (column
// c at T + c r) in shared memory, by blocks of 32 rows: a warp per column solves the diagonal block
// with a row per lane, then all threads update the other rows.
template <int CB>
__device__ void ga_trsv(const double* L, int r, double* T, int trans, double* xs) {
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  double* D = xs;  // 32 x 33, diagonal as reciprocals
  const int nb = (r + 31) / 32;
  for (int b = 0; b < nb; ++b) {
    const int i0 = 32 * (trans ? nb - 1 - b : b), ib = min(32, r - i0);
    __syncthreads();
    for (int e = tid; e < 32 * 32; e += kGaThreads) {
      const int i = e & 31, l = e >> 5;
      if (i < ib && l <= i) {
        const double v = L[i0 + i + (int64_t)(i0 + l) * r];
        D[i * 33 + l] = l == i ? 1.0 / v : v;
      }
    }
    __syncthreads();
    if (w < CB) {
      double t = lane < ib ? T[w * r + i0 + lane] : 0.0;
      for (int q = 0; q < ib; ++q) {
        const int l = trans ? ib - 1 - q : q;
        if (lane == l) t *= D[l * 33 + l];
        const double tl = __shfl_sync(0xffffffffu, t, l);
        if (trans ? lane < l : (lane > l && lane < ib)) t -= (trans ? D[l * 33 + lane] : D[lane * 33 + l]) * tl;
      }
      if (lane < ib) T[w * r + i0 + lane] = t;
    }
    __syncthreads();
    if (!trans) {
      for (int i = i0 + ib + tid; i < r; i += kGaThreads) {
        double acc[CB];
        ga_row<CB>(L, r, i, i0, i0 + ib, T, r, acc);
#pragma unroll
        for (int c = 0; c < CB; ++c) T[c * r + i] -= acc[c];
      }
    } else if (i0 > 0) {
      // rows l < i0 take the block's rows: column l of L, 32 consecutive entries
      ga_proj<CB>(L + i0, r, i0, ib, T + i0, r, T, r, -1.0);
    }
  }
  __syncthreads();
}

// The r x r part: from z1, z2 (in Z1, Z2) to the coefficients g1 (left in Z1; modes 1 and 3) and
// g2 (left in Z2) of the expansions y1 -/+= Q1 g1, y2 -/+= Q2 g2.
template <int CB>
__device__ void ga_middle(const GNodeDesc& N, int mode, double* Z1, double* Z2, double* T, double* xs) {
  const int r = N.r, tid = threadIdx.x;
  const double* C = N.C;
  const double* Lm = N.L22;
  if (mode == 0 || mode == 1) {
    for (int e = tid; e < CB * r; e += kGaThreads) T[e] = Z2[e];
    __syncthreads();
    if (mode == 0) ga_proj<CB>(C, r, r, r, Z1, r, T, r, -1.0);  // z2 - C' z1
    ga_trsv<CB>(Lm, r, T, mode, xs);
    for (int e = tid; e < CB * r; e += kGaThreads) Z2[e] -= T[e];
    if (mode == 1)
      for (int i = tid; i < r; i += kGaThreads) {
        double acc[CB];
        ga_row<CB>(C, r, i, 0, r, T, r, acc);
#pragma unroll
        for (int c = 0; c < CB; ++c) Z1[c * r + i] = acc[c];
      }
  } else {
    for (int e = tid; e < CB * r; e += kGaThreads) T[e] = -Z2[e];
    __syncthreads();
    if (mode == 2) {
      ga_proj<CB>(C, r, r, r, Z1, r, T, r, 1.0);
      __syncthreads();
    } else {
      ga_proj<CB>(Lm, r, r, r, Z2, r, T, r, 1.0);  // entries above the diagonal are stored zeros
    }
    for (int i = tid; i < r; i += kGaThreads) {
      double acc[CB];
      ga_row<CB>(mode == 2 ? Lm : C, r, i, 0, mode == 2 ? i + 1 : r, Z2, r, acc);
#pragma unroll
      for (int c = 0; c < CB; ++c) {
        if (mode == 2) T[c * r + i] += acc[c];
        else Z1[c * r + i] = acc[c];
      }
    }
    __syncthreads();
    for (int e = tid; e < CB * r; e += kGaThreads) Z2[e] = T[e];
  }
  __syncthreads();
}

template <int CB>
__global__ void __launch_bounds__(kGaThreads) k_gapply(const GApplyItem* __restrict__ items,
                                                       const GNodeDesc* __restrict__ nodes, int mode, double* X,
                                                       const double* Xin, int64_t ldX, int kX) {
  extern __shared__ double sm[];
  const GApplyItem I = items[blockIdx.x];
  if (I.big) return;  // large nodes go through the products over all SMs
  const GNodeDesc N = nodes[I.node];
  const int r = N.r;
  const int64_t ld = I.base ? I.ld : ldX;
  const int ncols = I.base ? I.ncols : kX, col = blockIdx.y * CB;
  if (col >= ncols || r == 0) return;
  const int nc = min(CB, ncols - col);
  double* Z1 = sm;
  double* Z2 = Z1 + CB * r;
  double* T = Z2 + CB * r;
  double* xs = T + CB * r;
  double* base = I.base ? I.base : X;
  double* y1 = base + I.off1 + (int64_t)col * ld;
  double* y2 = base + I.off2 + (int64_t)col * ld;
  if (mode == 4) {
    ga_proj_rows<CB>(N.Q2, N.s2, r, Xin + I.off2 + (int64_t)col * ldX, ldX, nc, xs, Z1);
    ga_proj_rows<CB>(N.Q1, N.s1, r, Xin + I.off1 + (int64_t)col * ldX, ldX, nc, xs, Z2);
    ga_expand<CB>(N.Q1, N.s1, r, Z1, y1, ld, nc, 1.0);
    ga_expand<CB>(N.Q2, N.s2, r, Z2, y2, ld, nc, 1.0);
    return;
  }
  if (mode == 0 || mode == 2) ga_proj_rows<CB>(N.Q1, N.s1, r, y1, ld, nc, xs, Z1);
  ga_proj_rows<CB>(N.Q2, N.s2, r, y2, ld, nc, xs, Z2);
  ga_middle<CB>(N, mode, Z1, Z2, T, xs);
  const double sign = mode < 2 ? -1.0 : 1.0;
  if (mode == 1 || mode == 3) ga_expand<CB>(N.Q1, N.s1, r, Z1, y1, ld, nc, sign);
  ga_expand<CB>(N.Q2, N.s2, r, Z2, y2, ld, nc, sign);
}

// The same in three launches for few items: the projections and the expansions spread over (item,
// columns, side and row chunk) CTAs, the r x r part in between.  Partial projections of item q,
// side d, chunk h, column c start at part + (((2 q + d) nchunk + h) ncol + c) ldr; the
// coefficients at coef + ((2 q + d) ncol + c) ldr (ncol: columns rounded up to CB, ldr: largest r).
// (One CTA a node took 4.1 and 8.1 ms for nodes of 4096 and 8192 rows with 8 right-hand sides.)
struct GSpread {
  double* part;
  double* coef;
  int nchunk, rows, ncol, ldr;
};

template <int CB>
__global__ void __launch_bounds__(kGaThreads) k_gproj(const GApplyItem* __restrict__ items,
                                                      const GNodeDesc* __restrict__ nodes, int mode, const double* X,
                                                      int64_t ldX, int kX, GSpread sp) {
  extern __shared__ double sm[];
  const GApplyItem I = items[blockIdx.x];
  if (I.big) return;
  const GNodeDesc N = nodes[I.node];
  const int r = N.r, d = blockIdx.z & 1, h = blockIdx.z >> 1, col = blockIdx.y * CB;
  const int ncols = I.base ? I.ncols : kX;
  const bool first = mode == 4 ? d == 1 : d == 0;  // Q1 and the rows c1 (mode 4: z1 = U' x2)
  if (col >= ncols || r == 0 || (d == 0 && (mode == 1 || mode == 3))) return;
  const int64_t s = first ? N.s1 : N.s2, i0 = (int64_t)h * sp.rows;
  if (i0 >= s) return;
  const int64_t ld = I.base ? I.ld : ldX;
  const double* x = (I.base ? I.base : X) + (first ? I.off1 : I.off2) + (int64_t)col * ld + i0;
  double* Z = sm;
  double* xs = Z + CB * r;
  const int nc = min(CB, ncols - col), n = (int)min((int64_t)sp.rows, s - i0);
  for (int e = threadIdx.x; e < CB * r; e += kGaThreads) Z[e] = 0.0;
  for (int j0 = 0; j0 < n; j0 += kGaStage) {
    const int nj = min(kGaStage, n - j0);
    __syncthreads();
    for (int c = 0; c < CB; ++c)
      for (int i = threadIdx.x; i < nj; i += kGaThreads) xs[c * kGaStage + i] = c < nc ? x[c * ld + j0 + i] : 0.0;
    __syncthreads();
    ga_proj<CB>((first ? N.Q1 : N.Q2) + i0 + j0, s, r, nj, xs, kGaStage, Z, r, 1.0);
  }
  __syncthreads();
  double* out = sp.part + ((((int64_t)2 * blockIdx.x + d) * sp.nchunk + h) * sp.ncol + col) * sp.ldr;
  for (int e = threadIdx.x; e < CB * r; e += kGaThreads) out[(int64_t)(e / r) * sp.ldr + e % r] = Z[e];
}

template <int CB>
__global__ void __launch_bounds__(kGaThreads) k_gmid(const GApplyItem* __restrict__ items,
                                                     const GNodeDesc* __restrict__ nodes, int mode, int kX,
                                                     GSpread sp) {
  extern __shared__ double sm[];
  const GApplyItem I = items[blockIdx.x];
  if (I.big) return;
  const GNodeDesc N = nodes[I.node];
  const int r = N.r, col = blockIdx.y * CB;
  if (col >= (I.base ? I.ncols : kX) || r == 0) return;
  double* z = sm;  // z1, z2, T
  double* xs = z + 3 * CB * r;
  for (int d = 0; d < 2; ++d) {
    const int64_t s = (mode == 4 ? d == 1 : d == 0) ? N.s1 : N.s2;
    const bool have = !(d == 0 && (mode == 1 || mode == 3));
    const int nh = (int)((s + sp.rows - 1) / sp.rows);
    const double* in = sp.part + (((int64_t)2 * blockIdx.x + d) * sp.nchunk * sp.ncol + col) * sp.ldr;
    for (int e = threadIdx.x; e < CB * r; e += kGaThreads) {
      double v = 0.0;
      const double* p = in + (int64_t)(e / r) * sp.ldr + e % r;
      if (have)
        for (int h = 0; h < nh; ++h) v += p[(int64_t)h * sp.ncol * sp.ldr];
      z[d * CB * r + e] = v;
    }
  }
  __syncthreads();
  if (mode != 4) ga_middle<CB>(N, mode, z, z + CB * r, z + 2 * CB * r, xs);
  for (int d = 0; d < 2; ++d) {
    double* out = sp.coef + (((int64_t)2 * blockIdx.x + d) * sp.ncol + col) * sp.ldr;
    for (int e = threadIdx.x; e < CB * r; e += kGaThreads) out[(int64_t)(e / r) * sp.ldr + e % r] = z[d * CB * r + e];
  }
}

template <int CB>
__global__ void __launch_bounds__(kGaThreads) k_gexpand(const GApplyItem* __restrict__ items,
                                                        const GNodeDesc* __restrict__ nodes, int mode, double* X,
                                                        int64_t ldX, int kX, GSpread sp) {
  extern __shared__ double G[];  // CB x r
  const GApplyItem I = items[blockIdx.x];
  if (I.big) return;
  const GNodeDesc N = nodes[I.node];
  const int r = N.r, d = blockIdx.z & 1, h = blockIdx.z >> 1, col = blockIdx.y * CB;
  const int ncols = I.base ? I.ncols : kX;
  if (col >= ncols || r == 0 || (d == 0 && (mode == 0 || mode == 2))) return;
  const int64_t s = d == 0 ? N.s1 : N.s2, i0 = (int64_t)h * sp.rows;
  if (i0 >= s) return;
  const int64_t i1 = min(s, i0 + sp.rows), ld = I.base ? I.ld : ldX;
  const int nc = min(CB, ncols - col);
  const double* in = sp.coef + (((int64_t)2 * blockIdx.x + d) * sp.ncol + col) * sp.ldr;
  for (int e = threadIdx.x; e < CB * r; e += kGaThreads) G[e] = in[(int64_t)(e / r) * sp.ldr + e % r];
  __syncthreads();
  double* y = (I.base ? I.base : X) + (d == 0 ? I.off1 : I.off2) + (int64_t)col * ld;
  const double* Q = d == 0 ? N.Q1 : N.Q2;
  for (int64_t i = i0 + threadIdx.x; i < i1; i += kGaThreads) {
    double acc[CB];
    ga_row<CB>(Q, s, i, 0, r, G, r, acc);
#pragma unroll
    for (int c = 0; c < CB; ++c)
      if (c < nc) y[c * ld + i] += mode < 2 ? -acc[c] : acc[c];
  }
}

// The r x r part of mode 0 alone for a node whose projections and expansion run as products over all SMs
// (columns of Z1, Z2, G2: r consecutive values), CB columns per CTA.
template <int CB>
__global__ void __launch_bounds__(kGaThreads) k_gsmall(const GNodeDesc* __restrict__ node,
                                                       const double* __restrict__ Z1, const double* __restrict__ Z2,
                                                       double* __restrict__ G2, int ncols) {
  extern __shared__ double sm[];
  const GNodeDesc N = *node;
  const int r = N.r, col = blockIdx.x * CB, nc = min(CB, ncols - col);
  double* z1 = sm;
  double* z2 = z1 + CB * r;
  double* T = z2 + CB * r;
  double* xs = T + CB * r;
  const int64_t off = (int64_t)col * r;
  for (int e = threadIdx.x; e < CB * r; e += kGaThreads) {
    z1[e] = e < nc * r ? Z1[off + e] : 0.0;
    z2[e] = e < nc * r ? Z2[off + e] : 0.0;
  }
  __syncthreads();
  ga_middle<CB>(N, 0, z1, z2, T, xs);
  for (int e = threadIdx.x; e < nc * r; e += kGaThreads) G2[off + e] = z2[e];
}

// shared memory of CB columns at rank r; the widest CB <= want whose vectors fit
size_t ga_smem(int cb, int r) {
  return ((size_t)3 * cb * std::max(r, 1) + std::max(cb * kGaStage, 32 * 33)) * sizeof(double);
}
int ga_width(int ncols, int r) {
  int cb = ncols == 1 ? 1 : ncols == 2 ? 2 : ncols <= 4 ? 4 : 8;
  while (cb > 1 && ga_smem(cb, r) > 200 * 1024) cb >>= 1;
  return cb;
}

// Shape of an application: how many columns a CTA takes and, when the items alone would not give
// six CTAs an SM, how the rows are split so that the projections and expansions do (chunks of 64
// rows or more, at most 64 of them, so that their sums stay a small part of the middle step and,
// with fewer than 12 CTAs an SM in all, their scratch small whatever the rows and columns).
struct GShape {
  int cb, cols, rows, nchunk;  // nchunk 0: one launch
};
GShape ga_shape(int n, int maxr, int maxcols, int64_t maxs) {
  GShape g{ga_width(maxcols, maxr), 0, 0, 0};
  if (n <= 0 || maxcols <= 0) return g;  // (a level without items, or with big ones only)
  g.cols = (maxcols + g.cb - 1) / g.cb;
  const int64_t ctas = (int64_t)n * g.cols;
  if (ctas >= 6 * 152) return g;
  const int64_t want = std::min<int64_t>((6 * 152 + 2 * ctas - 1) / (2 * ctas), 64);
  g.rows = (int)std::max<int64_t>(64, ((maxs + want - 1) / want + 31) / 32 * 32);
  g.nchunk = (int)((maxs + g.rows - 1) / g.rows);
  return g;
}

template <int CB>
void gapply_launch(const GApplyItem* items, int n, const GNodeDesc* nodes, int maxr, const GShape& g, int mode,
                   double* X, const double* Xin, int64_t ldX, int kX, double* scratch, cudaStream_t st) {
  const size_t sm = ga_smem(CB, maxr);
  if (g.nchunk == 0 || !scratch) {
    smem_limit((const void*)k_gapply<CB>, sm);
    k_gapply<CB><<<dim3((unsigned)n, (unsigned)g.cols), kGaThreads, sm, st>>>(items, nodes, mode, X, Xin, ldX, kX);
    return;
  }
  const int ncol = g.cols * CB;
  const GSpread sp{scratch, scratch + (int64_t)2 * n * g.nchunk * ncol * maxr, g.nchunk, g.rows, ncol, maxr};
  const size_t sp1 = ((size_t)CB * maxr + CB * kGaStage) * sizeof(double), sp2 = (size_t)CB * maxr * sizeof(double);
  smem_limit((const void*)k_gproj<CB>, sp1);
  smem_limit((const void*)k_gmid<CB>, sm);
  smem_limit((const void*)k_gexpand<CB>, sp2);
  const dim3 wide((unsigned)n, (unsigned)g.cols, (unsigned)(2 * g.nchunk));
  k_gproj<CB><<<wide, kGaThreads, sp1, st>>>(items, nodes, mode, mode == 4 ? Xin : X, ldX, kX, sp);
  k_gmid<CB><<<dim3((unsigned)n, (unsigned)g.cols), kGaThreads, sm, st>>>(items, nodes, mode, kX, sp);
  k_gexpand<CB><<<wide, kGaThreads, sp2, st>>>(items, nodes, mode, X, ldX, kX, sp);
}

template <int CB>
void gsmall_launch(const GNodeDesc* node, const double* Z1, const double* Z2, double* G2, int r, int ncols,
                   cudaStream_t st) {
  const size_t sm = ga_smem(CB, r);
  smem_limit((const void*)k_gsmall<CB>, sm);
  k_gsmall<CB><<<(unsigned)((ncols + CB - 1) / CB), kGaThreads, sm, st>>>(node, Z1, Z2, G2, ncols);
}

}  // namespace

// 2 sum log |diag(L22)| over the general nodes: one partial per node, a warp each (deterministic).
__global__ void k_glogdet(const GNodeDesc* __restrict__ nodes, double* __restrict__ partial) {
  const GNodeDesc N = nodes[blockIdx.x];
  double s = 0.0;
  for (int i = threadIdx.x; i < N.r; i += 32) s += 2.0 * log(fabs(N.L22[i + (int64_t)i * N.r]));
  s = warp_sum(s);
  if (threadIdx.x == 0) partial[blockIdx.x] = s;
}

}  // namespace

__global__ void __launch_bounds__(kAcaThreads, 3) k_aca(const double* __restrict__ pts, KParams kp,
                                                     const AcaBlock* __restrict__ blocks, int nblocks, int last_first,
                                                     double* P, uint8_t* F, int* __restrict__ piv, double rtol,
                                                     int* __restrict__ rank_out, int* __restrict__ status, int only,
                                                     int dyn) {
  extern __shared__ double dsm[];
  __shared__ AcaShared S;
  const int cid = (int)(blockIdx.x / cg::this_cluster().num_blocks());
  const int bid = only >= 0 ? only : (last_first ? nblocks - 1 - cid : cid);
  const AcaBlock B = blocks[bid];
  if (only < 0 && B.grid) return;  // compressed by k_aca_grid (the whole cluster leaves)
  const ClusterTeam team{&S, dsm + B.cap + 2 * kAcaChunk * kAcaSplit, B.cap + 1};
  const int fixed = 3 * B.cap + 2 + 2 * kAcaChunk * kAcaSplit;
  aca_run(team, S, dsm, dsm + fixed, dyn - fixed, cid, pts, kp, B, P, F, piv, rtol, rank_out + bid, status + bid);
}

__global__ void __launch_bounds__(kAcaThreads) k_aca_grid(const double* __restrict__ pts, KParams kp,
                                                          const AcaBlock* __restrict__ blocks, int bidx, double* P,
                                                          uint8_t* F, int* __restrict__ piv, double rtol,
                                                          int* __restrict__ rank_out, int* __restrict__ status,
                                                          double* scr, GridBar gb, int dyn) {
  extern __shared__ double dsm[];
  __shared__ AcaShared S;
  const AcaBlock B = blocks[bidx];
  const GridTeam team{gb, reinterpret_cast<AcaRec*>(scr), scr + 3 * gridDim.x * (sizeof(AcaRec) / sizeof(double)),
                      B.cap + 1};
  const int fixed = B.cap + 2 * kAcaChunk * kAcaSplit;
  aca_run(team, S, dsm, dsm + fixed, dyn - fixed, 0, pts, kp, B, P, F, piv, rtol, rank_out + bidx, status + bidx);
  if (blockIdx.x == 0 && threadIdx.x == 0 && *gb.err) status[bidx] = 3;
}

constexpr int kAcaGridMaxCtas = 152 * 2;
constexpr size_t kAcaSmem = 208 * 1024;  // dynamic shared memory of a CTA that has its SM to itself

// records, partial dots and (last) the barrier words of up to kAcaGridMaxCtas CTAs, in doubles
static int64_t aca_grid_words_at(int G, int cap) {
  return (int64_t)G * (3 * (int64_t)(sizeof(AcaRec) / sizeof(double)) + 2 * (cap + 1));
}
int64_t aca_grid_scratch(int cap) { return aca_grid_words_at(kAcaGridMaxCtas, cap) + 2; }

bool launch_aca_grid(const double* pts, KParams kp, const AcaBlock* blocks, int b, int cap, double* P, uint8_t* F,
                     int* piv, double rtol, int* rank, int* status, double* scratch, cudaStream_t st,
                     long long wait_limit) {
  int dev = 0, coop = 0, nsm = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (!coop) return false;
  const size_t sm = kAcaSmem;  // one CTA an SM: whatever the fixed arrays leave holds slices
  smem_limit((const void*)k_aca_grid, sm);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_aca_grid, kAcaThreads, sm) != cudaSuccess || per < 1) {
    cudaGetLastError();
    return false;
  }
  const int G = std::min(nsm, kAcaGridMaxCtas);
  int dyn = (int)(sm / sizeof(double));
  unsigned* words = reinterpret_cast<unsigned*>(scratch + aca_grid_words_at(G, cap));
  if (cudaMemsetAsync(words, 0, 4 * sizeof(unsigned), st) != cudaSuccess) return false;
  GridBar gb{words, words + 1, reinterpret_cast<volatile int*>(words + 2), wait_limit};
  void* args[] = {(void*)&pts, (void*)&kp, (void*)&blocks, (void*)&b, (void*)&P, (void*)&F, (void*)&piv,
                  (void*)&rtol, (void*)&rank, (void*)&status, (void*)&scratch, (void*)&gb, (void*)&dyn};
  if (cudaLaunchCooperativeKernel((const void*)k_aca_grid, dim3(G), dim3(kAcaThreads), args, sm, st) !=
      cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return true;
}

static void aca_launch(const double* pts, KParams kp, const AcaBlock* blocks, int nblocks, int last_first, int only,
                       int most, int maxcap, double* P, uint8_t* F, int* piv, double rtol, int* rank, int* status,
                       cudaStream_t st) {
  // the fixed arrays, then this CTA's share of an SM for slices when the CTAs fit at most three to
  // an SM (more, and the shared memory is worth more as L1 cache)
  size_t sm = ((size_t)3 * std::max(maxcap, 1) + 2 + 2 * kAcaChunk * kAcaSplit) * sizeof(double);
  smem_limit((const void*)k_aca, kAcaSmem);
  // CTAs per cluster: 16 where clusters of that size can be scheduled, else 8
  const int cs = std::min(most, cluster_limit((const void*)k_aca, kAcaThreads, kAcaSmem) >= 16 ? 16 : 8);
  const int per = ((only >= 0 ? 1 : nblocks) * cs + 151) / 152;
  if (per <= 3) sm = std::max(sm, kAcaSmem / per);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((only >= 0 ? 1 : nblocks) * cs));
  cfg.blockDim = dim3(kAcaThreads);
  cfg.dynamicSmemBytes = sm;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim = {(unsigned)cs, 1, 1};
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, k_aca, pts, kp, blocks, nblocks, last_first, P, F, piv, rtol, rank, status, only,
                     (int)(sm / sizeof(double)));
}

void launch_aca_one(const double* pts, KParams kp, const AcaBlock* blocks, int b, int maxcap, double* P,
                    uint8_t* F, int* piv, double rtol, int* rank, int* status, cudaStream_t st) {
  aca_launch(pts, kp, blocks, 1, 0, b, 16, maxcap, P, F, piv, rtol, rank, status, st);
}

// ---------------------------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------------------------
void launch_aca(const double* pts, KParams kp, const AcaBlock* blocks, int nblocks, int maxcap, double* P,
                uint8_t* F, int* piv, double rtol, int* rank, int* status, cudaStream_t st, int last_first, int cluster) {
  aca_launch(pts, kp, blocks, nblocks, last_first, -1, cluster, maxcap, P, F, piv, rtol, rank, status, st);
}

// ---------------------------------------------------------------------------------------------
// Factor and form steps of one 8-column block of ONE tall panel by all SMs (cooperative launch):
// CTA b owns the contiguous row slice [b*rows, (b+1)*rows); every sum over rows is formed as
// per-CTA partials that all CTAs add in CTA order after a bounded grid barrier (same value in
// every CTA, same bits on every run); the partial buffers alternate between two halves so that a
// phase never overwrites partials another CTA may still be reading; every element is updated by
// the CTA that owns its row.  The operations per element are those of k_pq_factor / k_pq_form
// (dgeqr2 / dlarfg and dorg2r rules); only the order of the row sums differs.
// ---------------------------------------------------------------------------------------------
constexpr int kPqParts = 32;  // partial slots per CTA per phase

__device__ __forceinline__ double sum_parts(const double* part, int G, int slot) {
  double s = 0.0;
  for (int q = 0; q < G; ++q) s += __ldcg(part + (int64_t)q * kPqParts + slot);
  return s;
}

// CTA partial of up to 28 values in one pass: red holds nw x kPqParts doubles
__device__ void cta_parts(double (&v)[kPqParts], int nv, double* red, double* out) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int t = 0; t < nv; ++t) {
    const double x = warp_sum(v[t]);
    if (lane == 0) red[w * kPqParts + t] = x;
  }
  __syncthreads();
  if (threadIdx.x < nv) {
    double s = 0.0;
    for (int q = 0; q < nw; ++q) s += red[q * kPqParts + threadIdx.x];
    out[threadIdx.x] = s;
  }
  __syncthreads();
}

__global__ void __launch_bounds__(256) k_pq_factor_grid(const PanelDesc* __restrict__ desc, int j0,
                                                        double* __restrict__ tau, double* __restrict__ Tout,
                                                        double* __restrict__ part, GridBar gb) {
  __shared__ double red[8 * kPqParts];
  const PanelDesc D = *desc;
  double* A = D.A;
  const int64_t m = D.m, lda = D.lda;
  const int jb = min(kQB, D.k - j0), j1 = j0 + jb;
  const int G = gridDim.x, b = blockIdx.x;
  const int64_t rows = (m + G - 1) / G, r0 = (int64_t)b * rows, r1 = min(m, r0 + rows);
  int phase = 0;
  auto slot = [&]() { return part + (int64_t)(phase & 1) * G * kPqParts; };
  for (int j = j0; j < j1; ++j) {
    double* aj = A + (int64_t)j * lda;
    const bool own_j = (j >= r0 && j < r1);
    // ||x||^2 over rows j+1 .. m-1
    double v[kPqParts];
    v[0] = 0.0;
    // alpha travels in slot 1 from the CTA owning row j (the other CTAs add exact zeros): the
    // owner overwrites A[j][j] with beta once it is past the barrier
    v[1] = (own_j && threadIdx.x == 0) ? aj[j] : 0.0;
    for (int64_t i = max(r0, (int64_t)j + 1) + threadIdx.x; i < r1; i += blockDim.x) v[0] += aj[i] * aj[i];
    cta_parts(v, 2, red, slot() + (int64_t)b * kPqParts);
    if (!grid_barrier(gb)) return;
    const double sig = sum_parts(slot(), G, 0);
    const double alpha = sum_parts(slot(), G, 1);
    ++phase;
    double tj = 0.0, beta = alpha, scal = 0.0;
    if (sig != 0.0) {
      const double nrm = sqrt(alpha * alpha + sig);
      beta = alpha >= 0.0 ? -nrm : nrm;
      tj = (beta - alpha) / beta;
      scal = 1.0 / (alpha - beta);
    }
    __syncthreads();  // every thread has read alpha before its owner overwrites it
    if (own_j && threadIdx.x == 0) aj[j] = beta;
    if (b == 0 && threadIdx.x == 0) tau[j] = tj;
    for (int64_t i = max(r0, (int64_t)j + 1) + threadIdx.x; i < r1; i += blockDim.x) aj[i] *= scal;
    __syncthreads();
    if (tj == 0.0 || j + 1 >= j1) continue;
    // v . A[:, c] for the block's columns c > j (unit entry of v at row j)
    const int nc = j1 - j - 1;
    for (int t = 0; t < nc; ++t) v[t] = 0.0;
    for (int64_t i = max(r0, (int64_t)j + 1) + threadIdx.x; i < r1; i += blockDim.x) {
      const double x = aj[i];
      for (int t = 0; t < nc; ++t) v[t] += x * A[(int64_t)(j + 1 + t) * lda + i];
    }
    if (own_j && threadIdx.x == 0)
      for (int t = 0; t < nc; ++t) v[t] += A[(int64_t)(j + 1 + t) * lda + j];
    cta_parts(v, nc, red, slot() + (int64_t)b * kPqParts);
    if (!grid_barrier(gb)) return;
    double acc[kQB];
    for (int t = 0; t < nc; ++t) acc[t] = sum_parts(slot(), G, t) * tj;
    ++phase;
    for (int64_t i = max(r0, (int64_t)j + 1) + threadIdx.x; i < r1; i += blockDim.x) {
      const double x = aj[i];
      for (int t = 0; t < nc; ++t) A[(int64_t)(j + 1 + t) * lda + i] -= acc[t] * x;
    }
    if (own_j && threadIdx.x == 0)
      for (int t = 0; t < nc; ++t) A[(int64_t)(j + 1 + t) * lda + j] -= acc[t];
    __syncthreads();
  }
  if (j1 >= D.k || Tout == nullptr) return;
  // T of the block (panel_block_T): G[p][q] = v_p[j0+q] + sum_{i > j0+q} v_p[i] v_q[i], p < q
  double v[kPqParts];
  int np = 0;
  for (int q = 1; q < jb; ++q)
    for (int p2 = 0; p2 < q; ++p2) v[np++] = 0.0;
  for (int64_t i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
    int t = 0;
    for (int q = 1; q < jb; ++q)
      for (int p2 = 0; p2 < q; ++p2, ++t)
        if (i > j0 + q) v[t] += A[(int64_t)(j0 + p2) * lda + i] * A[(int64_t)(j0 + q) * lda + i];
  }
  if (threadIdx.x == 0) {
    int t = 0;
    for (int q = 1; q < jb; ++q)
      for (int p2 = 0; p2 < q; ++p2, ++t)
        if (j0 + q >= r0 && j0 + q < r1) v[t] += A[(int64_t)(j0 + p2) * lda + j0 + q];
  }
  cta_parts(v, np, red, slot() + (int64_t)b * kPqParts);
  if (!grid_barrier(gb)) return;
  if (b != 0 || threadIdx.x != 0) return;
  double Gm[kQB * kQB], Tm[kQB * kQB];
  {
    int t = 0;
    for (int q = 1; q < jb; ++q)
      for (int p2 = 0; p2 < q; ++p2, ++t) Gm[p2 + q * kQB] = sum_parts(slot(), G, t);
  }
  for (int q = 0; q < jb; ++q) {
    const double tq = tau[j0 + q];
    for (int p2 = 0; p2 < q; ++p2) {
      double z = 0.0;
      for (int l = p2; l < q; ++l) z += Tm[p2 + l * kQB] * Gm[l + q * kQB];
      Tm[p2 + q * kQB] = -tq * z;
    }
    Tm[q + q * kQB] = tq;
    for (int p2 = q + 1; p2 < kQB; ++p2) Tm[p2 + q * kQB] = 0.0;
  }
  for (int e = 0; e < kQB * kQB; ++e) Tout[e] = (e % kQB < jb && e / kQB < jb) ? Tm[e] : 0.0;
}

// dorg2r on the block's own columns j0 .. j1-1 of one tall panel by all SMs
__global__ void __launch_bounds__(256) k_pq_form_grid(const PanelDesc* __restrict__ desc, int j0,
                                                      const double* __restrict__ tau, double* __restrict__ part,
                                                      GridBar gb) {
  __shared__ double red[8 * kPqParts];
  const PanelDesc D = *desc;
  double* A = D.A;
  const int64_t m = D.m, lda = D.lda;
  const int j1 = min(j0 + kQB, D.k);
  const int G = gridDim.x, b = blockIdx.x;
  const int64_t rows = (m + G - 1) / G, r0 = (int64_t)b * rows, r1 = min(m, r0 + rows);
  int phase = 0;
  for (int j = j1 - 1; j >= j0; --j) {
    double* aj = A + (int64_t)j * lda;
    const double tj = tau[j];
    const bool own_j = (j >= r0 && j < r1);
    if (j < j1 - 1) {
      // v = e_j + A[j+1:, j]; c <- c - tau (v . c) v for the block's columns c > j
      const int nc = j1 - j - 1;
      double v[kPqParts];
      for (int t = 0; t < nc; ++t) v[t] = 0.0;
      for (int64_t i = max(r0, (int64_t)j + 1) + threadIdx.x; i < r1; i += blockDim.x) {
        const double x = aj[i];
        for (int t = 0; t < nc; ++t) v[t] += x * A[(int64_t)(j + 1 + t) * lda + i];
      }
      if (own_j && threadIdx.x == 0)
        for (int t = 0; t < nc; ++t) v[t] += A[(int64_t)(j + 1 + t) * lda + j];
      double* sl = part + (int64_t)(phase & 1) * G * kPqParts;
      cta_parts(v, nc, red, sl + (int64_t)b * kPqParts);
      if (!grid_barrier(gb)) return;
      double acc[kQB];
      for (int t = 0; t < nc; ++t) acc[t] = sum_parts(sl, G, t) * tj;
      ++phase;
      for (int64_t i = max(r0, (int64_t)j + 1) + threadIdx.x; i < r1; i += blockDim.x) {
        const double x = aj[i];
        for (int t = 0; t < nc; ++t) A[(int64_t)(j + 1 + t) * lda + i] -= acc[t] * x;
      }
      if (own_j && threadIdx.x == 0)
        for (int t = 0; t < nc; ++t) A[(int64_t)(j + 1 + t) * lda + j] -= acc[t];
    }
    for (int64_t i = max(r0, (int64_t)j + 1) + threadIdx.x; i < r1; i += blockDim.x) aj[i] *= -tj;
    for (int64_t i = r0 + threadIdx.x; i < min(r1, (int64_t)j); i += blockDim.x) aj[i] = 0.0;
    if (own_j && threadIdx.x == 0) aj[j] = 1.0 - tj;
    __syncthreads();
  }
}

// explicit reflector block V (rows j0 .. m-1 of columns j0 .. j0+jb-1: unit diagonal, zeros
// above it, the stored vectors below), column-major with leading dimension m - j0
__global__ void k_pq_vcopy(const PanelDesc* __restrict__ desc, int j0, double* __restrict__ V) {
  const PanelDesc D = *desc;
  const int jb = min(kQB, D.k - j0);
  const int64_t mr = D.m - j0;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < mr * jb; e += (int64_t)gridDim.x * blockDim.x) {
    const int p = (int)(e / mr);
    const int64_t i = e - (int64_t)p * mr;
    V[e] = (i == p) ? 1.0 : (i > p ? D.A[(int64_t)(j0 + p) * D.lda + j0 + i] : 0.0);
  }
}

int64_t panel_qr_gemm_scratch(const PanelDesc* hdescs, int n, int kmax) {
  int64_t mbig = 0;
  for (int p = 0; p < n; ++p)
    if (hdescs[p].big) mbig = std::max<int64_t>(mbig, hdescs[p].m);
  return mbig * kQB + 2 * (int64_t)kQB * std::max(kmax, 1) + 2 * 152 * kPqParts + 8 +
         dgemm_scratch(1, kQB, std::max(kmax, 1), mbig);
}

// C[:, j1:k] <- (I - V op(T) V') C[:, j1:k] for big panel p, block j0: W = V' C, W2 = op(T) W,
// C -= V W2 (op(T) = T' while factoring, T while forming Q)
static void panel_block_gemm(const PanelDesc* descs, const PanelDesc& D, int p, int j0, int nblk, const double* Ts,
                             double* scr, int kmax, double* split, int64_t split_len, int transT, cudaStream_t st) {
  const int k = D.k;
  if (j0 >= k) return;
  const int jb = std::min(kQB, k - j0), j1 = j0 + jb;
  const int nt = k - j1;
  if (nt <= 0) return;
  const int64_t mr = D.m - j0;
  double* V = scr;
  double* W = V + mr * kQB;
  double* W2 = W + (int64_t)kQB * kmax;
  const unsigned g = (unsigned)std::min<int64_t>((mr * jb + 255) / 256, 4096);
  k_pq_vcopy<<<g, 256, 0, st>>>(descs + p, j0, V);
  const double* Tm = Ts + ((int64_t)p * nblk + j0 / kQB) * kQB * kQB;
  double* C = D.A + (int64_t)j1 * D.lda + j0;
  launch_dgemm(1, jb, nt, mr, 1.0, V, mr, C, D.lda, 0.0, W, jb, split, split_len, st);
  launch_dgemm(transT, jb, nt, jb, 1.0, Tm, kQB, W, jb, 0.0, W2, jb, nullptr, 0, st);
  launch_dgemm(0, mr, nt, jb, -1.0, V, mr, W2, jb, 1.0, C, D.lda, nullptr, 0, st);
}

// grid size of the cooperative factor / form steps of a tall panel (0: cooperative launch
// unavailable); every CTA must be resident at once
static int pq_grid_size(int64_t m) {
  static int nsm = -1, per = 0;
  if (nsm < 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    int coop = 0;
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    if (!coop || cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_pq_factor_grid, 256, 0) != cudaSuccess ||
        per < 1) {
      cudaGetLastError();
      per = 0;
    }
    int per2 = 0;
    if (per > 0 && (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per2, k_pq_form_grid, 256, 0) != cudaSuccess ||
                    per2 < 1)) {
      cudaGetLastError();
      per = 0;
    }
  }
  if (per == 0) return 0;
  return (int)std::max<int64_t>(1, std::min<int64_t>(nsm, m / 512));
}

void launch_panel_qr_gemm(const PanelDesc* descs, const PanelDesc* hdescs, int n, int kmax, double* taus,
                          double* Ts, double* gemm_scratch, int* grid_err, cudaStream_t st,
                          long long wait_limit) {
  if (n <= 0 || kmax <= 0) return;
  const int nblk = (kmax + kQB - 1) / kQB;
  // scratch after the GEMM buffers: partials of the cooperative steps and the barrier words
  int64_t mbig = 0;
  for (int p = 0; p < n; ++p)
    if (hdescs[p].big) mbig = std::max<int64_t>(mbig, hdescs[p].m);
  double* part = gemm_scratch + mbig * kQB + 2 * (int64_t)kQB * std::max(kmax, 1);
  unsigned* words = reinterpret_cast<unsigned*>(part + 2 * 152 * kPqParts);
  double* split = part + 2 * 152 * kPqParts + 8;  // partial products of the split V'C reductions
  const int64_t split_len = dgemm_scratch(1, kQB, std::max(kmax, 1), mbig);
  cudaMemsetAsync(words, 0, 4 * sizeof(unsigned), st);
  GridBar gb{words, words + 1, grid_err, wait_limit};
  auto factor_big = [&](int p, int b) {
    const int G = pq_grid_size(hdescs[p].m);
    const PanelDesc* dp = descs + p;
    int j0 = b * kQB;
    double* tau = taus + (int64_t)p * kmax;
    double* Tout = Ts + ((int64_t)p * nblk + b) * kQB * kQB;
    if (G > 0 && G <= 152) {
      void* args[] = {(void*)&dp, (void*)&j0, (void*)&tau, (void*)&Tout, (void*)&part, (void*)&gb};
      if (cudaLaunchCooperativeKernel((const void*)k_pq_factor_grid, dim3(G), dim3(256), args, 0, st) == cudaSuccess)
        return;
      cudaGetLastError();
    }
    k_pq_factor<<<1, 512, 0, st>>>(dp, j0, tau, kmax, Ts + (int64_t)p * nblk * kQB * kQB, nblk);
  };
  auto form_big = [&](int p, int b) {
    const int G = pq_grid_size(hdescs[p].m);
    const PanelDesc* dp = descs + p;
    int j0 = b * kQB;
    const double* tau = taus + (int64_t)p * kmax;
    if (G > 0 && G <= 152) {
      void* args[] = {(void*)&dp, (void*)&j0, (void*)&tau, (void*)&part, (void*)&gb};
      if (cudaLaunchCooperativeKernel((const void*)k_pq_form_grid, dim3(G), dim3(256), args, 0, st) == cudaSuccess)
        return;
      cudaGetLastError();
    }
    k_pq_form<<<1, 512, 0, st>>>(dp, j0, tau, kmax);
  };
  for (int b = 0; b < nblk; ++b) {
    for (int p = 0; p < n; ++p)
      if (hdescs[p].big && b * kQB < hdescs[p].k) factor_big(p, b);
    for (int p = 0; p < n; ++p)
      if (hdescs[p].big)
        panel_block_gemm(descs, hdescs[p], p, b * kQB, nblk, Ts, gemm_scratch, kmax, split, split_len, 1, st);
  }
  launch_panel_rout(descs, n, kmax, 1, st);
  for (int b = nblk - 1; b >= 0; --b) {
    for (int p = 0; p < n; ++p)
      if (hdescs[p].big)
        panel_block_gemm(descs, hdescs[p], p, b * kQB, nblk, Ts, gemm_scratch, kmax, split, split_len, 0, st);
    for (int p = 0; p < n; ++p)
      if (hdescs[p].big && b * kQB < hdescs[p].k) form_big(p, b);
  }
}

int64_t panel_qr_gemm_taus(int n, int kmax) {
  const int nblk = (kmax + kQB - 1) / kQB;
  return (int64_t)n * kmax + (int64_t)n * nblk * kQB * kQB;
}

int64_t gapply_scratch(int n, int maxr, int maxcols, int64_t maxs) {
  const GShape g = ga_shape(n, maxr, maxcols, maxs);
  return (int64_t)2 * n * (g.nchunk > 0 ? g.nchunk + 1 : 0) * g.cols * g.cb * maxr;
}

int launch_gapply(const GApplyItem* items, int n, const GNodeDesc* nodes, int maxr, int maxcols, int64_t maxs, int mode,
                  double* X, const double* Xin, int64_t ldX, int kX, double* scratch, cudaStream_t st) {
  if (n <= 0 || maxcols <= 0) return 0;
  const GShape g = ga_shape(n, maxr, maxcols, maxs);
  (g.cb == 8   ? gapply_launch<8>
   : g.cb == 4 ? gapply_launch<4>
   : g.cb == 2 ? gapply_launch<2>
               : gapply_launch<1>)(items, n, nodes, maxr, g, mode, X, Xin, ldX, kX, scratch, st);
  return g.nchunk > 0 && scratch ? 3 : 1;
}

void launch_gsmall(const GNodeDesc* node, const double* Z1, const double* Z2, double* G2, int r, int ncols,
                   cudaStream_t st) {
  if (ncols <= 0 || r <= 0) return;
  const int cb = ga_width(ncols, r);
  (cb == 8 ? gsmall_launch<8> : cb == 4 ? gsmall_launch<4> : cb == 2 ? gsmall_launch<2> : gsmall_launch<1>)(
      node, Z1, Z2, G2, r, ncols, st);
}

void launch_glogdet(const GNodeDesc* nodes, int nn, double* partial, cudaStream_t st) {
  k_glogdet<<<nn, 32, 0, st>>>(nodes, partial);
}

}  // namespace km
