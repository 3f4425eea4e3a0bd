// Dense symmetric FP64 eigensolver on the GPU: the Rayleigh-Ritz step of the
// block Krylov-Schur solver (sg_lanczos), which replaces the small eigenproblem
// ARPACK solves inside the reference's eigsh call
// (snapatac2-python/src/embedding.rs:155-171).
//
// GB300 runs FP64 at about two fused multiply-adds per clock per SM, so one
// CTA would need milliseconds for the O(n^3) reduction of a 200 x 200 matrix
// and tens of milliseconds at 576 x 576.  The work is spread instead:
//
//   tridiag    Householder reduction A = Q T Qᵀ on one thread-block cluster
//              (up to 16 CTAs).  Row i of A lives in the shared memory of CTA
//              i mod CS; each step passes the product A v on through
//              distributed shared memory, with one cluster barrier per step
//              (buffers alternate between steps).
//   bisect     eigenvalues of T by multisection on Sturm counts: one warp per
//              wanted eigenvalue, 32 shifts per round, to absolute accuracy
//              eps·‖T‖ (LAPACK dstebz's default).
//   invit      eigenvectors of T by inverse iteration with a pivoted
//              tridiagonal LU (as LAPACK dstein): one warp per cluster of
//              near-degenerate eigenvalues (1e-9 ‖T‖), modified Gram-Schmidt
//              inside a cluster.
//   backtr     eigenvectors of A = Q z: one CTA per vector applies the
//              reflectors in reverse order, eight at a time.
//   orth       all the vectors to the closest orthonormal set: separately
//              iterated vectors of eigenvalues 1e-9..1e-3 ‖T‖ apart are
//              orthogonal only to eps ‖T‖ / gap; moving them by that much
//              moves their residuals by ~eps ‖T‖.  Two steps of a quadratic
//              iteration spread over the GPU (0.26 ms for 288 vectors of
//              length 336; a Cholesky-QR with its factor on one CTA took 7.0);
//              vectors too far off for two steps (an inverse iteration that
//              did not converge) still take the Cholesky-QR.
//
// Every sum runs in a fixed order, so results are reproducible run to run.
#include <cooperative_groups.h>
#include <float.h>

#include <atomic>

#include "common.cuh"
#include "internal.h"

namespace cg = cooperative_groups;

namespace sg {
namespace {

constexpr int kTriThreads = 256;
constexpr int kMaxCluster = 16;
// The reduction forms products of three entries of the matrix (uᵀv), so it
// runs on entries scaled by a power of two when the largest is not within
// 2^±kTriRange (d and e are scaled back).
constexpr int kTriRange = 100;

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Shared memory of the reduction: rows [R][n], v[2][n], u[2][n], 2 x
// kMaxCluster x kTriWarps partial sums of uᵀv, one per warp of the cluster,
// per-warp partials, 8 scalars.
constexpr int kTriWarps = kTriThreads / 32;
inline size_t tridiag_smem(int n, int CS) {
  const int R = (n + CS - 1) / CS;
  return ((size_t)R * n + 4 * (size_t)n + 2 * kMaxCluster * kTriWarps + kTriWarps + 8) * sizeof(double);
}

// GB300 runs FP64 at about two lanes per clock per SM: a warp-wide FP64
// instruction holds its SM sub-partition for 64 clocks and the next one that
// needs its result waits longer, so a step costs its FP64 work plus a chain of
// dependent operations.  One cluster barrier per step: step j
//   1. forms w = τ u + K v of the reflector before it (u = A v arrived over
//      distributed shared memory in step j - 1, K = -τ² uᵀv / 2 from the
//      warps' partial sums),
//   2. pulls row j from its owner, applies that reflector to it and finds
//      reflector j from the result -- in every CTA, with the same operations,
//      so nothing is broadcast,
//   3. applies the rank-2 update to the rows this CTA owns and multiplies them
//      by the new v in the same pass, and sends the products to every CTA.
// The reflector is not scaled to a unit first element (H = I - τ v vᵀ with
// τ = 1 / (μ (μ + |α|)), μ the norm of the row's part below the diagonal), so
// the matrix pass starts after one square root; the reciprocal for τ, first
// used in the next step, runs beside the pass.  With the reflector made by the
// owner and broadcast, and the update and the product as two passes between
// two cluster barriers, a step at n = 336 took 7.9 us; it takes 6.6 (FP64 work
// about 2.5; the rest is the chain: a cluster barrier behind remote stores is
// 1,650 clocks, each butterfly 500).  128 threads take 2.60 ms at n = 336, 256
// 2.21, 512 2.35.
template <int CS>
__global__ void __launch_bounds__(kTriThreads)
tridiag_kernel(int n, const double* __restrict__ A, int64_t lda, double* __restrict__ d, double* __restrict__ e,
               double* __restrict__ tau, double* __restrict__ V) {
  static_assert(CS <= kMaxCluster, "slots");
  cg::cluster_group cl = cg::this_cluster();
  const int rank = CS > 1 ? (int)cl.block_rank() : 0;
  extern __shared__ double smem_d[];
  const int R = (n + CS - 1) / CS;
  double* Al = smem_d;
  double* vb = Al + (size_t)R * n;
  double* ub = vb + 2 * n;
  double* slots = ub + 2 * n;
  double* red = slots + 2 * kMaxCluster * kTriWarps;
  double* sc = red + kTriWarps;  // 0: K, 1: w_j, 2: μ (μ + |α|), 3: τ, 4: the scaling back
  constexpr int kSlots = CS * kTriWarps, kPer = (kRitzMaxN + kTriThreads - 1) / kTriThreads;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned top = 0;  // high word of the largest |A_ij| of this CTA's rows
  for (int t = threadIdx.x; t < R * n; t += blockDim.x) {
    const int li = t / n, c = t % n;
    const int i = li * CS + rank;
    const double x = i < n ? A[(int64_t)i * lda + c] : 0.0;
    Al[t] = x;
    const unsigned h = (unsigned)__double2hiint(x) & 0x7fffffffu;
    top = h > top ? h : top;
  }
  top = __reduce_max_sync(0xffffffffu, top);
  if (lane == 0) slots[warp] = __hiloint2double((int)top, 0);
  if (CS > 1) cl.sync(); else __syncthreads();
  top = 0;
  for (int q = lane; q < kSlots; q += 32) {
    const double* other = CS > 1 ? cl.map_shared_rank(slots, q / kTriWarps) : slots;
    top = max(top, (unsigned)__double2hiint(other[q % kTriWarps]));
  }
  top = __reduce_max_sync(0xffffffffu, top);  // the same in every warp of the cluster
  double back = 1.0;
  if (top < (1023u - kTriRange) << 20 || (top >= (1023u + kTriRange) << 20 && top < 0x7ff00000u)) {
    const int te = (int)(top >> 20), up = max(min(1023 - te, 1000), -1022);  // the largest entry to about 1
    const double f = __longlong_as_double((long long)(1023 + up) << 52);
    back = __longlong_as_double((long long)(1023 - up) << 52);
    for (int t = threadIdx.x; t < R * n; t += blockDim.x) Al[t] *= f;
  }
  if (threadIdx.x == 0) sc[4] = back;
  if (CS > 1) cl.sync(); else __syncthreads();
  // steps 0 .. n-3 make reflectors; step n-2 only finishes the last 2 x 2 block
  for (int j = 0; j + 1 < n; ++j) {
    double* v = vb + (j & 1) * n;
    const double* vp = vb + ((j & 1) ^ 1) * n;
    double* w = ub + ((j & 1) ^ 1) * n;  // u of step j - 1, then its w
    double* un = ub + (j & 1) * n;
    const double* row_j = (CS > 1 ? cl.map_shared_rank(Al, j % CS) : Al) + (size_t)(j / CS) * n;
    double rr[kPer];
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
      const int k = j + (int)threadIdx.x + q * kTriThreads;
      rr[q] = k < n ? row_j[k] : 0.0;
    }
    if (j > 0) {
      if (warp == 0) {
        const double* sl = slots + ((j & 1) ^ 1) * (kMaxCluster * kTriWarps);
        double x = 0.0;
        for (int q = lane; q < kSlots; q += 32) x += sl[q];
        x = warp_sum_d(x);
        if (lane == 0) {
          const double tp = sc[3], K = -0.5 * tp * (tp * x);
          sc[0] = K;
          sc[1] = fma(tp, w[j], K * vp[j]);
        }
      }
      __syncthreads();
      const double tp = sc[3], K = sc[0], wj = sc[1], vj = vp[j];
#pragma unroll
      for (int q = 0; q < kPer; ++q) {
        const int k = j + (int)threadIdx.x + q * kTriThreads;
        if (k < n) {
          const double wk = fma(tp, w[k], K * vp[k]);
          w[k] = wk;
          rr[q] = fma(-vj, wk, fma(-wj, vp[k], rr[q]));
        }
      }
    }
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
      const int k = j + (int)threadIdx.x + q * kTriThreads;
      if (k < n) {
        v[k] = rr[q];
        if (k >= j + 2) s = fma(rr[q], rr[q], s);
      }
    }
    if (j + warp * 32 < n) s = warp_sum_d(s);  // a warp past the row's end has nothing to add
    if (lane == 0) red[warp] = s;
    __syncthreads();
    if (j + 2 == n) break;
    if (warp == 0) {
      double sigma = lane < kTriWarps ? red[lane] : 0.0;
#pragma unroll
      for (int o = kTriWarps / 2; o; o >>= 1) sigma += __shfl_xor_sync(0xffffffffu, sigma, o);
      if (lane == 0) {
        const double alpha = v[j + 1];
        double beta = alpha, den = 0.0;
        const double x = fma(alpha, alpha, sigma);
        if (sigma > 0.0 && x >= 0x1p-1000) {  // below, the row is done: 2^-400 of the matrix at most
          // x rsqrt(x): 350 + 64 clocks of this chain, a square root 675
          const double mu = x * rsqrt(x);
          beta = alpha <= 0.0 ? mu : -mu;
          den = mu * (mu + fabs(alpha));
          v[j + 1] = alpha - beta;
        }
        sc[2] = den;
        if (rank == j % CS) {
          d[j] = v[j] * sc[4];
          e[j] = beta * sc[4];
        }
      }
    }
    __syncthreads();
    if (threadIdx.x == kTriThreads - 1) {  // the last warp has the fewest rows
      const double den = sc[2], tj = den > 0.0 ? 1.0 / den : 0.0;
      sc[3] = tj;
      if (rank == j % CS) tau[j] = tj;
    }
    if (rank == (j + 1) % CS)  // not the CTA with the most rows left
      for (int k = j + 1 + (int)threadIdx.x; k < n; k += kTriThreads) V[(int64_t)j * n + k] = v[k];
    // owned trailing rows: A <- A - v_{j-1} wᵀ - w v_{j-1}ᵀ, u_i = A_i v
    const int first = j + 1 - rank;
    const int li0 = first <= 0 ? 0 : (first + CS - 1) / CS;
    double sv = 0.0;
    for (int li = li0 + warp; li < R; li += kTriWarps) {
      const int i = li * CS + rank;
      if (i >= n) break;
      double* row = Al + (size_t)li * n;
      double acc = 0.0;
      if (j > 0) {
        const double vi = vp[i], wi = w[i];
        for (int k = j + 1 + lane; k < n; k += 32) {
          const double x = fma(-vi, w[k], fma(-wi, vp[k], row[k]));
          row[k] = x;
          acc = fma(x, v[k], acc);
        }
      } else {
        for (int k = 1 + lane; k < n; k += 32) acc = fma(row[k], v[k], acc);
      }
      acc = warp_sum_d(acc);
      sv = fma(acc, v[i], sv);
      if (lane < CS) (CS > 1 ? cl.map_shared_rank(un, lane) : un)[i] = acc;
    }
    if (lane < CS)
      (CS > 1 ? cl.map_shared_rank(slots, lane) : slots)[(j & 1) * (kMaxCluster * kTriWarps) + rank * kTriWarps + warp] =
          sv;
    if (CS > 1) cl.sync(); else __syncthreads();
  }
  // the last 2 x 2 block: row n-2 is in v of step n-2; the last diagonal
  // element still lacks the last reflector's update
  if (rank == 0 && threadIdx.x == 0) {
    const double* row = (CS > 1 ? cl.map_shared_rank(Al, (n - 1) % CS) : Al) + (size_t)((n - 1) / CS) * n;
    double x = row[n - 1];
    if (n >= 2) {
      const double* v = vb + ((n - 2) & 1) * n;
      d[n - 2] = v[n - 2] * sc[4];
      e[n - 2] = v[n - 1] * sc[4];
      tau[n - 2] = 0.0;
      if (n >= 3) {
        const double vl = vb[((n - 3) & 1) * n + n - 1], wl = ub[((n - 3) & 1) * n + n - 1];
        x = fma(-vl, wl, fma(-wl, vl, x));
      }
    }
    d[n - 1] = x * sc[4];
    tau[n - 1] = 0.0;
  }
  if (CS > 1) cl.sync();
}

// Gershgorin interval, ‖T‖ (max absolute row sum) and the pivot floor of the
// Sturm recurrence (LAPACK: safe minimum x max(1, max e²)); one warp.
struct TriBounds {
  double lo, hi, tnorm, pivmin;
};

__device__ TriBounds tri_bounds_warp(int n, const double* __restrict__ d, const double* __restrict__ e) {
  const int lane = threadIdx.x & 31;
  double lo = DBL_MAX, hi = -DBL_MAX, tn = 0.0, e2 = 0.0;
  for (int i = lane; i < n; i += 32) {
    const double r = (i > 0 ? fabs(e[i - 1]) : 0.0) + (i + 1 < n ? fabs(e[i]) : 0.0);
    lo = fmin(lo, d[i] - r);
    hi = fmax(hi, d[i] + r);
    tn = fmax(tn, fabs(d[i]) + r);
    if (i + 1 < n) e2 = fmax(e2, e[i] * e[i]);
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    tn = fmax(tn, __shfl_xor_sync(0xffffffffu, tn, o));
    e2 = fmax(e2, __shfl_xor_sync(0xffffffffu, e2, o));
  }
  TriBounds b;
  b.tnorm = tn;
  b.pivmin = DBL_MIN * fmax(1.0, e2);
  const double pad = 2.0 * DBL_EPSILON * tn + 2.0 * b.pivmin;
  b.lo = lo - pad;
  b.hi = hi + pad;
  return b;
}

// Number of eigenvalues of T below x (e2 = squared off-diagonal), as the
// number of sign changes of the Sturm sequence of leading principal minors
// p_i = (d_i - x) p_{i-1} - e²_{i-1} p_{i-2} (Givens; Wilkinson, The
// Algebraic Eigenvalue Problem, 5.37-5.45): q_i = p_i / p_{i-1} <= 0 exactly
// when p_i and p_{i-1} differ in sign.  This form has no division: GB300
// runs an FP64 division as a chain of dependent FP64 operations (several
// hundred clocks), so the ratio form q_i = (d_i - x) - e²/q_{i-1} costs about
// four times as much per step.  The pair (p_i, p_{i-1}) is rescaled by an
// exact power of two whenever its larger exponent leaves [2^-400, 2^400], so
// it neither overflows nor underflows.  A zero minor is replaced by a tiny
// value of the sign opposite to its predecessor, which counts it as
// negative, as the ratio form's pivot floor does.  Signs and exponents are
// read as integers, off the FP64 pipe.
// The common step is three FP64 operations and a range test on the high words;
// the zero and rescaling cases, in which the whole warp takes part, are behind
// one warp-uniform branch: as two conditions per lane they were compiled to
// FP64 selects in every step, 695 clocks a step against 280 (1,280 -> 520 us
// for 288 values of a 336 x 336 matrix).
__device__ __forceinline__ int sturm_count(int n, const double* __restrict__ d, const double* __restrict__ e2,
                                           double x) {
  constexpr unsigned kLow = (1023u - 400u) << 20, kHigh = (1023u + 401u) << 20;
  double pm = 1.0;
  double p = d[0] - x;
  if (p == 0.0) p = -DBL_MIN;
  unsigned hp = (unsigned)__double2hiint(p);
  int c = (int)(hp >> 31);
  for (int i = 1; i < n; ++i) {
    double pn = fma(-e2[i - 1], pm, (d[i] - x) * p);
    unsigned hn = (unsigned)__double2hiint(pn);
    // in range: the larger exponent of the pair within 2^±400 and the new
    // minor a normal number
    const unsigned an = hn & 0x7fffffffu, ap = hp & 0x7fffffffu, big = an > ap ? an : ap;
    if (__any_sync(0xffffffffu, big - kLow >= kHigh - kLow || an < 0x00100000u)) {
      if (pn == 0.0) {  // opposite sign to p, 2^-600 of the pair's scale (a normal number)
        const double mag = fmax(fabs(p), fabs(pm)) * 0x1p-600;
        pn = p < 0.0 ? mag : -mag;
      }
      c += (int)(((unsigned)__double2hiint(pn) ^ hp) >> 31);
      pm = p;
      p = pn;
      const int ex = (__double2hiint(p) >> 20) & 0x7ff, ey = (__double2hiint(pm) >> 20) & 0x7ff;
      const int emax = ex > ey ? ex : ey;
      if (emax > 1023 + 400 || emax < 1023 - 400) {
        // multiply both by 2^(1023 - emax), built from its bits
        const double sc = __longlong_as_double((long long)(2046 - emax) << 52);
        p *= sc;
        pm *= sc;
      }
      hp = (unsigned)__double2hiint(p);
    } else {
      c += (int)((hn ^ hp) >> 31);
      pm = p;
      p = pn;
      hp = hn;
    }
  }
  return c;
}

// lam[w] = eigenvalue of ascending rank ranks[w].  A warp per wanted value
// evaluates 32 shifts per round (multisection into 33 parts).  A warp's FP64
// instructions run one after another on its sub-partition's FP64 unit, 64
// clocks each whatever the number of active lanes, so the time is rounds x
// steps x FP64 operations per step of one warp, with one warp per
// sub-partition (two-warp blocks); two shifts per lane take twice as long per
// round and save two rounds in eleven.  d and e² are staged in shared memory.
constexpr int kBisThreads = 64;
__global__ void __launch_bounds__(kBisThreads)
bisect_kernel(int n, const double* __restrict__ d, const double* __restrict__ e, const int* __restrict__ ranks, int nw,
              double* __restrict__ lam) {
  __shared__ double ds[kRitzMaxN], e2s[kRitzMaxN];
  __shared__ TriBounds bs;
  if (threadIdx.x < 32) {
    const TriBounds b = tri_bounds_warp(n, d, e);
    if (threadIdx.x == 0) bs = b;
  }
  __syncthreads();
  // T and the shifts scaled by the power of two that brings ‖T‖ into [0.5, 1):
  // exact, and it bounds the growth of the minors per step
  const long long tb = __double_as_longlong(bs.tnorm);
  const int te = (int)((tb >> 52) & 0x7ff);
  const double sc = bs.tnorm > 0.0 && te > 0 ? __longlong_as_double((long long)(2045 - te) << 52) : 1.0;
  const double isc = bs.tnorm > 0.0 && te > 0 ? __longlong_as_double((long long)(te + 1) << 52) : 1.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    ds[i] = d[i] * sc;
    const double es = i + 1 < n ? e[i] * sc : 0.0;
    e2s[i] = es * es;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int w = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
  if (w >= nw) return;
  const int r = ranks[w];
  constexpr double kStep = 1.0 / 33.0;
  const double tnorm = bs.tnorm * sc;
  double lo = bs.lo * sc, hi = bs.hi * sc;
  for (int it = 0; it < 64; ++it) {
    const double width = hi - lo;
    if (width <= 0.0 || width <= fmax(DBL_EPSILON * tnorm, 2.0 * DBL_EPSILON * fmax(fabs(lo), fabs(hi)))) break;
    const int c = sturm_count(n, ds, e2s, lo + width * ((lane + 1) * kStep));
    const unsigned above = __ballot_sync(0xffffffffu, c > r);
    const int l = above ? __ffs(above) - 1 : 32;
    const double nlo = l == 0 ? lo : lo + width * (l * kStep);
    const double nhi = l == 32 ? hi : lo + width * ((l + 1) * kStep);
    lo = nlo;
    hi = nhi;
  }
  if (lane == 0) lam[w] = 0.5 * (lo + hi) * isc;
}

__device__ __forceinline__ double hash_unit(uint64_t a, uint64_t b) {
  uint64_t x = a * 0x9e3779b97f4a7c15ull + b + 0x632be59bd9b4e019ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  x ^= x >> 31;
  return (double)(x >> 11) * (2.0 / 9007199254740992.0) - 1.0;  // [-1, 1)
}

// Eigenvectors of T for the selected eigenvalues: sel[0..nsel) are indices
// into (ranks, lam), ascending (identity when sel is null).  One warp per
// cluster of selected eigenvalues with consecutive ranks closer than
// 1e-9 ‖T‖ (near-degenerate pairs).  Outside a cluster a converged vector is
// within eps ‖T‖ / gap <= 2.2e-7 of its eigenvector, and orth_step_kernel then
// restores orthonormality; LAPACK dstein clusters at 1e-3 ‖T‖ instead,
// which chains the dense bulk of a Ritz spectrum (tiny eigenvalues 1e-7
// apart) into long sequential runs.  Inside a cluster the vectors are done in
// order, each orthogonalised against the cluster's earlier ones after every
// solve (the dot products and updates spread over the lanes).  The pivoted
// LU and the triangular solves run on lane 0.  lu: per-cluster scratch of 4n
// doubles + n pivot flags.  Zt row t = eigenvector of selection t (unit
// 2-norm, largest component positive).
__global__ void invit_kernel(int n, const double* __restrict__ d, const double* __restrict__ e,
                             const int* __restrict__ ranks, const double* __restrict__ lam,
                             const int* __restrict__ sel, int nsel, double* __restrict__ Zt,
                             double* __restrict__ lu, unsigned char* __restrict__ piv) {
  const int lane = threadIdx.x & 31;
  const int t = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
  if (t >= nsel) return;
  double tnorm = 0.0;
  for (int i = lane; i < n; i += 32)
    tnorm = fmax(tnorm, fabs(d[i]) + (i > 0 ? fabs(e[i - 1]) : 0.0) + (i + 1 < n ? fabs(e[i]) : 0.0));
#pragma unroll
  for (int o = 16; o; o >>= 1) tnorm = fmax(tnorm, __shfl_xor_sync(0xffffffffu, tnorm, o));
  const double ortol = 1e-9 * tnorm;
  auto idx = [&](int w) { return sel ? sel[w] : w; };
  auto joined = [&](int w) {  // selection w continues the cluster of w - 1
    return w > 0 && ranks[idx(w)] == ranks[idx(w - 1)] + 1 && lam[idx(w)] - lam[idx(w - 1)] <= ortol;
  };
  if (joined(t)) return;  // not the first vector of its cluster (warp-uniform)
  int end = t + 1;
  while (end < nsel && joined(end)) ++end;
  double* L = lu + (size_t)t * 4 * n;  // multipliers
  double* U0 = L + n;                  // reciprocal pivots
  double* U1 = U0 + n;
  double* U2 = U1 + n;
  unsigned char* P = piv + (size_t)t * n;
  const double eps = DBL_EPSILON;
  const double tiny = eps * fmax(tnorm, DBL_MIN);
  double prev = 0.0;
  for (int w = t; w < end; ++w) {
    double x = lam[idx(w)];
    const double pertol = 10.0 * fabs(eps * x) + tiny;
    if (w > t && x - prev < pertol) x = prev + pertol;  // separate equal shifts, as dstein
    prev = x;
    double* z = Zt + (size_t)w * n;
    if (lane == 0) {
      // pivoted LU of T - x I: U has two superdiagonals; U0 keeps the
      // reciprocal of each pivot (tiny pivots replaced by ±eps‖T‖, as
      // dlagts does), so the solves below divide nothing
      double cd = d[0] - x, cs = n > 1 ? e[0] : 0.0;
      for (int i = 0; i + 1 < n; ++i) {
        const double sub = e[i], dn = d[i + 1] - x, sp = i + 2 < n ? e[i + 1] : 0.0;
        double pv;
        // one reciprocal per row (an FP64 division is a long chain of FP64
        // operations here): the multiplier is formed from the pivot's
        // reciprocal
        if (fabs(cd) >= fabs(sub)) {
          pv = cd;
          if (fabs(pv) < tiny) pv = pv < 0.0 ? -tiny : tiny;
          const double rp = 1.0 / pv;
          const double l = cd != 0.0 ? sub * rp : 0.0;
          U0[i] = rp; U1[i] = cs; U2[i] = 0.0; L[i] = l; P[i] = 0;
          cd = dn - l * cs;
          cs = sp;
        } else {
          pv = sub;
          const double rp = 1.0 / pv;
          const double l = cd * rp;
          U0[i] = fabs(pv) < tiny ? (pv < 0.0 ? -1.0 / tiny : 1.0 / tiny) : rp;
          U1[i] = dn; U2[i] = sp; L[i] = l; P[i] = 1;
          cd = cs - l * dn;
          cs = -l * sp;
        }
      }
      if (fabs(cd) < tiny) cd = cd < 0.0 ? -tiny : tiny;
      U0[n - 1] = 1.0 / cd;
    }
    for (int i = lane; i < n; i += 32) z[i] = hash_unit((uint64_t)ranks[idx(w)], (uint64_t)i);
    __syncwarp();
    // iterate until the solve grows a unit vector by 1e-3 / (eps ‖T‖) (the
    // shift is then an eigenvalue to working accuracy), then once more, at
    // most five times (LAPACK dstein's scheme)
    double mx = 1.0;
    for (int it = 0, extra = 0; it < 5 && extra < 2; ++it) {
      // scale to unit max norm, then solve (T - x I) y = z in place (lane 0)
      const double sc = mx > 0.0 ? 1.0 / mx : 1.0;
      for (int i = lane; i < n; i += 32) z[i] *= sc;
      __syncwarp();
      if (lane == 0) {
        for (int i = 0; i + 1 < n; ++i) {
          if (P[i]) { const double tmp = z[i]; z[i] = z[i + 1]; z[i + 1] = tmp; }
          z[i + 1] -= L[i] * z[i];
        }
        for (int i = n - 1; i >= 0; --i) {
          double r = z[i];
          if (i + 1 < n) r -= U1[i] * z[i + 1];
          if (i + 2 < n) r -= U2[i] * z[i + 2];
          z[i] = r * U0[i];
        }
      }
      __syncwarp();
      for (int s2 = t; s2 < w; ++s2) {  // modified Gram-Schmidt inside the cluster
        const double* q = Zt + (size_t)s2 * n;
        double dot = 0.0;
        for (int i = lane; i < n; i += 32) dot = fma(q[i], z[i], dot);
        dot = warp_sum_d(dot);
        for (int i = lane; i < n; i += 32) z[i] = fma(-dot, q[i], z[i]);
        __syncwarp();
      }
      mx = 0.0;
      for (int i = lane; i < n; i += 32) mx = fmax(mx, fabs(z[i]));
#pragma unroll
      for (int o = 16; o; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      if (extra > 0 || mx * tiny >= 1e-3) ++extra;
    }
    double nrm = 0.0, big = 0.0;
    int ib = n;
    for (int i = lane; i < n; i += 32) {
      nrm = fma(z[i], z[i], nrm);
      if (fabs(z[i]) > big) { big = fabs(z[i]); ib = i; }
    }
    nrm = warp_sum_d(nrm);
#pragma unroll
    for (int o = 16; o; o >>= 1) {  // the largest |component|, lowest index on ties
      const double bo = __shfl_xor_sync(0xffffffffu, big, o);
      const int io = __shfl_xor_sync(0xffffffffu, ib, o);
      if (bo > big || (bo == big && io < ib)) { big = bo; ib = io; }
    }
    double sc = nrm > 0.0 ? 1.0 / sqrt(nrm) : 0.0;
    if (ib < n && z[ib] < 0.0) sc = -sc;
    __syncwarp();
    for (int i = lane; i < n; i += 32) z[i] *= sc;
    __syncwarp();
  }
}

// E = Zt Ztᵀ - I over the nw rows of length n, both triangles; one warp per
// entry of the lower one.  *wide counts the entries too large for the two
// steps below: with every |E_ij| <= kOrthNear / nw, ‖E‖ <= kOrthNear, and two
// steps of E -> 3/4 E² leave 0.42 kOrthNear⁴ = 4e-17.  Vectors of an inverse
// iteration that converged are within it: eps / 1e-9 for the closest pairs.
constexpr double kOrthNear = 1e-4;
__global__ void gram_rows_kernel(int nw, int n, const double* __restrict__ Zt, double* __restrict__ E,
                                 int* __restrict__ wide) {
  const int lane = threadIdx.x & 31;
  const int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t tot = (int64_t)nw * (nw + 1) / 2;
  if (w >= tot) return;
  // w -> (i, j), j <= i
  int i = (int)((sqrtf(8.0f * (float)w + 1.0f) - 1.0f) * 0.5f);
  while ((int64_t)i * (i + 1) / 2 > w) --i;
  while ((int64_t)(i + 1) * (i + 2) / 2 <= w) ++i;
  const int j = (int)(w - (int64_t)i * (i + 1) / 2);
  const double* a = Zt + (size_t)i * n;
  const double* b = Zt + (size_t)j * n;
  double s = 0.0;
  for (int c = lane; c < n; c += 32) s = fma(a[c], b[c], s);
  s = warp_sum_d(s);
  if (lane == 0) {
    if (i == j) s -= 1.0;
    E[(size_t)i * nw + j] = s;
    E[(size_t)j * nw + i] = s;
    if (wide && !(fabs(s) * nw <= kOrthNear)) atomicAdd(wide, 1);
  }
}

// out = Zt - E Zt / 2 (rows): one step of Björck and Bowie's iteration for
// the closest orthonormal matrix (SIAM J. Numer. Anal. 8 (1971) 358), whose
// error E becomes 3/4 E².  A warp holds 32 columns of kOrthRows rows, so a
// load of Zt serves kOrthRows FMAs.  Nothing is done when *wide is set.
constexpr int kOrthRows = 4;
__global__ void __launch_bounds__(128)
orth_step_kernel(int nw, int n, const double* __restrict__ E, const double* __restrict__ Zt,
                 double* __restrict__ out, const int* __restrict__ wide) {
  if (*wide) return;
  const int c = (blockIdx.x * 4 + (threadIdx.x >> 5)) * 32 + (threadIdx.x & 31);
  if (c >= n) return;
  const int i0 = blockIdx.y * kOrthRows;
  double acc[kOrthRows];
  const double* er[kOrthRows];
#pragma unroll
  for (int r = 0; r < kOrthRows; ++r) {
    acc[r] = 0.0;
    er[r] = E + (size_t)min(i0 + r, nw - 1) * nw;
  }
#pragma unroll 4
  for (int q = 0; q < nw; ++q) {
    const double z = Zt[(size_t)q * n + c];
#pragma unroll
    for (int r = 0; r < kOrthRows; ++r) acc[r] = fma(er[r][q], z, acc[r]);
  }
#pragma unroll
  for (int r = 0; r < kOrthRows; ++r)
    if (i0 + r < nw) out[(size_t)(i0 + r) * n + c] = fma(-0.5, acc[r], Zt[(size_t)(i0 + r) * n + c]);
}

// For vectors too far from orthonormal for the iteration (*wide set; nothing
// is done otherwise): G = E + I = L Lᵀ in place (lower), then Zt <- L⁻¹ Zt
// (rows orthonormal).  One CTA; a non-positive pivot leaves Zt as it is.
__global__ void __launch_bounds__(1024)
orth_kernel(int nw, int n, double* __restrict__ G, double* __restrict__ Zt, const int* __restrict__ wide) {
  if (!*wide) return;
  __shared__ int bad;
  if (threadIdx.x == 0) bad = 0;
  for (int i = threadIdx.x; i < nw; i += blockDim.x) G[(size_t)i * nw + i] += 1.0;
  __syncthreads();
  for (int j = 0; j < nw; ++j) {
    if (threadIdx.x == 0) {
      const double piv = G[(size_t)j * nw + j];
      if (!(piv > 0.0)) bad = 1;
      else G[(size_t)j * nw + j] = sqrt(piv);
    }
    __syncthreads();
    if (bad) return;
    const double ljj = G[(size_t)j * nw + j];
    for (int i = j + 1 + threadIdx.x; i < nw; i += blockDim.x) G[(size_t)i * nw + j] /= ljj;
    __syncthreads();
    // trailing update of the lower triangle: G[i][k] -= L[i][j] L[k][j],
    // j < k <= i; warp per row, lanes over k
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    for (int i = j + 1 + warp; i < nw; i += nwarps) {
      const double lij = G[(size_t)i * nw + j];
      for (int k = j + 1 + lane; k <= i; k += 32) G[(size_t)i * nw + k] -= lij * G[(size_t)k * nw + j];
    }
    __syncthreads();
  }
  for (int c = threadIdx.x; c < n; c += blockDim.x) {  // forward substitution, one column per thread
    for (int i = 0; i < nw; ++i) {
      double y = Zt[(size_t)i * n + c];
      for (int q = 0; q < i; ++q) y -= G[(size_t)i * nw + q] * Zt[(size_t)q * n + c];
      Zt[(size_t)i * n + c] = y / G[(size_t)i * nw + i];
    }
  }
}

// Reflectors are applied kWy at a time: H_j H_{j+1} ... H_{j+kWy-1} =
// I - W T Wᵀ with the reflectors as the columns of W and T upper triangular
// (the compact WY form; Schreiber and Van Loan, SIAM J. Sci. Stat. Comput. 10
// (1989) 53): T_cc = τ_c, T_{0..c-1,c} = -τ_c T_{0..c-1,0..c-1} W_{0..c-1}ᵀ w_c.
// One warp per block of reflectors; row j of V holds reflector j from j + 1 on.
constexpr int kWy = 8;
__global__ void __launch_bounds__(32)
wy_kernel(int n, const double* __restrict__ V, const double* __restrict__ tau, double* __restrict__ T) {
  const int j0 = blockIdx.x * kWy, nr = n - 2, lane = threadIdx.x;
  __shared__ double g[kWy][kWy], t[kWy][kWy];
  double acc[kWy * kWy / 2 + kWy];  // packed pairs a < c
#pragma unroll
  for (int x = 0; x < kWy * (kWy - 1) / 2; ++x) acc[x] = 0.0;
  for (int k = j0 + 1 + lane; k < n; k += 32) {
    double v[kWy];
#pragma unroll
    for (int c = 0; c < kWy; ++c) v[c] = j0 + c < nr && k > j0 + c ? V[(int64_t)(j0 + c) * n + k] : 0.0;
    int x = 0;
#pragma unroll
    for (int a = 0; a < kWy; ++a)
#pragma unroll
      for (int c = a + 1; c < kWy; ++c) acc[x] = fma(v[a], v[c], acc[x]), ++x;
  }
  int x = 0;
#pragma unroll
  for (int a = 0; a < kWy; ++a)
#pragma unroll
    for (int c = a + 1; c < kWy; ++c) {
      const double s = warp_sum_d(acc[x++]);
      if (lane == 0) g[a][c] = s;
    }
  for (int q = lane; q < kWy * kWy; q += 32) t[q / kWy][q % kWy] = 0.0;
  __syncwarp();
  for (int c = 0; c < kWy; ++c) {
    const double tc = j0 + c < nr ? tau[j0 + c] : 0.0;
    double s = 0.0;
    if (lane < c)
      for (int q = lane; q < c; ++q) s = fma(t[lane][q], g[q][c], s);
    __syncwarp();
    if (lane < c) t[lane][c] = -tc * s;
    if (lane == c) t[c][c] = tc;
    __syncwarp();
  }
  for (int q = lane; q < kWy * kWy; q += 32) T[(int64_t)blockIdx.x * kWy * kWy + q] = t[q / kWy][q % kWy];
}

// Zt rows <- Q Zt rows, Q = H_0 H_1 ... H_{n-3}; one CTA per vector, its
// elements in registers.  A block of reflectors costs eight dot products side
// by side (one transpose butterfly), eight FMAs for T and the update, instead
// of eight dependent dot products of five additions each by one warp: 586 ->
// 300 us (and 22 us for T) for 288 vectors at n = 336.
constexpr int kBackThreads = 128;
__global__ void __launch_bounds__(kBackThreads)
backtr_kernel(int n, const double* __restrict__ V, const double* __restrict__ T, double* __restrict__ Zt) {
  constexpr int kPer = (kRitzMaxN + kBackThreads - 1) / kBackThreads, kWarps = kBackThreads / 32;
  __shared__ double ys[2][kWarps][kWy];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nr = n - 2;
  double* g = Zt + (size_t)blockIdx.x * n;
  double z[kPer];
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    const int k = (int)threadIdx.x + q * kBackThreads;
    z[q] = k < n ? g[k] : 0.0;
  }
  for (int b = (nr + kWy - 1) / kWy - 1; b >= 0; --b) {
    const int j0 = b * kWy;
    const double* Tb = T + (int64_t)b * kWy * kWy;
    double v[kPer][kWy], y[kWy];
#pragma unroll
    for (int c = 0; c < kWy; ++c) y[c] = 0.0;
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
      const int k = (int)threadIdx.x + q * kBackThreads;
#pragma unroll
      for (int c = 0; c < kWy; ++c)
        v[q][c] = k < n && j0 + c < nr && k > j0 + c ? V[(int64_t)(j0 + c) * n + k] : 0.0;
    }
    // lane c's row of T, in flight beside the reflectors
    double tr[kWy];
#pragma unroll
    for (int c = 0; c < kWy; ++c) tr[c] = Tb[(lane % kWy) * kWy + c];
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
      if (warp * 32 + q * kBackThreads < n && warp * 32 + q * kBackThreads + 31 > j0) {
#pragma unroll
        for (int c = 0; c < kWy; ++c) y[c] = fma(v[q][c], z[q], y[c]);
      }
    }
    warp_colsum<double, kWy>(y, lane);
    if (lane % (32 / kWy) == 0) ys[b & 1][warp][lane / (32 / kWy)] = y[0];
    __syncthreads();
    // lane: y_c of c = lane mod 8 summed over the warps, then (T y)_c
    double yc = 0.0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) yc += ys[b & 1][w][lane % kWy];
    double t = 0.0;
#pragma unroll
    for (int c = 0; c < kWy; ++c) t = fma(tr[c], __shfl_sync(0xffffffffu, yc, c), t);
#pragma unroll
    for (int c = 0; c < kWy; ++c) {
      const double tc = -__shfl_sync(0xffffffffu, t, c);
#pragma unroll
      for (int q = 0; q < kPer; ++q)
        if (warp * 32 + q * kBackThreads < n && warp * 32 + q * kBackThreads + 31 > j0) z[q] = fma(tc, v[q][c], z[q]);
    }
  }
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    const int k = (int)threadIdx.x + q * kBackThreads;
    if (k < n) g[k] = z[q];
  }
}

__global__ void ranks_kernel(int n, int p, int q, int* __restrict__ ranks) {
  // the q smallest and p largest ranks, ascending (all n when they overlap)
  const int nw = p + q >= n ? n : p + q;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nw; t += gridDim.x * blockDim.x)
    ranks[t] = (p + q >= n || t < q) ? t : n - p + (t - q);
}

// cluster size the reduction kernel launches with (0: not yet chosen; every
// thread that chooses finds the same value)
std::atomic<int> g_cluster_cs{0};

template <int CS>
int launch_tridiag_cs(int n, const double* A, int64_t lda, double* d, double* e, double* tau, double* V,
                      cudaStream_t s, bool probe_only) {
  const size_t smem = tridiag_smem(n, CS);
  if (smem > 227 * 1024) return SG_ERR_ARG;
  // the cap is set to the largest size any call needs, never to this call's:
  // calls on other host threads set the same value, so none can lower the
  // cap between another thread's set and its launch
  if (cudaFuncSetAttribute(tridiag_kernel<CS>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) !=
      cudaSuccess)
    return SG_ERR_CUDA;
  if (CS > 8 && cudaFuncSetAttribute(tridiag_kernel<CS>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
                    cudaSuccess)
    return SG_ERR_CUDA;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(CS, 1, 1);
  cfg.blockDim = dim3(kTriThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = CS;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (probe_only) {
    int nc = 0;
    if (cudaOccupancyMaxActiveClusters(&nc, tridiag_kernel<CS>, &cfg) != cudaSuccess) {
      cudaGetLastError();
      return SG_ERR_CUDA;
    }
    return nc > 0 ? SG_OK : SG_ERR_CAP;
  }
  if (cudaLaunchKernelEx(&cfg, tridiag_kernel<CS>, n, A, lda, d, e, tau, V) != cudaSuccess) return SG_ERR_CUDA;
  return SG_OK;
}

int launch_tridiag_any(int cs, int n, const double* A, int64_t lda, double* d, double* e, double* tau, double* V,
                       cudaStream_t s, bool probe) {
  switch (cs) {
    case 16: return launch_tridiag_cs<16>(n, A, lda, d, e, tau, V, s, probe);
    case 8: return launch_tridiag_cs<8>(n, A, lda, d, e, tau, V, s, probe);
    case 4: return launch_tridiag_cs<4>(n, A, lda, d, e, tau, V, s, probe);
    case 2: return launch_tridiag_cs<2>(n, A, lda, d, e, tau, V, s, probe);
    case 1: return launch_tridiag_cs<1>(n, A, lda, d, e, tau, V, s, probe);
    default: return SG_ERR_ARG;
  }
}

}  // namespace

// The largest cluster size (16, 8, 4, 2, 1) whose CTAs hold the n-row
// matrix in shared memory and that this device can launch.
int ritz_cluster_size(int n) {
  for (int cs = kMaxCluster; cs >= 1; cs >>= 1) {
    if (tridiag_smem(n, cs) > 227 * 1024) break;  // smaller clusters hold more rows each
    if (launch_tridiag_any(cs, n, nullptr, 0, nullptr, nullptr, nullptr, nullptr, nullptr, true) == SG_OK)
      return cs;
  }
  return 0;
}

RitzLayout ritz_layout(char* base, int n, int nw) {
  RitzLayout L{};
  int64_t o = 0;
  auto take = [&](int64_t b) { const int64_t r = o; o += (b + 255) / 256 * 256; return r; };
  const int64_t od = take(8 * (int64_t)n), oe = take(8 * (int64_t)n), ot = take(8 * (int64_t)n),
                oV = take(8 * (int64_t)n * n), orr = take(4 * (int64_t)n), ol = take(8 * (int64_t)n),
                oz = take(8 * (int64_t)n * nw), olu = take(32 * (int64_t)n * nw), op = take((int64_t)n * nw),
                oG = take(8 * (int64_t)nw * nw), oT = take(8 * kWy * ((int64_t)n + kWy)), ow = take(4);
  if (base) {
    L.d = (double*)(base + od);
    L.e = (double*)(base + oe);
    L.tau = (double*)(base + ot);
    L.V = (double*)(base + oV);
    L.ranks = (int*)(base + orr);
    L.lam = (double*)(base + ol);
    L.Zt = (double*)(base + oz);
    L.lu = (double*)(base + olu);
    L.piv = (unsigned char*)(base + op);
    L.G = (double*)(base + oG);
    L.T = (double*)(base + oT);
    L.wide = (int*)(base + ow);
  }
  L.bytes = o;
  return L;
}

// Eigenvalues of the symmetric n x n matrix A (row-major, lda): the q
// smallest and p largest (all n when p + q >= n), ascending into L.lam, their
// ranks into L.ranks, the count into *nw.  Leaves the reduction (L.d, L.e,
// L.tau, L.V) for ritz_vectors.
int ritz_values(int n, const double* A, int64_t lda, int p, int q, const RitzLayout& L, int* nw, cudaStream_t s) {
  if (n < 1 || p < 0 || q < 0 || p + q < 1) return SG_ERR_ARG;
  const int cnt = p + q >= n ? n : p + q;
  *nw = cnt;
  int cs = g_cluster_cs.load();
  if (cs == 0 || tridiag_smem(n, cs) > 227 * 1024) {
    cs = ritz_cluster_size(n);
    if (cs == 0) return SG_ERR_CAP;
    g_cluster_cs.store(cs);
  }
  int err = launch_tridiag_any(cs, n, A, lda, L.d, L.e, L.tau, L.V, s, false);
  if (err) return err;
  ranks_kernel<<<grid_for(cnt, 256), 256, 0, s>>>(n, p, q, L.ranks);
  SG_CHECK_LAUNCH();
  bisect_kernel<<<grid_for((int64_t)cnt * 32, kBisThreads), kBisThreads, 0, s>>>(n, L.d, L.e, L.ranks, cnt, L.lam);
  SG_CHECK_LAUNCH();
  return SG_OK;
}

// The nw rows of Z (length n) to the closest orthonormal set, by two steps of
// the iteration, or by Cholesky-QR where they are too far off.  Z2: as large
// as Z; G: nw x nw.
static int orth_rows(int nw, int n, double* Z, double* Z2, double* G, int* wide, cudaStream_t s) {
  if (nw < 2) return SG_OK;
  const int64_t pairs = (int64_t)nw * (nw + 1) / 2;
  const dim3 grid((n + 127) / 128, (nw + kOrthRows - 1) / kOrthRows);
  if (cudaMemsetAsync(wide, 0, sizeof(int), s) != cudaSuccess) return SG_ERR_CUDA;
  gram_rows_kernel<<<grid_for(pairs * 32, 256), 256, 0, s>>>(nw, n, Z, G, wide);
  SG_CHECK_LAUNCH();
  orth_kernel<<<1, 1024, 0, s>>>(nw, n, G, Z, wide);
  SG_CHECK_LAUNCH();
  orth_step_kernel<<<grid, 128, 0, s>>>(nw, n, G, Z, Z2, wide);
  SG_CHECK_LAUNCH();
  gram_rows_kernel<<<grid_for(pairs * 32, 256), 256, 0, s>>>(nw, n, Z2, G, nullptr);
  SG_CHECK_LAUNCH();
  orth_step_kernel<<<grid, 128, 0, s>>>(nw, n, G, Z2, Z, wide);
  SG_CHECK_LAUNCH();
  return SG_OK;
}

// Eigenvectors of the nsel selected eigenvalues (sel: ascending indices into
// L.lam, device; null = all *nw of them) into the first nsel rows of L.Zt.
int ritz_vectors(int n, const RitzLayout& L, const int* sel, int nsel, cudaStream_t s) {
  if (nsel < 1) return SG_OK;
  invit_kernel<<<grid_for((int64_t)nsel * 32, 128), 128, 0, s>>>(n, L.d, L.e, L.ranks, L.lam, sel, nsel, L.Zt, L.lu,
                                                                  L.piv);
  SG_CHECK_LAUNCH();
  if (n > 2) {
    wy_kernel<<<(n - 2 + kWy - 1) / kWy, 32, 0, s>>>(n, L.V, L.tau, L.T);
    SG_CHECK_LAUNCH();
    backtr_kernel<<<nsel, kBackThreads, 0, s>>>(n, L.V, L.T, L.Zt);
    SG_CHECK_LAUNCH();
  }
  // two steps through the inverse iteration's scratch and back
  return orth_rows(nsel, n, L.Zt, L.lu, L.G, L.wide, s);
}

}  // namespace sg

using namespace sg;

extern "C" int64_t sg_sym_eig_work_bytes(int n, int p, int q) {
  if (n < 1 || p < 0 || q < 0 || p + q < 1 || n > kRitzMaxN) return -1;
  const int cnt = p + q >= n ? n : p + q;
  return ritz_layout(nullptr, n, cnt).bytes;
}

extern "C" int sg_sym_eig(int n, const double* A, int64_t lda, int p, int q, double* evals, double* evecs,
                          void* work, int64_t work_bytes, void* stream) {
  if (n < 1 || n > kRitzMaxN || lda < n || !A || !evals || !evecs || !work || p < 0 || q < 0 || p + q < 1)
    return SG_ERR_ARG;
  if (((uintptr_t)work & 255u) != 0) return SG_ERR_ARG;
  const int cnt = p + q >= n ? n : p + q;
  RitzLayout L = ritz_layout((char*)work, n, cnt);
  if (work_bytes < L.bytes) return SG_ERR_CAP;
  cudaStream_t s = as_stream(stream);
  int nw = 0;
  int err = ritz_values(n, A, lda, p, q, L, &nw, s);
  if (!err) err = ritz_vectors(n, L, nullptr, nw, s);
  if (err) return err;
  if (cudaMemcpyAsync(evals, L.lam, sizeof(double) * nw, cudaMemcpyDeviceToDevice, s) != cudaSuccess ||
      cudaMemcpyAsync(evecs, L.Zt, sizeof(double) * nw * (size_t)n, cudaMemcpyDeviceToDevice, s) != cudaSuccess)
    return SG_ERR_CUDA;
  return SG_OK;
}

extern "C" int64_t sg_orth_rows_work_bytes(int nw, int n) {
  if (nw < 1 || n < nw || n > kRitzMaxN) return -1;
  return 8 * ((int64_t)nw * n + (int64_t)nw * nw) + 8;
}

extern "C" int sg_orth_rows(int nw, int n, double* Z, void* work, int64_t work_bytes, void* stream) {
  if (nw < 1 || n < nw || n > kRitzMaxN || !Z || !work || ((uintptr_t)work & 7u) != 0) return SG_ERR_ARG;
  if (work_bytes < sg_orth_rows_work_bytes(nw, n)) return SG_ERR_CAP;
  double* Z2 = static_cast<double*>(work);
  double* G = Z2 + (int64_t)nw * n;
  return orth_rows(nw, n, Z, Z2, G, reinterpret_cast<int*>(G + (int64_t)nw * nw), as_stream(stream));
}
