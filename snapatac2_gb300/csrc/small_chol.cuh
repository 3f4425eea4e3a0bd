// Cholesky factor and inverse factor of a small symmetric FP64 matrix by four
// warps of one CTA (the Gram matrices of the block eigensolver, up to 32 x 32).
#pragma once
#include "common.cuh"

namespace sg {

constexpr int kCholThreads = 128;

// barrier of the first kCholThreads threads only (the CTA may have more)
__device__ __forceinline__ void chol_barrier() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

// G = RᵀR, eliminated from the left on [G | I]: after step k row k of the left
// half is row k of R and row k of the right half is column k of R⁻¹.  Called
// by the first kCholThreads threads of the CTA, which all return the same
// answer: false when a pivot is not above tol x its diagonal (or not positive,
// or NaN); that pivot is then taken as 1 and the elimination goes on.
//
// GB300 runs FP64 at about half a lane per clock on each of the SM's four
// sub-partitions, whatever the number of active lanes, and one warp on one of
// them had the whole chain: dot products of up to k terms one after another
// for each pivot and each back-substituted entry (11 us for an 8 x 8 matrix).
// Here a step is one reciprocal square root, one product (row k, written to r)
// and one FMA per remaining element, spread over four warps: a chain of three
// operations per step instead of 2k, and the terms of each element are still
// subtracted in the order 0, 1, ..., k - 1.
template <int P>  // row length of each half: a power of two, B <= P <= 32
struct CholSmem {
  double a[P][2 * P];  // [G | I], updated in place
  double r[P][2 * P];  // row k: R[k][k..B-1] at k.., R⁻¹[0..k][k] at P..P+k
};

template <int P>
__device__ bool chol_inv(int B, CholSmem<P>& m, double tol) {
  constexpr int kRows = kCholThreads / (2 * P) > 0 ? kCholThreads / (2 * P) : 1;  // rows per pass
  static_assert(kCholThreads % (2 * P) == 0, "a pass covers whole rows");
  const int c = threadIdx.x % (2 * P), i0 = threadIdx.x / (2 * P);
  // the original diagonal, for the pivot test, read before any update
  __shared__ double dg[P];
  if (threadIdx.x < P) dg[threadIdx.x] = (int)threadIdx.x < B ? m.a[threadIdx.x][threadIdx.x] : 1.0;
  chol_barrier();
  bool ok = true;
  for (int k = 0; k < B; ++k) {
    double s = m.a[k][k];
    const double gkk = dg[k];
    if (!(s > tol * (gkk > 0.0 ? gkk : 1.0)) || !(s > 0.0)) {
      ok = false;
      s = 1.0;
    }
    // columns with an entry in row k: k .. B-1 on the left, 0 .. k on the right
    const bool live = c < P ? (c >= k && c < B) : c - P <= k;
    if (i0 == 0 && live) {
      const double rs = rsqrt(s);
      m.r[k][c] = (c == k ? s : m.a[k][c]) * rs;
    }
    chol_barrier();
    for (int i = k + 1 + i0; i < B; i += kRows)
      if (live && (c >= P || c >= i)) m.a[i][c] = fma(-m.r[k][i], m.r[k][c], m.a[i][c]);
    chol_barrier();
  }
  return ok;
}

}  // namespace sg
