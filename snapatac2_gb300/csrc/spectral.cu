// Matrix-free cosine spectral operator: feature selection, deterministic CSR
// transpose, IDF weights, row normalisation, degree, and the two CSR SpMM
// kernels of the Gram product.
//
// Reference arithmetic (snapatac2-python/src/embedding.rs):
//   idf        269-286   w_j = ln(n / c_j), c_j = nnz of column j (0 -> 1,
//                        n -> n-1; all counts equal -> w = 1)
//   normalize  315-326   Xn = diag(1/||(XW)_i||) X W
//   degree     139-152   colsum = 1ᵀXn, d = Xn colsum, D⁻¹ = 1/(d - 1)
//   eigen      155-171   operator v -> X̂ (X̂ᵀ v) - D⁻¹ v, X̂ = diag(sqrt(D⁻¹)) Xn
// With a_i = sqrt(D⁻¹_i)/||(XW)_i|| the operator is
//   A v = a ⊙ (X (w² ⊙ (Xᵀ (a ⊙ v)))) - D⁻¹ ⊙ v
// so X is kept as an index-only pattern (or with its integer counts) and the
// scalings are folded into the SpMM prologue/epilogue.
#include <algorithm>

#include "common.cuh"
#include "internal.h"

namespace sg {
namespace {

// ---------------------------------------------------------------------------
// column selection: keep entries whose column maps to >= 0, renumbered
// ---------------------------------------------------------------------------
__global__ void select_count(int64_t n, const int64_t* __restrict__ ptr, const int32_t* __restrict__ idx,
                             const int32_t* __restrict__ colmap, int64_t* __restrict__ cnt) {
  const int lane = threadIdx.x & 31;
  const int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t r = w; r < n; r += nw) {
    int64_t c = 0;
    for (int64_t e = ptr[r] + lane; e < ptr[r + 1]; e += 32) c += colmap[idx[e]] >= 0;
    for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if (lane == 0) cnt[r + 1] = c;
  }
}

__global__ void select_fill(int64_t n, const int64_t* __restrict__ ptr, const int32_t* __restrict__ idx,
                            const float* __restrict__ val, const int32_t* __restrict__ colmap,
                            const int64_t* __restrict__ optr, int32_t* __restrict__ oidx,
                            float* __restrict__ oval) {
  const int lane = threadIdx.x & 31;
  const int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t r = w; r < n; r += nw) {
    int64_t o = optr[r];
    const int64_t b = ptr[r], e = ptr[r + 1];
    for (int64_t k0 = b; k0 < e; k0 += 32) {
      const int64_t k = k0 + lane;
      int nc = -1;
      if (k < e) nc = colmap[idx[k]];
      const unsigned keep = __ballot_sync(0xffffffffu, nc >= 0);
      if (nc >= 0) {
        const int64_t p = o + __popc(keep & lanemask_lt());
        oidx[p] = nc;
        if (oval) oval[p] = val[k];
      }
      o += __popc(keep);
    }
  }
}

// ---------------------------------------------------------------------------
// deterministic transpose (CSR -> CSC) with rows ascending inside each column
//
// Columns are cut into panels of kTrPanel columns and rows into nblk blocks;
// a CTA works on one (row block, panel).  seg[p][r] is the offset (from the
// row start) of row r's first entry in panel p (rows are sorted, so a row's
// entries of one panel are contiguous).
//   count  : shared-memory histogram of the panel's columns, written to
//            cnt[b][col] (coalesced);
//   offsets: cnt[b][col] <- sum over earlier row blocks (column-wise scan);
//   fill   : kTrRows rows at a time, in any order within them: every entry
//            sets its row's bit in its column's mask, and after a barrier its
//            place is the column's cursor plus the number of lower bits set;
//            then the cursors move and the masks are cleared.  Rows ascend in
//            every column whatever order the threads run in, so the result is
//            identical run to run.
// What bounds it: about 34 entries per (row, panel) at 500,000 columns, so the
// work is short segments of dependent loads and shared-memory atomics.  The
// form before took the rows of a block one at a time with a barrier after
// each (136 of 512 threads busy: 9.9 ms of fill, 4.3 of count) and 304 row
// blocks (2.6 ms for the offsets).  Half a warp per row segment, three barriers
// per 128 rows and some 20 row blocks took 5.0 ms (fill), 1.2 (count) and 1.1
// (segments, before 2.1) at 100,000 x 500,000 and 4.1e8 nonzeros with 2,048
// columns per panel and 512 threads; 4,096 columns and 1,024 threads take 4.6,
// 0.88 and 0.98 (8,192 columns and one CTA per SM 5.0, 0.88, 0.83; 256 rows per
// step 5.1 and more; a whole warp per segment 5.0 and more).  The fill is
// bound by its scattered 4-byte stores (L1 and L2 at two thirds); gathering a
// column's rows in shared memory until a 32-byte sector is full took 12.5 ms
// (the columns' unequal counts leave most lanes of a warp idle).  The partly
// written sectors of all resident CTAs (two per SM) are 40 MB of the 129 MB of
// L2.
// ---------------------------------------------------------------------------
constexpr int kTrLog = 12;
constexpr int kTrPanel = 1 << kTrLog;
constexpr int kTrRows = 128;             // rows per step of the fill: four mask words per column
constexpr int kTrThreads = 1024;
constexpr int kTrHalf = 16;              // lanes per row segment
constexpr int kTrSlots = kTrThreads / kTrHalf;  // segments at a time

__global__ void seg_kernel(int64_t n, const int64_t* __restrict__ ptr, const int32_t* __restrict__ idx, int P,
                           int64_t m, int32_t* __restrict__ seg, int* status) {
  const int lane = threadIdx.x & 31;
  const int64_t gw = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t r = gw; r < n; r += nw) {
    const int64_t s = ptr[r], e = ptr[r + 1];
    int last = -1;  // column before this chunk
    bool bad = false;
    for (int64_t k0 = s; k0 < e; k0 += 64) {
      const int64_t k1 = k0 + lane, k2 = k1 + 32;
      const int c1 = k1 < e ? __ldg(idx + k1) : 0x7fffffff, c2 = k2 < e ? __ldg(idx + k2) : 0x7fffffff;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int64_t k = h ? k2 : k1;
        const int c = h ? c2 : c1;
        int prev = __shfl_up_sync(0xffffffffu, c, 1);
        if (lane == 0) prev = last;
        last = __shfl_sync(0xffffffffu, c, 31);
        if (k < e) {
          if (c < 0 || c >= m || prev >= c) {  // need sorted, unique, in range
            bad = true;
          } else {
            const int pc = c >> kTrLog;
            for (int p = (prev < 0 ? -1 : prev >> kTrLog) + 1; p <= pc; ++p) seg[(int64_t)p * n + r] = (int32_t)(k - s);
          }
        }
      }
    }
    if (bad) report_error(status, nullptr, SG_ERR_ARG, 0);
    if (__any_sync(0xffffffffu, bad)) continue;  // seg is not read once the status is set
    const int64_t tail = e > s ? (int64_t)(__ldg(idx + e - 1) >> kTrLog) + 1 : 0;
    for (int64_t p = tail + lane; p <= P; p += 32) seg[p * n + r] = (int32_t)(e - s);
  }
}

__global__ void __launch_bounds__(kTrThreads)
tr_count(int64_t n, int64_t m, const int64_t* __restrict__ ptr, const int32_t* __restrict__ idx,
         const int32_t* __restrict__ seg, int p0, int nblk, int32_t* __restrict__ cnt, const int* status) {
  __shared__ int32_t c_s[kTrPanel];
  if (*status) return;  // invalid column indices: seg is not trustworthy
  const int b = blockIdx.x, p = p0 + blockIdx.y;
  const int64_t r0 = n * b / nblk, r1 = n * (b + 1) / nblk;
  const int64_t col0 = (int64_t)p << kTrLog;
  const int width = (int)min((int64_t)kTrPanel, m - col0);
  for (int j = threadIdx.x; j < width; j += kTrThreads) c_s[j] = 0;
  __syncthreads();
  const int32_t* lo = seg + (int64_t)p * n;
  const int32_t* hi = lo + n;
  const int l = threadIdx.x % kTrHalf;
  int64_t r = r0 + threadIdx.x / kTrHalf;
  int64_t s = 0, e = 0;
  if (r < r1) {
    const int64_t base = __ldg(ptr + r);
    s = base + __ldg(lo + r);
    e = base + __ldg(hi + r);
  }
  while (r < r1) {
    const int64_t rn = r + kTrSlots;
    int64_t sn = 0, en = 0;
    if (rn < r1) {  // the next segment's bounds, in flight during this one
      const int64_t base = __ldg(ptr + rn);
      sn = base + __ldg(lo + rn);
      en = base + __ldg(hi + rn);
    }
    for (int64_t k = s + l; k < e; k += kTrHalf) atomicAdd(&c_s[__ldg(idx + k) - (int)col0], 1);
    r = rn;
    s = sn;
    e = en;
  }
  __syncthreads();
  int32_t* out = cnt + (int64_t)b * m + col0;
  for (int j = threadIdx.x; j < width; j += kTrThreads) out[j] = c_s[j];
}

// colptr[j+1] = total count of column j
__global__ void tr_total(int64_t m, int nblk, const int32_t* __restrict__ cnt, int64_t* __restrict__ colptr) {
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < m; j += (int64_t)gridDim.x * blockDim.x) {
    int64_t t = 0;
#pragma unroll 8
    for (int b = 0; b < nblk; ++b) t += cnt[(int64_t)b * m + j];
    colptr[j + 1] = t;
    if (j == 0) colptr[0] = 0;
  }
}

// cnt[b][j] <- sum_{b' < b} cnt[b'][j]  (row block b's offset inside column j)
__global__ void tr_offsets(int64_t m, int nblk, int32_t* __restrict__ cnt) {
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < m; j += (int64_t)gridDim.x * blockDim.x) {
    int32_t run = 0;
    for (int b0 = 0; b0 < nblk; b0 += 8) {  // eight loads in flight
      int32_t c[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) c[i] = b0 + i < nblk ? cnt[(int64_t)(b0 + i) * m + j] : 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (b0 + i < nblk) cnt[(int64_t)(b0 + i) * m + j] = run;
        run += c[i];
      }
    }
  }
}

__global__ void __launch_bounds__(kTrThreads, 2)
tr_fill(int64_t n, int64_t m, const int64_t* __restrict__ ptr, const int32_t* __restrict__ idx,
        const float* __restrict__ val, const int32_t* __restrict__ seg, int p0, int nblk,
        const int32_t* __restrict__ cnt, const int64_t* __restrict__ colptr, int32_t* __restrict__ rowidx, float* __restrict__ cval,
        const int* status) {
  constexpr int W = kTrRows / 32;               // mask words per column
  constexpr int R = kTrRows / kTrSlots;         // rows per half warp and step
  extern __shared__ __align__(16) unsigned char tr_smem[];
  int64_t* cur = reinterpret_cast<int64_t*>(tr_smem);                 // [kTrPanel] next place of the column
  uint32_t(*mask)[kTrPanel] = reinterpret_cast<uint32_t(*)[kTrPanel]>(cur + kTrPanel);  // [W][kTrPanel]
  if (*status) return;
  const int b = blockIdx.x, p = p0 + blockIdx.y;
  const int64_t r0 = n * b / nblk, r1 = n * (b + 1) / nblk;
  const int64_t col0 = (int64_t)p << kTrLog;
  const int width = (int)min((int64_t)kTrPanel, m - col0);
  const int32_t* in = cnt + (int64_t)b * m + col0;
  for (int j = threadIdx.x; j < width; j += kTrThreads) {
    cur[j] = colptr[col0 + j] + in[j];
#pragma unroll
    for (int w = 0; w < W; ++w) mask[w][j] = 0;
  }
  __syncthreads();
  const int32_t* lo = seg + (int64_t)p * n;
  const int32_t* hi = lo + n;
  const int l = threadIdx.x % kTrHalf, slot = threadIdx.x / kTrHalf;
  auto place = [&](int j, int w, uint32_t bit) -> int {  // rows of this step below the entry's in its column
    int below = 0;
#pragma unroll
    for (int v = 0; v < W; ++v) below += v <= w ? __popc(v < w ? mask[v][j] : mask[v][j] & (bit - 1u)) : 0;
    return below;
  };
  for (int64_t q0 = r0; q0 < r1; q0 += kTrRows) {
    int64_t s[R], e[R];
    int c[R];  // the first piece of each segment stays in registers
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int64_t r = q0 + i * kTrSlots + slot;
      s[i] = e[i] = 0;
      if (r < r1) {
        const int64_t base = __ldg(ptr + r);
        s[i] = base + __ldg(lo + r);
        e[i] = base + __ldg(hi + r);
      }
    }
#pragma unroll
    for (int i = 0; i < R; ++i) c[i] = s[i] + l < e[i] ? __ldg(idx + s[i] + l) - (int)col0 : -1;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int t = i * kTrSlots + slot;
      const uint32_t bit = 1u << (t & 31);
      if (c[i] >= 0) atomicOr(&mask[t >> 5][c[i]], bit);
      for (int64_t k = s[i] + l + kTrHalf; k < e[i]; k += kTrHalf)
        atomicOr(&mask[t >> 5][__ldg(idx + k) - (int)col0], bit);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int t = i * kTrSlots + slot;
      const uint32_t bit = 1u << (t & 31);
      const int32_t row = (int32_t)(q0 + t);
      if (c[i] >= 0) {
        const int64_t dst = cur[c[i]] + place(c[i], t >> 5, bit);
        rowidx[dst] = row;
        if (cval) cval[dst] = val[s[i] + l];
      }
      for (int64_t k = s[i] + l + kTrHalf; k < e[i]; k += kTrHalf) {
        const int j = __ldg(idx + k) - (int)col0;
        const int64_t dst = cur[j] + place(j, t >> 5, bit);
        rowidx[dst] = row;
        if (cval) cval[dst] = val[k];
      }
    }
    __syncthreads();
    for (int j = threadIdx.x; j < width; j += kTrThreads) {  // move the cursors past these rows
      int t = 0;
#pragma unroll
      for (int w = 0; w < W; ++w) t += __popc(mask[w][j]);
      if (t) {
        cur[j] += t;
#pragma unroll
        for (int w = 0; w < W; ++w) mask[w][j] = 0;
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// IDF weights, row norms, degree (FP64, as the reference)
// ---------------------------------------------------------------------------
__global__ void colcount_minmax(int64_t m, const int64_t* __restrict__ colptr, unsigned long long* mm) {
  unsigned long long lo = ~0ull, hi = 0;
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < m; j += (int64_t)gridDim.x * blockDim.x) {
    unsigned long long c = (unsigned long long)(colptr[j + 1] - colptr[j]);
    lo = min(lo, c);
    hi = max(hi, c);
  }
  for (int o = 16; o; o >>= 1) {
    lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMin(mm, lo);
    atomicMax(mm + 1, hi);
  }
}

__global__ void init_minmax(unsigned long long* mm) {
  mm[0] = ~0ull;
  mm[1] = 0ull;
}

__global__ void idf_kernel(int64_t n, int64_t m, const int64_t* __restrict__ colptr,
                           const unsigned long long* __restrict__ mm, double* __restrict__ w) {
  const bool equal = mm[0] == mm[1];
  const double dn = (double)n;
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < m; j += (int64_t)gridDim.x * blockDim.x) {
    if (equal) { w[j] = 1.0; continue; }
    double c = (double)(colptr[j + 1] - colptr[j]);
    if (c == 0.0) c = 1.0;
    else if (c == dn) c = dn - 1.0;
    w[j] = log(dn / c);
  }
}

// rinv_i = 1 / ||(x_i ⊙ w)||_2
__global__ void rownorm_kernel(int64_t n, const int64_t* __restrict__ ptr, const int32_t* __restrict__ idx,
                               const float* __restrict__ val, const double* __restrict__ w,
                               double* __restrict__ rinv, int* status, unsigned long long* bad) {
  const int lane = threadIdx.x & 31;
  const int64_t gw = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t r = gw; r < n; r += nw) {
    double s = 0.0;
    for (int64_t k = ptr[r] + lane; k < ptr[r + 1]; k += 32) {
      double x = w[idx[k]];
      if (val) x *= (double)val[k];
      s = fma(x, x, s);
    }
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) {
      if (!(s > 0.0)) report_error(status, bad, SG_ERR_NUMERIC, (unsigned long long)r);
      rinv[r] = 1.0 / sqrt(s);
    }
  }
}

// colsum_j = w_j * sum_{i in col j} x_ij rinv_i   (CSC gather); prod_j = w_j colsum_j
__global__ void colsum_kernel(int64_t m, const int64_t* __restrict__ cptr, const int32_t* __restrict__ ridx,
                              const float* __restrict__ cval, const double* __restrict__ w,
                              const double* __restrict__ rinv, double* __restrict__ colsum,
                              double* __restrict__ prod) {
  const int lane = threadIdx.x & 31;
  const int64_t gw = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t j = gw; j < m; j += nw) {
    double s = 0.0;
    for (int64_t k = cptr[j] + lane; k < cptr[j + 1]; k += 32) {
      double x = rinv[ridx[k]];
      if (cval) x *= (double)cval[k];
      s += x;
    }
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) {
      const double c = s * w[j];
      colsum[j] = c;
      prod[j] = w[j] * c;
    }
  }
}

// d_i = rinv_i * sum_j x_ij prod_j ; dinv = 1/(d-1) ; a = rinv*sqrt(dinv).  The
// gathers bind (one 32-byte sector of L2 per nonzero, one L1 lookup a clock):
// one per nonzero instead of two, 2.62 -> 1.37 ms at 4.1e8 nonzeros.
__global__ void degree_kernel(int64_t n, const int64_t* __restrict__ ptr, const int32_t* __restrict__ idx,
                              const float* __restrict__ val, const double* __restrict__ prod,
                              const double* __restrict__ rinv, double* __restrict__ a, double* __restrict__ dinv, float* __restrict__ a32,
                              float* __restrict__ dinv32, int* status, unsigned long long* bad) {
  const int lane = threadIdx.x & 31;
  const int64_t gw = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t r = gw; r < n; r += nw) {
    double s = 0.0;
    for (int64_t k = ptr[r] + lane; k < ptr[r + 1]; k += 32) {
      double x = prod[idx[k]];
      if (val) x *= (double)val[k];
      s += x;
    }
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) {
      const double d = s * rinv[r];
      const double di = 1.0 / (d - 1.0);
      if (!(di > 0.0) || isinf(di)) report_error(status, bad, SG_ERR_NUMERIC, (unsigned long long)r);
      const double ai = rinv[r] * sqrt(di);
      a[r] = ai;
      dinv[r] = di;
      if (a32) a32[r] = (float)ai;
      if (dinv32) dinv32[r] = (float)di;
    }
  }
}

__global__ void square_weights(int64_t m, const double* __restrict__ w, double* __restrict__ w2,
                               float* __restrict__ w2f) {
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < m; j += (int64_t)gridDim.x * blockDim.x) {
    const double v = w[j] * w[j];
    w2[j] = v;
    if (w2f) w2f[j] = (float)v;
  }
}

// ---------------------------------------------------------------------------
// CSR SpMM over a block of B dense columns:
//   out[r,:] = s_r * sum_{e in row r} x_e * in[col_e,:]  (- d_r * y[r,:])
// One warp per row.  The B values of a gathered row are split into 16-byte
// vectors, LPN lanes per nonzero, so each warp step gathers 32/LPN rows with
// coalesced 128-bit loads; the 32 column indices of a chunk are read once
// (one coalesced 128-byte load) and broadcast by shuffles.  Partial sums are
// combined by a fixed xor-shuffle tree: results are deterministic.
// ---------------------------------------------------------------------------
// Variants (same arithmetic, same result, picked by the autotuner): bits 0-1
// select 1, 2, 4 or 8 chunks of 32 column indices in flight per iteration
// (more gathers outstanding per lane against fewer resident warps); bit 2
// sends the gathers through L2 only (ld.global.cg).
template <typename VT>
__device__ __forceinline__ VT gather16(const VT* p, bool l2only) {
  return l2only ? __ldcg(p) : __ldg(p);
}

// DYN: a persistent grid whose warps take kDynRows rows at a time from an
// atomic counter (zeroed by the host before the launch), so that the long
// rows of a skewed matrix do not leave a tail of idle SMs; each row is still
// summed by one warp in the same order (same result as the static schedule).
constexpr int kDynRows = 4;
// With `order` the counter walks positions instead of rows: order[p] is the
// row at position p (-1: none), laid out by sg_row_order so that the longest
// rows are taken first, one per 4-row fetch (longest-first scheduling: the
// last rows to finish are short ones).  Each row is still summed by one warp
// in the same order: the result does not change.

template <typename T, int B, bool VALUED, bool SHIFT, int VAR, bool DYN = false>
__global__ void __launch_bounds__(256)
spmm_kernel(int64_t rows, const int64_t* __restrict__ ptr, const int32_t* __restrict__ idx,
            const float* __restrict__ val, const T* __restrict__ in, T* __restrict__ out,
            const T* __restrict__ scale, const T* __restrict__ dshift, const T* __restrict__ y,
            const unsigned char* __restrict__ row_mask, unsigned int* __restrict__ counter = nullptr,
            const int32_t* __restrict__ order = nullptr) {
  using VT = typename V16<T>::type;
  constexpr int VW = V16<T>::n;
  constexpr int LPN = B / VW;          // lanes per nonzero
  constexpr int NPS = 32 / LPN;        // nonzeros per warp step
  constexpr int CH = 1 << (VAR & 3);   // 32-index chunks per iteration
  constexpr bool L2ONLY = (VAR & 4) != 0;
  constexpr bool STREAM = false;
  static_assert(B % VW == 0 && LPN >= 1 && LPN <= 32, "unsupported block width");
  const int lane = threadIdx.x & 31;
  const int sub = lane % LPN, slot = lane / LPN;
  const int64_t gw = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  int64_t r = DYN ? 0 : gw, rend = DYN ? 0 : rows;
  while (true) {
    if (DYN) {
      if (r >= rend) {  // next chunk of rows for this warp
        unsigned int c0 = 0;
        if (lane == 0) c0 = atomicAdd(counter, (unsigned int)kDynRows);
        c0 = __shfl_sync(0xffffffffu, c0, 0);
        r = c0;
        rend = r + kDynRows < rows ? r + kDynRows : rows;
        if (r >= rows) break;
      }
    } else if (r >= rows) {
      break;
    }
    int64_t rr = r;
    r += DYN ? 1 : nw;
    if (DYN && order) {  // position -> row (-1: no row at this position)
      rr = order[rr];
      if (rr < 0) continue;
    }
    if (row_mask && !row_mask[rr]) continue;  // frozen row (warp-uniform)
    const int64_t s = ptr[rr], e = ptr[rr + 1];
    VT acc = V16<T>::zero();
    for (int64_t base = s; base < e; base += 32 * CH) {
      int ci[CH];
      float cv[CH];
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        const int64_t k = base + c * 32 + lane;
        ci[c] = k < e ? (STREAM ? __ldcs(idx + k) : __ldg(idx + k)) : -1;
        cv[c] = (VALUED && k < e) ? (STREAM ? __ldcs(val + k) : __ldg(val + k)) : 1.0f;
      }
      VT g[CH * LPN];
      float gv[CH * LPN];
#pragma unroll
      for (int c = 0; c < CH; ++c)
#pragma unroll
        for (int j = 0; j < LPN; ++j) {
          const int col = __shfl_sync(0xffffffffu, ci[c], j * NPS + slot);
          if (VALUED) gv[c * LPN + j] = __shfl_sync(0xffffffffu, cv[c], j * NPS + slot);
          g[c * LPN + j] = col >= 0 ? gather16(reinterpret_cast<const VT*>(in + (int64_t)col * B) + sub, L2ONLY)
                                    : V16<T>::zero();
        }
#pragma unroll
      for (int t = 0; t < CH * LPN; ++t) {
        if (VALUED) V16<T>::fma(acc, (T)gv[t], g[t]);
        else V16<T>::add(acc, g[t]);
      }
    }
#pragma unroll
    for (int o = LPN; o < 32; o <<= 1) V16<T>::add(acc, V16<T>::shfl_xor(acc, o));
    if (slot == 0) {
      const T sc = scale[rr];
      T* op = out + rr * B + sub * VW;
      const T* a = reinterpret_cast<const T*>(&acc);
      VT o;
      T* ov = reinterpret_cast<T*>(&o);
      if (SHIFT) {
        const T d = dshift[rr];
        const T* yp = y + rr * B + sub * VW;
#pragma unroll
        for (int q = 0; q < VW; ++q) ov[q] = sc * a[q] - d * yp[q];
      } else {
#pragma unroll
        for (int q = 0; q < VW; ++q) ov[q] = sc * a[q];
      }
      *reinterpret_cast<VT*>(op) = o;
    }
  }
}

constexpr int kSpmmVariants = 8;

template <typename T, int B, int VAR>
void launch_spmm_v(int64_t rows, const int64_t* ptr, const int32_t* idx, const float* val, const T* in, T* out,
                   const T* scale, const T* dshift, const T* y, int grid, cudaStream_t s, const unsigned char* mk) {
  if (val) {
    if (dshift) spmm_kernel<T, B, true, true, VAR><<<grid, 256, 0, s>>>(rows, ptr, idx, val, in, out, scale, dshift, y, mk);
    else spmm_kernel<T, B, true, false, VAR><<<grid, 256, 0, s>>>(rows, ptr, idx, val, in, out, scale, dshift, y, mk);
  } else {
    if (dshift) spmm_kernel<T, B, false, true, VAR><<<grid, 256, 0, s>>>(rows, ptr, idx, val, in, out, scale, dshift, y, mk);
    else spmm_kernel<T, B, false, false, VAR><<<grid, 256, 0, s>>>(rows, ptr, idx, val, in, out, scale, dshift, y, mk);
  }
}

template <typename T, int B>
int launch_spmm_t(int variant, int64_t rows, const int64_t* ptr, const int32_t* idx, const float* val, const T* in,
                  T* out, const T* scale, const T* dshift, const T* y, int grid, cudaStream_t s,
                  const unsigned char* mk) {
  switch (variant) {
    case 0: launch_spmm_v<T, B, 0>(rows, ptr, idx, val, in, out, scale, dshift, y, grid, s, mk); break;
    case 1: launch_spmm_v<T, B, 1>(rows, ptr, idx, val, in, out, scale, dshift, y, grid, s, mk); break;
    case 2: launch_spmm_v<T, B, 2>(rows, ptr, idx, val, in, out, scale, dshift, y, grid, s, mk); break;
    case 3: launch_spmm_v<T, B, 3>(rows, ptr, idx, val, in, out, scale, dshift, y, grid, s, mk); break;
    case 4: launch_spmm_v<T, B, 4>(rows, ptr, idx, val, in, out, scale, dshift, y, grid, s, mk); break;
    case 5: launch_spmm_v<T, B, 5>(rows, ptr, idx, val, in, out, scale, dshift, y, grid, s, mk); break;
    case 6: launch_spmm_v<T, B, 6>(rows, ptr, idx, val, in, out, scale, dshift, y, grid, s, mk); break;
    case 7: launch_spmm_v<T, B, 7>(rows, ptr, idx, val, in, out, scale, dshift, y, grid, s, mk); break;
    default: return SG_ERR_ARG;
  }
  return cudaGetLastError() == cudaSuccess ? SG_OK : SG_ERR_CUDA;
}

template <typename T>
int launch_spmm(int variant, int B, int64_t rows, const int64_t* ptr, const int32_t* idx, const float* val,
                const T* in, T* out, const T* scale, const T* dshift, const T* y, int grid, cudaStream_t s,
                const unsigned char* mk) {
  switch (B) {
    case 4: return launch_spmm_t<T, 4>(variant, rows, ptr, idx, val, in, out, scale, dshift, y, grid, s, mk);
    case 8: return launch_spmm_t<T, 8>(variant, rows, ptr, idx, val, in, out, scale, dshift, y, grid, s, mk);
    case 16: return launch_spmm_t<T, 16>(variant, rows, ptr, idx, val, in, out, scale, dshift, y, grid, s, mk);
    case 32: return launch_spmm_t<T, 32>(variant, rows, ptr, idx, val, in, out, scale, dshift, y, grid, s, mk);
    default: return SG_ERR_ARG;
  }
}

int sm_count() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms > 0 ? sms : 1;
}

}  // namespace
}  // namespace sg

using namespace sg;

extern "C" int sg_csr_select_cols(int64_t n, const int64_t* indptr, const int32_t* indices, const float* values,
                                  const int32_t* colmap, int64_t* out_indptr, int32_t* out_indices,
                                  float* out_values, void* scan_scratch, void* stream) {
  if (n < 0) return SG_ERR_ARG;
  cudaStream_t s = as_stream(stream);
  if (n == 0) return cudaMemsetAsync(out_indptr, 0, sizeof(int64_t), s) == cudaSuccess ? SG_OK : SG_ERR_CUDA;
  const int grid = grid_for(n * 32, 256, 8 * sm_count() * 8);
  if (cudaMemsetAsync(out_indptr, 0, sizeof(int64_t), s) != cudaSuccess) return SG_ERR_CUDA;
  select_count<<<grid, 256, 0, s>>>(n, indptr, indices, colmap, out_indptr);
  SG_CHECK_LAUNCH();
  if (inclusive_scan_i64(out_indptr + 1, n, scan_scratch, s) != cudaSuccess) return SG_ERR_CUDA;
  select_fill<<<grid, 256, 0, s>>>(n, indptr, indices, values, colmap, out_indptr, out_indices, out_values);
  SG_CHECK_LAUNCH();
  return SG_OK;
}

extern "C" int sg_transpose_blocks(void) { return 2 * sm_count(); }

// Row blocks of a transpose: sixteen waves of the two CTAs that an SM holds,
// and at least one step of the fill per block.
extern "C" int sg_transpose_row_blocks(int64_t n, int64_t m) {
  const int64_t P = (m + kTrPanel - 1) / kTrPanel;
  const int64_t want = P > 0 ? (32 * (int64_t)sm_count() + P - 1) / P : 1, most = n / kTrRows;
  return (int)std::max<int64_t>(1, std::min(want, most));
}

extern "C" int64_t sg_transpose_work_bytes(int64_t n, int64_t m, int nblk) {
  if (n < 0 || m <= 0 || nblk <= 0) return -1;
  const int64_t P = (m + kTrPanel - 1) / kTrPanel;
  const int64_t cnt = (int64_t)nblk * m * 4;
  return (cnt + 255) / 256 * 256 + n * (P + 1) * 4;
}

extern "C" int sg_csr_transpose(int64_t n, int64_t m, const int64_t* indptr, const int32_t* indices,
                                const float* values, int nblk, void* work, int64_t work_bytes, int64_t* colptr,
                                int32_t* rowidx, float* cvalues, void* scan_scratch, int* status, void* stream) {
  if (n <= 0 || m <= 0 || nblk <= 0 || m > 0x7fffffffLL || n > 0x7fffffffLL) return SG_ERR_ARG;
  if (work_bytes < sg_transpose_work_bytes(n, m, nblk) || ((uintptr_t)work & 255u)) return SG_ERR_CAP;
  cudaStream_t s = as_stream(stream);
  const int64_t P64 = (m + kTrPanel - 1) / kTrPanel;
  const int P = (int)P64;
  int32_t* cnt = reinterpret_cast<int32_t*>(work);
  int32_t* seg = reinterpret_cast<int32_t*>(reinterpret_cast<char*>(work) + ((int64_t)nblk * m * 4 + 255) / 256 * 256);
  const size_t smem = kTrPanel * (sizeof(int64_t) + (kTrRows / 32) * sizeof(uint32_t));
  if (cudaFuncSetAttribute(tr_fill, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return SG_ERR_CUDA;
  seg_kernel<<<grid_for(n * 32, 256, 8 * sm_count() * 4), 256, 0, s>>>(n, indptr, indices, P, m, seg, status);
  SG_CHECK_LAUNCH();
  constexpr int kGridY = 32768;  // panels per launch (the grid's second dimension ends at 65,535)
  for (int p0 = 0; p0 < P; p0 += kGridY)
    tr_count<<<dim3(nblk, std::min(P - p0, kGridY)), kTrThreads, 0, s>>>(n, m, indptr, indices, seg, p0, nblk, cnt,
                                                                         status);
  SG_CHECK_LAUNCH();
  const int g = grid_for(m, 256, 4096);
  tr_total<<<g, 256, 0, s>>>(m, nblk, cnt, colptr);
  SG_CHECK_LAUNCH();
  if (inclusive_scan_i64(colptr + 1, m, scan_scratch, s) != cudaSuccess) return SG_ERR_CUDA;
  tr_offsets<<<g, 256, 0, s>>>(m, nblk, cnt);
  SG_CHECK_LAUNCH();
  for (int p0 = 0; p0 < P; p0 += kGridY)
    tr_fill<<<dim3(nblk, std::min(P - p0, kGridY)), kTrThreads, smem, s>>>(n, m, indptr, indices, values, seg, p0, nblk,
                                                                           cnt, colptr, rowidx, cvalues, status);
  SG_CHECK_LAUNCH();
  return SG_OK;
}

extern "C" int sg_spectral_prepare(int64_t n, int64_t m, const int64_t* indptr, const int32_t* indices,
                                   const float* values, const int64_t* colptr, const int32_t* rowidx,
                                   const float* cvalues, const double* feature_weights, double* w,
                                   double* w2, float* w2_32, double* rinv, double* colsum, double* a,
                                   double* dinv, float* a32, float* dinv32, unsigned long long* minmax,
                                   int* status, unsigned long long* bad, void* stream) {
  if (n <= 0 || m <= 0) return SG_ERR_ARG;
  cudaStream_t s = as_stream(stream);
  const int sms = sm_count();
  const int gm = grid_for(m, 256, 8 * sms);
  const int gw_rows = grid_for(n * 32, 256, 8 * sms * 4);
  const int gw_cols = grid_for(m * 32, 256, 8 * sms * 4);
  if (feature_weights) {
    if (cudaMemcpyAsync(w, feature_weights, (size_t)m * sizeof(double), cudaMemcpyDeviceToDevice, s) != cudaSuccess)
      return SG_ERR_CUDA;
  } else {
    init_minmax<<<1, 1, 0, s>>>(minmax);
    colcount_minmax<<<gm, 256, 0, s>>>(m, colptr, minmax);
    SG_CHECK_LAUNCH();
    idf_kernel<<<gm, 256, 0, s>>>(n, m, colptr, minmax, w);
    SG_CHECK_LAUNCH();
  }
  rownorm_kernel<<<gw_rows, 256, 0, s>>>(n, indptr, indices, values, w, rinv, status, bad);
  colsum_kernel<<<gw_cols, 256, 0, s>>>(m, colptr, rowidx, cvalues, w, rinv, colsum, w2);  // w2 holds the product until it is set below
  degree_kernel<<<gw_rows, 256, 0, s>>>(n, indptr, indices, values, w2, rinv, a, dinv, a32, dinv32, status, bad);
  square_weights<<<gm, 256, 0, s>>>(m, w, w2, w2_32);
  SG_CHECK_LAUNCH();
  return SG_OK;
}

template <int B, int VAR>
int launch_spmm_dyn_v(int64_t rows, const int64_t* ptr, const int32_t* idx, const float* val, const float* in,
                      float* out, const float* scale, const float* dshift, const float* y, cudaStream_t s,
                      const unsigned char* mk, unsigned int* counter, const int32_t* order) {
  auto run = [&](auto kern) -> int {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 256, 0) != cudaSuccess || per_sm < 1)
      per_sm = 1;
    const int64_t need = (rows + kDynRows * 8 - 1) / (kDynRows * 8);  // blocks that can get a chunk
    int64_t grid = (int64_t)per_sm * sm_count();
    if (grid > need) grid = need;
    if (grid < 1) grid = 1;
    if (cudaMemsetAsync(counter, 0, sizeof(unsigned int), s) != cudaSuccess) return SG_ERR_CUDA;
    kern<<<(unsigned)grid, 256, 0, s>>>(rows, ptr, idx, val, in, out, scale, dshift, y, mk, counter, order);
    return cudaGetLastError() == cudaSuccess ? SG_OK : SG_ERR_CUDA;
  };
  if (val) {
    if (dshift) return run(spmm_kernel<float, B, true, true, VAR, true>);
    return run(spmm_kernel<float, B, true, false, VAR, true>);
  }
  if (dshift) return run(spmm_kernel<float, B, false, true, VAR, true>);
  return run(spmm_kernel<float, B, false, false, VAR, true>);
}

template <int B>
int launch_spmm_dyn_b(int variant, int64_t rows, const int64_t* ptr, const int32_t* idx, const float* val,
                      const float* in, float* out, const float* scale, const float* dshift, const float* y,
                      cudaStream_t s, const unsigned char* mk, unsigned int* counter, const int32_t* order) {
  switch (variant) {
    case 0: return launch_spmm_dyn_v<B, 0>(rows, ptr, idx, val, in, out, scale, dshift, y, s, mk, counter, order);
    case 1: return launch_spmm_dyn_v<B, 1>(rows, ptr, idx, val, in, out, scale, dshift, y, s, mk, counter, order);
    case 2: return launch_spmm_dyn_v<B, 2>(rows, ptr, idx, val, in, out, scale, dshift, y, s, mk, counter, order);
    case 3: return launch_spmm_dyn_v<B, 3>(rows, ptr, idx, val, in, out, scale, dshift, y, s, mk, counter, order);
    case 4: return launch_spmm_dyn_v<B, 4>(rows, ptr, idx, val, in, out, scale, dshift, y, s, mk, counter, order);
    case 5: return launch_spmm_dyn_v<B, 5>(rows, ptr, idx, val, in, out, scale, dshift, y, s, mk, counter, order);
    case 6: return launch_spmm_dyn_v<B, 6>(rows, ptr, idx, val, in, out, scale, dshift, y, s, mk, counter, order);
    case 7: return launch_spmm_dyn_v<B, 7>(rows, ptr, idx, val, in, out, scale, dshift, y, s, mk, counter, order);
    default: return SG_ERR_ARG;
  }
}

__global__ void count_minmax(int64_t m, const double* __restrict__ cnt, unsigned long long* mm) {
  unsigned long long lo = ~0ull, hi = 0;
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < m; j += (int64_t)gridDim.x * blockDim.x) {
    const unsigned long long c = (unsigned long long)cnt[j];
    lo = c < lo ? c : lo;
    hi = c > hi ? c : hi;
  }
  for (int o = 16; o; o >>= 1) {
    const unsigned long long a = __shfl_xor_sync(0xffffffffu, lo, o), b = __shfl_xor_sync(0xffffffffu, hi, o);
    lo = a < lo ? a : lo;
    hi = b > hi ? b : hi;
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMin(mm, lo);
    atomicMax(mm + 1, hi);
  }
}

// idf_kernel's rules from per-column cell counts instead of CSC column pointers
__global__ void idf_from_counts(int64_t n, int64_t m, const double* __restrict__ cnt,
                                const unsigned long long* __restrict__ mm, double* __restrict__ w) {
  const bool equal = mm[0] == mm[1];
  const double dn = (double)n;
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < m; j += (int64_t)gridDim.x * blockDim.x) {
    if (equal) { w[j] = 1.0; continue; }
    double c = cnt[j];
    if (c == 0.0) c = 1.0;
    else if (c == dn) c = dn - 1.0;
    w[j] = log(dn / c);
  }
}

__global__ void init_mm(unsigned long long* mm) { mm[0] = ~0ull; mm[1] = 0; }

extern "C" int sg_idf_from_counts(int64_t n, int64_t m, const double* counts, double* w, unsigned long long* mm,
                                  void* stream) {
  if (n < 1 || m < 0 || (m > 0 && (!counts || !w || !mm))) return SG_ERR_ARG;
  if (m == 0) return SG_OK;
  cudaStream_t s = as_stream(stream);
  const int g = grid_for(m, 256, 4 * sm_count());
  init_mm<<<1, 1, 0, s>>>(mm);
  count_minmax<<<g, 256, 0, s>>>(m, counts, mm);
  idf_from_counts<<<g, 256, 0, s>>>(n, m, counts, mm, w);
  SG_CHECK_LAUNCH();
  return SG_OK;
}

extern "C" int sg_csr_row_norms(int64_t n, const int64_t* indptr, const int32_t* indices, const float* values,
                                const double* w, double* rinv, int* status, unsigned long long* bad, void* stream) {
  if (n < 0 || (n > 0 && (!indptr || !w || !rinv || !status))) return SG_ERR_ARG;
  if (n == 0) return SG_OK;
  cudaStream_t s = as_stream(stream);
  rownorm_kernel<<<grid_for(n * 32, 256, 8 * sm_count()), 256, 0, s>>>(n, indptr, indices, values, w, rinv, status,
                                                                      bad);
  SG_CHECK_LAUNCH();
  return SG_OK;
}

extern "C" int sg_spmm_variants(void) { return kSpmmVariants; }

namespace sg {
namespace {
int spmm_dyn_impl(int dtype, int block, int64_t rows, const int64_t* ptr, const int32_t* idx, const float* val,
                  const void* in, void* out, const void* scale, const void* dshift, const void* y, int variant,
                  const int32_t* order, const unsigned char* row_mask, unsigned int* counter, void* stream) {
  if (rows < 0 || rows >= (int64_t(1) << 31) || !scale || (dshift && !y) || !counter || variant < 0 ||
      variant >= kSpmmVariants || dtype != 0)
    return SG_ERR_ARG;
  if (rows == 0) return SG_OK;
  cudaStream_t s = as_stream(stream);
  const float *fi = (const float*)in, *fs = (const float*)scale, *fd = (const float*)dshift, *fy = (const float*)y;
  float* fo = (float*)out;
  switch (block) {
    case 4: return launch_spmm_dyn_b<4>(variant, rows, ptr, idx, val, fi, fo, fs, fd, fy, s, row_mask, counter, order);
    case 8: return launch_spmm_dyn_b<8>(variant, rows, ptr, idx, val, fi, fo, fs, fd, fy, s, row_mask, counter, order);
    case 16:
      return launch_spmm_dyn_b<16>(variant, rows, ptr, idx, val, fi, fo, fs, fd, fy, s, row_mask, counter, order);
    case 32:
      return launch_spmm_dyn_b<32>(variant, rows, ptr, idx, val, fi, fo, fs, fd, fy, s, row_mask, counter, order);
    default: return SG_ERR_ARG;
  }
}

// keys: ~len (descending length under an ascending sort), values: row index
__global__ void order_keys_kernel(int64_t rows, const int64_t* __restrict__ ptr, uint64_t* __restrict__ keys,
                                  uint64_t* __restrict__ vals) {
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < rows; r += (int64_t)gridDim.x * blockDim.x) {
    const int64_t len = ptr[r + 1] - ptr[r];
    keys[r] = 0xffffffffull - (uint64_t)(len < 0xffffffffll ? len : 0xffffffffll);
    vals[r] = (uint64_t)r;
  }
}

// position p = 4c + j holds the row of sorted rank c + j·C (C = ceil(rows/4)):
// each 4-row fetch gets one row of every quarter of the length order
__global__ void order_deal_kernel(int64_t rows, int64_t C, const uint64_t* __restrict__ sorted_rows,
                                  int32_t* __restrict__ order) {
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < 4 * C; p += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = p >> 2, j = p & 3;
    const int64_t q = c + j * C;
    order[p] = q < rows ? (int32_t)sorted_rows[q] : -1;
  }
}

struct OrderLayout {
  uint64_t *keys, *vals, *keys_alt, *vals_alt;
  void* radix;
  int64_t bytes;
};

OrderLayout order_layout(char* base, int64_t rows) {
  OrderLayout L{};
  int64_t o = 0;
  auto take = [&](int64_t b) { const int64_t r = o; o += (b + 255) / 256 * 256; return r; };
  const int64_t R = rows > 0 ? rows : 1;
  const int64_t ok = take(8 * R), ov = take(8 * R), oka = take(8 * R), ova = take(8 * R), orad = take(radix_scratch_bytes(R));
  if (base) {
    L.keys = (uint64_t*)(base + ok);
    L.vals = (uint64_t*)(base + ov);
    L.keys_alt = (uint64_t*)(base + oka);
    L.vals_alt = (uint64_t*)(base + ova);
    L.radix = base + orad;
  }
  L.bytes = o;
  return L;
}
}  // namespace
}  // namespace sg

extern "C" int sg_spmm_dyn(int dtype, int block, int64_t rows, const int64_t* ptr, const int32_t* idx,
                           const float* val, const void* in, void* out, const void* scale, const void* dshift,
                           const void* y, int variant, const unsigned char* row_mask, unsigned int* counter,
                           void* stream) {
  return spmm_dyn_impl(dtype, block, rows, ptr, idx, val, in, out, scale, dshift, y, variant, nullptr, row_mask,
                       counter, stream);
}

extern "C" int sg_spmm_dyn_ordered(int dtype, int block, int64_t positions, const int64_t* ptr, const int32_t* idx,
                                   const float* val, const void* in, void* out, const void* scale,
                                   const void* dshift, const void* y, int variant, const int32_t* order,
                                   unsigned int* counter, void* stream) {
  if (!order) return SG_ERR_ARG;
  return spmm_dyn_impl(dtype, block, positions, ptr, idx, val, in, out, scale, dshift, y, variant, order, nullptr,
                       counter, stream);
}

extern "C" int64_t sg_row_order_positions(int64_t rows) { return rows < 0 ? -1 : 4 * ((rows + 3) / 4); }

extern "C" int64_t sg_row_order_scratch_bytes(int64_t rows) { return rows < 0 ? -1 : order_layout(nullptr, rows).bytes; }

extern "C" int sg_row_order(int64_t rows, const int64_t* ptr, int32_t* order, void* scratch, int64_t scratch_bytes,
                            void* stream) {
  if (rows < 0 || rows >= (int64_t(1) << 31) || (rows > 0 && (!ptr || !order || !scratch))) return SG_ERR_ARG;
  if (((uintptr_t)scratch & 255u) != 0) return SG_ERR_ARG;
  if (rows == 0) return SG_OK;
  OrderLayout L = order_layout((char*)scratch, rows);
  if (scratch_bytes < L.bytes) return SG_ERR_CAP;
  cudaStream_t s = as_stream(stream);
  const int g = grid_for(rows, 256, 16 * sm_count());
  order_keys_kernel<<<g, 256, 0, s>>>(rows, ptr, L.keys, L.vals);
  SG_CHECK_LAUNCH();
  bool alt = false;
  if (radix_sort_u64(rows, L.keys, L.vals, L.keys_alt, L.vals_alt, 0, 32, L.radix, s, &alt) != cudaSuccess)
    return SG_ERR_CUDA;
  const int64_t C = (rows + 3) / 4;
  order_deal_kernel<<<grid_for(4 * C, 256, 16 * sm_count()), 256, 0, s>>>(rows, C, alt ? L.vals_alt : L.vals, order);
  SG_CHECK_LAUNCH();
  return SG_OK;
}

extern "C" int sg_spmm_masked(int dtype, int block, int64_t rows, const int64_t* ptr, const int32_t* idx,
                              const float* val, const void* in, void* out, const void* scale, const void* dshift,
                              const void* y, int grid, int variant, const unsigned char* row_mask, void* stream) {
  if (rows < 0 || !scale || (dshift && !y) || variant < 0 || variant >= kSpmmVariants) return SG_ERR_ARG;
  if (rows == 0) return SG_OK;
  if (grid <= 0) grid = grid_for(rows * 32, 256, 8 * sm_count() * 4);
  cudaStream_t s = as_stream(stream);
  if (dtype == 0)
    return launch_spmm<float>(variant, block, rows, ptr, idx, val, (const float*)in, (float*)out,
                              (const float*)scale, (const float*)dshift, (const float*)y, grid, s, row_mask);
  if (dtype == 1)
    return launch_spmm<double>(variant, block, rows, ptr, idx, val, (const double*)in, (double*)out,
                               (const double*)scale, (const double*)dshift, (const double*)y, grid, s, row_mask);
  return SG_ERR_ARG;
}

extern "C" int sg_spmm_ex(int dtype, int block, int64_t rows, const int64_t* ptr, const int32_t* idx,
                          const float* val, const void* in, void* out, const void* scale, const void* dshift,
                          const void* y, int grid, int variant, void* stream) {
  return sg_spmm_masked(dtype, block, rows, ptr, idx, val, in, out, scale, dshift, y, grid, variant, nullptr, stream);
}

extern "C" int sg_spmm(int dtype, int block, int64_t rows, const int64_t* ptr, const int32_t* idx,
                       const float* val, const void* in, void* out, const void* scale, const void* dshift,
                       const void* y, int grid, void* stream) {
  return sg_spmm_ex(dtype, block, rows, ptr, idx, val, in, out, scale, dshift, y, grid, 0, stream);
}
