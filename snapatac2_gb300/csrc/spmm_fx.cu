// FP64 SpMM of an implicit-ones CSR, or of one that holds counts, by exact
// fixed-point sums:
//   out[r,:] = scale[r] * sum_{e in row r} val_e in[col_e,:]  (- dshift[r] * y[r,:])
// for a dense block of B FP64 columns: the Gram matvec of the double-precision
// solve (snapatac2-python/src/embedding.rs:133-152), the adjoint's passes and
// the Nyström extension.
//
// What bounds it.  GB300 retires about two FP64 lanes per clock and SM, so
// summing the gathered rows with DADD is bound by the FP64 pipe at a quarter
// of the rate at which the rows arrive.  Here every column of `in` is scaled
// by a power of two (its largest magnitude becomes just below 2^63), rounded
// once to a 64-bit integer, and summed in 96-bit integers: three integer adds
// per value, no FP64 instruction per nonzero.  The sums are exact, so the
// result does not depend on the order of the additions (any split of a row
// gives the same bits).
//
// Accuracy.  An operand is off by one unit at most (2^-62 of its column's
// largest magnitude), a sum of len terms by len units, where FP64 additions
// are off by up to len 2^-53 sum|terms|.  So the fixed-point sum is the better
// one wherever sum|terms| is 2^53 units or more, and is used only where that
// is known: an operand of 2^kVouch = 2^55 units or more (a 128th to a 256th of
// the column's largest magnitude) is stored as an odd integer, every other as
// an even one, and the last bits of a row's operands are ORed on the way.  A
// row without an odd one in a column (its operands are all small beside the
// column's largest, or all zero) gets its sums there by FP64 additions
// (fx_plain), as does every row when a column holds an infinity or a NaN.
// 2^55 and not 2^53: where one operand alone vouches for many smaller ones, the
// additions round at its size in one lane of eight only, and at 2^55 the two
// errors are equal (0.6 sqrt(len) units).  In solves of 1,200 to 12,000 cells
// with IDF weights no row goes that way; with weights spread as e^N(0,1) 0.3 %
// of the rows of the X pass, as e^(3 N(0,1)) 8 % (an embedding of 5,000 cells:
// 21.5 ms, then 26.2; by FP64 additions alone 57).  Looking costs 3 % of the Xᵀ
// pass (137 -> 141 us below), nothing in the X pass.
//
// Layout: CTAs of 8 warps own R consecutive rows, and each warp an equal slice
// of their nonzeros, wherever the row ends fall: a row that lies in several
// slices is put together in shared memory at the end (a warp per row, with the
// rows above 512 nonzeros shared by the CTA and a barrier for each, waited 21 %
// of its time at barriers on rows of unequal length).  B/2 lanes take one
// nonzero (16-byte gathers); a row's sum is folded over the warp and left in
// shared memory, and one epilogue with all lanes busy (an idle lane costs an
// FP64 slot too) scales all the CTA's rows, a thread to two columns of one.
// Column indices are loaded one step ahead of the gathers, and a step's unused
// lanes read a row of zeros (3-9 % faster than a test per gather).
// Four CTAs per SM (64 registers) beat three by 1-40 % and five by more; two
// index chunks in flight at 8 columns beat one (10-30 %) and four (twice).
//
// Measured, Xᵀ / X pass with the FP64 kernel's best variant in brackets:
// 5,000 x 200,003, 2.1e7 nonzeros, 8 columns: 141 / 124 us (502 / 495); 2,000
// x 50,000, 3.1e6, 8 columns: 38 / 36 us (95 / 88); 20,000 x 300,000, 8.3e7:
// 4 columns 0.34 / 0.33 ms (0.97 / 0.74), 32 columns 0.99 / 1.17 ms (6.1 /
// 5.9), where the 256-byte rows arrive at 22 / 18 TB/s.  (A warp per short row
// and a CTA per long one: 167 / 159, 39 / 40, 390 / 430, 1,390 / 1,850.)  The
// L1's lookups bind now (83-90 % of its peak throughput).
//
// Counts (COUNTS): a tile matrix holds whole numbers; an operand's integer
// times a count below 2^16 is two wide integer multiplications, and with a
// row's counts summing to less than 2^32 the 96 bits still hold every sum
// exactly (the bias is taken out with the sum of the counts in place of the
// row's length).  The error is the sum of the counts in units, so the counts
// of the odd operands are summed instead of ORed: with a sum of V, sum|terms|
// is V 2^55 units or more, and V x (entries that are not zero) has to reach half
// of the counts' sum.  Of rows of more than 32 entries one gather in four is
// looked at (all: 222 / 185 us, none 186 / 153).  Three CTAs per SM (80
// registers).  The same matrices with counts 1 to 4: 213 / 164 us, 50 / 43, 0.41
// / 0.35 and 1.73 / 1.77 ms (FP64 multiply-adds: 664 / 682, 121 / 118, 1.27 /
// 1.02, 8.36 / 8.04).
#include "common.cuh"
#include "internal.h"

namespace sg {
namespace {

constexpr int kFxThreads = 256;
constexpr int kFxWarps = kFxThreads / 32;
constexpr int kFxCtas = 4;       // CTAs per SM (64 registers)
constexpr int kFxCtasCounts = 3;
template <int B>
constexpr int kFxMaxRows = kFxWarps * (64 / B);  // rows per CTA at most
constexpr int kHeadBytes = 256;    // per-column maxima in front of the integers
constexpr unsigned kNonFinite = 0x7ff00000u;
constexpr unsigned kVouch = 55;    // exponent of the magnitudes that vouch for a sum
constexpr int kLook = 4;           // COUNTS: every fourth gather of 32 entries (4 columns: every second) is looked at for
                                   // such, and all of a row's last 32 entries

// scale exponent of a column whose largest |x| has this high word: |x| 2^s < 2^63
__device__ __forceinline__ int fx_shift(unsigned maxhi) {
  const int ex = (int)(maxhi >> 20);
  return 1085 - (ex < 1 ? 1 : ex);
}

// x 2^s, -1084 <= s <= 1084 (a column near the bottom of the exponent range takes two steps)
__device__ __forceinline__ double scale2(double x, int s) {
  const int a = s < -1022 ? -1022 : (s > 1022 ? 1022 : s);
  x *= __longlong_as_double((long long)(a + 1023) << 52);
  if (a != s) x *= __longlong_as_double((long long)(s - a + 1023) << 52);
  return x;
}

// the high word of |x|, its last bit set where the low word is not zero: 0 for
// zero alone, and ordered as the magnitudes are as far as it goes
__device__ __forceinline__ unsigned abs_hi(double x) {
  return ((unsigned)__double2hiint(x) & 0x7fffffffu) | (__double2loint(x) != 0 ? 1u : 0u);
}

// per-column maximum of abs_hi (0: a column of zeros)
template <int B>
__global__ void __launch_bounds__(kFxThreads)
fx_max_kernel(int64_t nvec, const double2* __restrict__ in, unsigned* __restrict__ head) {
  __shared__ unsigned m[B];
  if (threadIdx.x < B) m[threadIdx.x] = 0;
  __syncthreads();
  unsigned a = 0, b = 0;
  const int64_t stride = (int64_t)gridDim.x * kFxThreads;  // a multiple of B / 2: a thread's columns stay
  for (int64_t i = blockIdx.x * (int64_t)kFxThreads + threadIdx.x; i < nvec; i += stride) {
    const double2 v = in[i];
    a = max(a, abs_hi(v.x));
    b = max(b, abs_hi(v.y));
  }
  const int c = 2 * (threadIdx.x % (B / 2));
  atomicMax(&m[c], a);
  atomicMax(&m[c + 1], b);
  __syncthreads();
  if (threadIdx.x < B) atomicMax(head + threadIdx.x, m[threadIdx.x]);
}

// Twice h = x 2^(s-1) as an integer: odd where it vouches for the sums it is in
// (kVouch), even elsewhere.  Magnitudes of 2^54 and more are even integers as
// they are, and turned odd by one, up in one row and down in the next.
__device__ __forceinline__ unsigned long long fx_integer(double h, bool zero_column, bool up) {
  const bool vouch = zero_column || ((unsigned)__double2hiint(h) & 0x7fffffffu) >= (1022u + kVouch) << 20;
  const long long q = 2 * __double2ll_rn(h) + (vouch ? (up ? 1 : -1) : 0);
  return (unsigned long long)q ^ (1ull << 63);  // biased, so that the sums need no sign extension
}

template <int B>
__global__ void __launch_bounds__(kFxThreads)
fx_quantize_kernel(int64_t nvec, const double2* __restrict__ in, const unsigned* __restrict__ head,
                   ulonglong2* __restrict__ q) {
  const int64_t stride = (int64_t)gridDim.x * kFxThreads;
  const int c = 2 * (threadIdx.x % (B / 2));
  const unsigned ha = head[c], hb = head[c + 1];
  if (ha >= kNonFinite || hb >= kNonFinite) return;  // the sums are taken in FP64 then
  if (blockIdx.x == 0 && threadIdx.x < B / 2) q[nvec + threadIdx.x] = make_ulonglong2(0, 0);  // read past a row's end
  const int sa = fx_shift(ha) - 1, sb = fx_shift(hb) - 1;
  for (int64_t i = blockIdx.x * (int64_t)kFxThreads + threadIdx.x; i < nvec; i += stride) {
    const double2 v = in[i];
    ulonglong2 o;
    const bool up = (i / (B / 2)) & 1;
    o.x = fx_integer(scale2(v.x, sa), ha == 0, up);
    o.y = fx_integer(scale2(v.y, sb), hb == 0, up);
    q[i] = o;
  }
}

// the largest of val, all of them whole numbers from 0 to 65,535, else 2^32 - 1
__global__ void __launch_bounds__(kFxThreads)
counts_max_kernel(int64_t nnz, const float* __restrict__ val, uint32_t* __restrict__ out) {
  unsigned m = 0;
  for (int64_t i = blockIdx.x * (int64_t)kFxThreads + threadIdx.x; i < nnz; i += (int64_t)gridDim.x * kFxThreads) {
    const float v = val[i];
    m = max(m, v >= 0.f && v <= 65535.f && v == truncf(v) ? (unsigned)v : 0xffffffffu);
  }
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

struct Sum96 {
  unsigned lo, mid, hi;
  __device__ __forceinline__ void add(unsigned l, unsigned m) {
    asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, 0;"
        : "+r"(lo), "+r"(mid), "+r"(hi)
        : "r"(l), "r"(m));
  }
  __device__ __forceinline__ void add(unsigned l, unsigned m, unsigned h) {
    asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, %5;"
        : "+r"(lo), "+r"(mid), "+r"(hi)
        : "r"(l), "r"(m), "r"(h));
  }
  // the sum of n biased integers, without the bias, times 2^-s
  __device__ __forceinline__ double value(unsigned n, int s) const {
    unsigned l = lo, m = mid, h = hi;
    asm("sub.cc.u32 %0, %0, %2;\n\tsubc.u32 %1, %1, %3;" : "+r"(m), "+r"(h) : "r"(n << 31), "r"(n >> 1));
    const long long top = (long long)(((unsigned long long)h << 32) | m);
    return scale2(fma(__ll2double_rn(top), 4294967296.0, (double)l), -s);
  }
};

// v times the 64-bit integer (v below 2^16)
__device__ __forceinline__ void add_times(Sum96& s, unsigned long long g, unsigned v) {
  const unsigned long long p = (unsigned long long)(unsigned)g * v;
  const unsigned long long r = (g >> 32) * v + (p >> 32);
  s.add((unsigned)p, (unsigned)r, (unsigned)(r >> 32));
}

template <int B, bool COUNTS>
struct Acc {
  Sum96 a, b;       // the lane's two columns
  unsigned va, vb;  // last bit: an operand that vouches was among them (COUNTS: their counts' sum)
  unsigned n;       // COUNTS: the sum of the counts
  __device__ __forceinline__ void zero() { a = {0, 0, 0}; b = {0, 0, 0}; va = vb = n = 0; }
  __device__ __forceinline__ void add(const ulonglong2& g, unsigned v, bool look) {
    add_times(a, g.x, v);
    add_times(b, g.y, v);
    if (look) {
      va += ((unsigned)g.x & 1u) * v;
      vb += ((unsigned)g.y & 1u) * v;
    }
    n += v;
  }
  __device__ __forceinline__ void add(const ulonglong2& g) {
    a.add((unsigned)g.x, (unsigned)(g.x >> 32));
    b.add((unsigned)g.y, (unsigned)(g.y >> 32));
    va |= (unsigned)g.x;
    vb |= (unsigned)g.y;
  }
  __device__ __forceinline__ void fold() {  // over the lanes of the same columns
#pragma unroll
    for (int o = B / 2; o < 32; o <<= 1) {
      const unsigned x0 = __shfl_xor_sync(0xffffffffu, a.lo, o), x1 = __shfl_xor_sync(0xffffffffu, a.mid, o),
                     x2 = __shfl_xor_sync(0xffffffffu, a.hi, o);
      const unsigned y0 = __shfl_xor_sync(0xffffffffu, b.lo, o), y1 = __shfl_xor_sync(0xffffffffu, b.mid, o),
                     y2 = __shfl_xor_sync(0xffffffffu, b.hi, o);
      a.add(x0, x1, x2);
      b.add(y0, y1, y2);
      if (COUNTS) {
        n += __shfl_xor_sync(0xffffffffu, n, o);
        va += __shfl_xor_sync(0xffffffffu, va, o);
        vb += __shfl_xor_sync(0xffffffffu, vb, o);
      }
    }
  }
};

// column indices of the first CH chunks of 32 of n nonzeros; past them the row
// of zeros behind the operand, which the gathers read without a test
template <int CH>
__device__ __forceinline__ void fx_load(int (&ci)[CH], const int32_t* __restrict__ p, int n, int zero, int lane) {
#pragma unroll
  for (int c = 0; c < CH; ++c) ci[c] = c * 32 + lane < n ? __ldg(p + c * 32 + lane) : zero;
}

// their counts (0 past them)
template <int CH>
__device__ __forceinline__ void fx_load_counts(float (&cv)[CH], const float* __restrict__ p, int n, int lane) {
#pragma unroll
  for (int c = 0; c < CH; ++c) cv[c] = c * 32 + lane < n ? __ldg(p + c * 32 + lane) : 0.f;
}

// adds the rows named by the first N chunks of ci (COUNTS: cv times each)
template <int B, int CH, int N, int LOOK, bool COUNTS>
__device__ __forceinline__ void fx_add(Acc<B, COUNTS>& acc, const int (&ci)[CH], const float (&cv)[CH],
                                       const ulonglong2* __restrict__ q, int lane) {
  constexpr int LPN = B / 2, NPS = 32 / LPN;
  constexpr int GB = LPN < 8 ? LPN : 8;  // gathers in flight per chunk
  const int sub = lane % LPN, slot = lane / LPN;
#pragma unroll
  for (int j0 = 0; j0 < LPN; j0 += GB) {
    ulonglong2 g[N * GB];
#pragma unroll
    for (int c = 0; c < N; ++c)
#pragma unroll
      for (int j = 0; j < GB; ++j) {
        const unsigned col = (unsigned)__shfl_sync(0xffffffffu, ci[c], (j0 + j) * NPS + slot);
        g[c * GB + j] = __ldg(q + (uint64_t)col * LPN + sub);
      }
#pragma unroll
    for (int t = 0; t < N * GB; ++t) {
      if constexpr (COUNTS)
        acc.add(g[t], __shfl_sync(0xffffffffu, (unsigned)cv[t / GB], (j0 + t % GB) * NPS + slot),
                (j0 + t % GB) % LOOK == 0);
      else
        acc.add(g[t]);
    }
  }
}

template <int B>
constexpr int kChunks = B == 4 ? 4 : (B == 8 ? 2 : 1);

// n nonzeros of a row from p on; ci holds the indices of the first
// chunks and receives those of the next nn nonzeros after the row (the warp's
// next row).  Indices are loaded one step ahead, so a step waits for the
// gathers alone.
template <int B, bool COUNTS>
__device__ __forceinline__ void fx_row(Acc<B, COUNTS>& acc, unsigned& nz, int (&ci)[kChunks<B>], float (&cv)[kChunks<B>],
                                       const int32_t* __restrict__ p, const float* __restrict__ pv, int n, int nn,
                                       int zero, const ulonglong2* __restrict__ q, int lane) {
  constexpr int CH = kChunks<B>, STEP = 32 * CH;
  while (n > 0) {
    int next[CH];
    float nextv[CH];
    const int adv = n < STEP ? n : STEP;
    p += adv;
    fx_load<CH>(next, p, n > STEP ? n - STEP : nn, zero, lane);
    if (COUNTS) {
      pv += adv;
      fx_load_counts<CH>(nextv, pv, n > STEP ? n - STEP : nn, lane);
    }
    if (COUNTS) {
#pragma unroll
      for (int c = 0; c < CH; ++c) nz += __popc(__ballot_sync(0xffffffffu, cv[c] != 0.f));
    }
    if (COUNTS && n <= 32) fx_add<B, CH, 1, 1>(acc, ci, cv, q, lane);
    else if (CH == 1 || n > 16 * CH) fx_add<B, CH, CH, kLook>(acc, ci, cv, q, lane);
    else if (CH == 4 && n > 32) fx_add<B, CH, CH == 4 ? 2 : 1, kLook>(acc, ci, cv, q, lane);
    else fx_add<B, CH, 1, kLook>(acc, ci, cv, q, lane);
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      ci[c] = next[c];
      if (COUNTS) cv[c] = nextv[c];
    }
    n -= STEP;
  }
}

// columns 2 sub and 2 sub + 1 of row r, those that are wanted
template <int B, bool SHIFT>
__device__ __forceinline__ void fx_store(int64_t r, int sub, bool wa, bool wb, double a, double b, double* __restrict__ out,
                                         const double* __restrict__ scale, const double* __restrict__ dshift,
                                         const double* __restrict__ y) {
  const double sc = scale[r];
  double2 o;
  if (SHIFT) {
    const double d = dshift[r];
    const double2 yv = *reinterpret_cast<const double2*>(y + r * B + 2 * sub);
    o.x = sc * a - d * yv.x;
    o.y = sc * b - d * yv.y;
  } else {
    o.x = sc * a;
    o.y = sc * b;
  }
  double* p = out + r * B + 2 * sub;
  if (wa && wb) {
    *reinterpret_cast<double2*>(p) = o;
  } else {
    if (wa) p[0] = o.x;
    if (wb) p[1] = o.y;
  }
}

// FP64 additions for the columns marked in s_plain (bit sub: 2 sub, bit 16 +
// sub: 2 sub + 1), a warp per row, four gathers in flight
template <int B, bool SHIFT, bool COUNTS>
__device__ __noinline__ void fx_plain(int64_t r0, int nr, const int* s_off, const unsigned* s_plain,
                                      const int32_t* __restrict__ idx, const float* __restrict__ val,
                                      const double* __restrict__ in, double* __restrict__ out,
                                      const double* __restrict__ scale, const double* __restrict__ dshift,
                                      const double* __restrict__ y, int warp, int lane) {
  constexpr int LPN = B / 2, NPS = 32 / LPN, U = 4;
  const int sub = lane % LPN, slot = lane / LPN;
  for (int i = warp; i < nr; i += kFxWarps) {
    const unsigned want = s_plain[i];
    if (!want) continue;
    double2 acc = make_double2(0.0, 0.0);
    const int e = s_off[i + 1];
    int k = s_off[i] + slot;
    for (; k + (U - 1) * NPS < e; k += U * NPS) {
      double2 g[U];
      double v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        v[u] = COUNTS ? (double)val[k + u * NPS] : 1.0;
        g[u] = *reinterpret_cast<const double2*>(in + (int64_t)idx[k + u * NPS] * B + 2 * sub);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) V16<double>::fma(acc, v[u], g[u]);
    }
    for (; k < e; k += NPS)
      V16<double>::fma(acc, COUNTS ? (double)val[k] : 1.0,
                       *reinterpret_cast<const double2*>(in + (int64_t)idx[k] * B + 2 * sub));
    __syncwarp();
#pragma unroll
    for (int o = LPN; o < 32; o <<= 1) V16<double>::add(acc, V16<double>::shfl_xor(acc, o));
    if (slot == 0)
      fx_store<B, SHIFT>(r0 + i, sub, want >> sub & 1u, want >> (16 + sub) & 1u, acc.x, acc.y, out, scale, dshift, y);
  }
}

template <int B, bool SHIFT, bool COUNTS>
__global__ void __launch_bounds__(kFxThreads, COUNTS ? kFxCtasCounts : kFxCtas)
spmm_fx_kernel(int64_t rows, int R, int zero, const int64_t* __restrict__ ptr, const int32_t* __restrict__ idx,
               const float* __restrict__ val,
               const double* __restrict__ in, const ulonglong2* __restrict__ q, const unsigned* __restrict__ head,
               double* __restrict__ out, const double* __restrict__ scale, const double* __restrict__ dshift,
               const double* __restrict__ y) {
  constexpr int LPN = B / 2, NPS = 32 / LPN;
  constexpr int CH = kChunks<B>;
  __shared__ int s_off[kFxMaxRows<B> + 2];  // row offsets in the CTA's nonzeros (below 2^31), the last one twice
  constexpr int NW = COUNTS ? 9 : 6;
  __shared__ unsigned s_sum[NW][kFxMaxRows<B> * LPN];  // of the rows, less the pieces in s_piece
  __shared__ unsigned s_piece[NW][kFxWarps * LPN];    // a warp's piece of the row that its slice ends inside of
  __shared__ int s_tail[kFxWarps];                    // that row, or -1
  // per row and per piece: the lanes that had an operand that vouches, for the
  // first and the second column of a lane (COUNTS: entries that are not zero)
  __shared__ unsigned s_sure[2][kFxMaxRows<B>], s_psure[2][kFxWarps];
  __shared__ unsigned s_plain[kFxMaxRows<B>];         // columns of the row by FP64 additions
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = lane % LPN, slot = lane / LPN;
  const int64_t r0 = blockIdx.x * (int64_t)R;
  const int nr = (int)(rows - r0 < R ? rows - r0 : R);
  const int64_t p0 = ptr[r0];
  if (threadIdx.x <= nr + 1) s_off[threadIdx.x] = (int)(ptr[r0 + min((int)threadIdx.x, nr)] - p0);
  idx += p0;
  if (COUNTS) val += p0;
  const unsigned ha = head[2 * sub], hb = head[2 * sub + 1];
  const bool finite = __all_sync(0xffffffffu, ha < kNonFinite && hb < kNonFinite);  // the same in every warp
  __syncthreads();
  if (!finite) {
    for (int i = threadIdx.x; i < nr; i += kFxThreads) s_plain[i] = ~0u;
    __syncthreads();
    fx_plain<B, SHIFT, COUNTS>(r0, nr, s_off, s_plain, idx, val, in, out, scale, dshift, y, warp, lane);
    return;
  }
  // this warp's slice [sl, sh) of the CTA's nonzeros; it finishes the rows
  // that end in (sl, sh] (warp 0 also the empty ones in front)
  const int total = s_off[nr], per = (total / kFxWarps + 32) / 32 * 32;
  const int sl = (int)min((int64_t)warp * per, (int64_t)total), sh = min((int64_t)sl + per, (int64_t)total);
  int t = 0;
  if (warp > 0)
    for (int i = 0; i < nr; i += 32) t += __popc(__ballot_sync(0xffffffffu, i + lane < nr && s_off[i + lane + 1] <= sl));
  const int32_t* p = idx + sl;
  int ci[CH], e = s_off[min(t, nr) + 1], n = t < nr ? min(e, sh) - sl : 0;
  int tail = -1;
  const float* pv = COUNTS ? val + sl : nullptr;
  float cv[CH];
  fx_load<CH>(ci, p, n, zero, lane);
  if (COUNTS) fx_load_counts<CH>(cv, pv, n, lane);
  for (; t < nr; ++t) {
    const bool ends = e <= sh;
    if (!ends && n == 0) break;
    const int e2 = s_off[t + 2], nn = min(e2, sh) - min(e, sh);
    Acc<B, COUNTS> acc;
    acc.zero();
    unsigned nz = 0;
    if (n == 0) {
      fx_load<CH>(ci, p, nn, zero, lane);
      if (COUNTS) fx_load_counts<CH>(cv, pv, nn, lane);
    } else {
      fx_row<B, COUNTS>(acc, nz, ci, cv, p, pv, n, nn, zero, q, lane);
    }
    p += n;
    if (COUNTS) pv += n;
    const unsigned sx = COUNTS ? nz : __ballot_sync(0xffffffffu, acc.va & 1u),
                   sy = COUNTS ? 0u : __ballot_sync(0xffffffffu, acc.vb & 1u);
    if (lane < 2) (ends ? s_sure[lane] + t : s_psure[lane] + warp)[0] = lane ? sy : sx;
    acc.fold();
    if (slot == 0) {
      unsigned* o = ends ? &s_sum[0][t * LPN + sub] : &s_piece[0][warp * LPN + sub];
      const int st = ends ? kFxMaxRows<B> * LPN : kFxWarps * LPN;
      o[0] = acc.a.lo; o[st] = acc.a.mid; o[2 * st] = acc.a.hi;
      o[3 * st] = acc.b.lo; o[4 * st] = acc.b.mid; o[5 * st] = acc.b.hi;
      if (COUNTS) {
        o[6 * st] = acc.n;
        o[7 * st] = acc.va;
        o[8 * st] = acc.vb;
      }
    }
    if (!ends) {
      tail = t;
      break;
    }
    n = nn;
    e = e2;
  }
  if (lane == 0) s_tail[warp] = tail;
  __syncthreads();
  // a thread per pair of columns of a row (an idle lane costs an FP64 slot too)
  static_assert(kFxMaxRows<B> * LPN == kFxThreads, "one item a thread");
  const int row = threadIdx.x / LPN;
  bool pa = false, pb = false;  // these columns of the row by FP64 additions
  if (row < nr) {
    Acc<B, COUNTS> acc;
    const int x = threadIdx.x;
    acc.a = {s_sum[0][x], s_sum[1][x], s_sum[2][x]};
    acc.b = {s_sum[3][x], s_sum[4][x], s_sum[5][x]};
    acc.n = COUNTS ? s_sum[6][x] : 0;
    acc.va = COUNTS ? s_sum[NW - 2][x] : 0;
    acc.vb = COUNTS ? s_sum[NW - 1][x] : 0;
    unsigned sx = s_sure[0][row], sy = s_sure[1][row];
#pragma unroll
    for (int w = 0; w < kFxWarps; ++w)
      if (s_tail[w] == row) {
        const int y2 = w * LPN + sub;
        acc.a.add(s_piece[0][y2], s_piece[1][y2], s_piece[2][y2]);
        acc.b.add(s_piece[3][y2], s_piece[4][y2], s_piece[5][y2]);
        if (COUNTS) {
          acc.n += s_piece[6][y2];
          acc.va += s_piece[NW - 2][y2];
          acc.vb += s_piece[NW - 1][y2];
          sx += s_psure[0][w];
        } else {
          sx |= s_psure[0][w];
          sy |= s_psure[1][w];
        }
      }
    const unsigned len = COUNTS ? acc.n : (unsigned)(s_off[row + 1] - s_off[row]);
    if (COUNTS) {
      pa = 2ull * acc.va * sx < acc.n;
      pb = 2ull * acc.vb * sx < acc.n;
    } else {
      constexpr unsigned kLanes = 0xffffffffu / ((1u << LPN) - 1u);  // lanes of the columns 0 and 1
      pa = len && !(sx & kLanes << sub);
      pb = len && !(sy & kLanes << sub);
    }
    fx_store<B, SHIFT>(r0 + row, sub, !pa, !pb, ha ? acc.a.value(len, fx_shift(ha)) : 0.0,
                       hb ? acc.b.value(len, fx_shift(hb)) : 0.0, out, scale, dshift, y);
  }
  constexpr unsigned kSubs = (1u << LPN) - 1u;
  const unsigned ma = __ballot_sync(0xffffffffu, pa) >> (lane / LPN * LPN),
                 mb = __ballot_sync(0xffffffffu, pb) >> (lane / LPN * LPN);
  if (sub == 0) s_plain[row] = (ma & kSubs) | (mb & kSubs) << 16;
  if (__syncthreads_or(pa || pb))
    fx_plain<B, SHIFT, COUNTS>(r0, nr, s_off, s_plain, idx, val, in, out, scale, dshift, y, warp, lane);
}

template <int B>
int launch_fx(int64_t rows, const int64_t* ptr, const int32_t* idx, const float* val, int64_t in_rows, const double* in, double* out,
              const double* scale, const double* dshift, const double* y, char* work, cudaStream_t s) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (sms < 1) sms = 1;
  unsigned* head = reinterpret_cast<unsigned*>(work);
  ulonglong2* q = reinterpret_cast<ulonglong2*>(work + kHeadBytes);
  const int64_t nvec = in_rows * (B / 2);
  if (cudaMemsetAsync(head, 0, 32 * sizeof(unsigned), s) != cudaSuccess) return SG_ERR_CUDA;
  const double2* v = reinterpret_cast<const double2*>(in);
  fx_max_kernel<B><<<grid_for(nvec, kFxThreads, 4 * sms), kFxThreads, 0, s>>>(nvec, v, head);
  SG_CHECK_LAUNCH();
  fx_quantize_kernel<B><<<grid_for(nvec, kFxThreads, 8 * sms), kFxThreads, 0, s>>>(nvec, v, head, q);
  SG_CHECK_LAUNCH();
  // rows per CTA: the shortest schedule in waves of resident CTAs, a CTA's
  // start counted as one row (5,000 equal rows as 1,250 CTAs on 608 places
  // left the third wave nearly empty)
  const int64_t slots = (int64_t)(val ? kFxCtasCounts : kFxCtas) * sms;
  int R = 1;
  int64_t best = INT64_MAX;
  for (int r = 1; r <= kFxMaxRows<B> && (r == 1 || r * in_rows <= INT32_MAX); ++r) {
    const int64_t cost = ((rows + r - 1) / r + slots - 1) / slots * (r + 1);
    if (cost < best) { best = cost; R = r; }
  }
  const int64_t grid = (rows + R - 1) / R;
  if (grid > 0x7fffffffLL) return SG_ERR_ARG;
  auto run = [&](auto kern) {
    kern<<<(unsigned)grid, kFxThreads, 0, s>>>(rows, R, (int)in_rows, ptr, idx, val, in, q, head, out, scale, dshift, y);
  };
  if (val) {
    if (dshift) run(spmm_fx_kernel<B, true, true>);
    else run(spmm_fx_kernel<B, false, true>);
  } else {
    if (dshift) run(spmm_fx_kernel<B, true, false>);
    else run(spmm_fx_kernel<B, false, false>);
  }
  SG_CHECK_LAUNCH();
  return SG_OK;
}

}  // namespace
}  // namespace sg

using namespace sg;

extern "C" int64_t sg_spmm_fx_work_bytes(int block, int64_t in_rows) {
  if (in_rows < 0 || (block != 4 && block != 8 && block != 16 && block != 32)) return -1;
  return kHeadBytes + 8 * (int64_t)block * (in_rows + 1);
}

namespace {
int spmm_fx_any(int block, int64_t rows, const int64_t* ptr, const int32_t* idx, const float* val, int64_t in_rows,
                const double* in, double* out, const double* scale, const double* dshift, const double* y, void* work,
                int64_t work_bytes, void* stream) {
  const int64_t need = sg_spmm_fx_work_bytes(block, in_rows);
  if (rows < 0 || need < 0 || in_rows > INT32_MAX || !scale || (dshift && !y)) return SG_ERR_ARG;
  if (rows == 0) return SG_OK;
  if (!work || work_bytes < need) return SG_ERR_CAP;
  if (((uintptr_t)work | (uintptr_t)in | (uintptr_t)out | (uintptr_t)y) & 15u) return SG_ERR_ARG;
  cudaStream_t s = as_stream(stream);
  char* w = reinterpret_cast<char*>(work);
  switch (block) {
    case 4: return launch_fx<4>(rows, ptr, idx, val, in_rows, in, out, scale, dshift, y, w, s);
    case 8: return launch_fx<8>(rows, ptr, idx, val, in_rows, in, out, scale, dshift, y, w, s);
    case 16: return launch_fx<16>(rows, ptr, idx, val, in_rows, in, out, scale, dshift, y, w, s);
    default: return launch_fx<32>(rows, ptr, idx, val, in_rows, in, out, scale, dshift, y, w, s);
  }
}
}  // namespace

extern "C" int sg_spmm_fx(int block, int64_t rows, const int64_t* ptr, const int32_t* idx, int64_t in_rows,
                          const double* in, double* out, const double* scale, const double* dshift, const double* y,
                          void* work, int64_t work_bytes, void* stream) {
  return spmm_fx_any(block, rows, ptr, idx, nullptr, in_rows, in, out, scale, dshift, y, work, work_bytes, stream);
}

extern "C" int sg_spmm_fx_counts(int block, int64_t rows, const int64_t* ptr, const int32_t* idx, const float* val,
                                 int64_t in_rows, const double* in, double* out, const double* scale,
                                 const double* dshift, const double* y, void* work, int64_t work_bytes,
                                 void* stream) {
  if (!val) return SG_ERR_ARG;
  return spmm_fx_any(block, rows, ptr, idx, val, in_rows, in, out, scale, dshift, y, work, work_bytes, stream);
}

extern "C" int sg_counts_max(int64_t nnz, const float* val, uint32_t* out, void* stream) {
  if (nnz < 0 || !out || (nnz > 0 && !val)) return SG_ERR_ARG;
  cudaStream_t s = as_stream(stream);
  if (cudaMemsetAsync(out, 0, sizeof(uint32_t), s) != cudaSuccess) return SG_ERR_CUDA;
  if (nnz == 0) return SG_OK;
  counts_max_kernel<<<grid_for(nnz, kFxThreads * 8, 16384), kFxThreads, 0, s>>>(nnz, val, out);
  SG_CHECK_LAUNCH();
  return SG_OK;
}
