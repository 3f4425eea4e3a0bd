// FP64 SpMM of an implicit-ones CSR by exact fixed-point sums:
//   out[r,:] = scale[r] * sum_{e in row r} in[col_e,:]  (- dshift[r] * y[r,:])
// for a dense block of B FP64 columns: the Gram matvec of the double-precision
// solve (snapatac2-python/src/embedding.rs:133-152), the adjoint's passes and
// the Nyström extension.
//
// What bounds it.  GB300 retires about two FP64 lanes per clock and SM, so
// summing the gathered rows with DADD is bound by the FP64 pipe at a quarter
// of the rate at which the rows arrive.  Here every column of `in` is scaled
// by a power of two (its largest magnitude becomes just below 2^62), rounded
// once to a 64-bit integer, and summed in 96-bit integers: three integer adds
// per value, no FP64 instruction per nonzero.  The sums are exact, so the
// result does not depend on the order of the additions (any split of a row
// gives the same bits).  An operand is off by at most 2^-63 of its column's
// largest magnitude, where each FP64 addition would round at 2^-53 of the
// running sum; measured against 64-bit sums of higher precision the result is
// no further off than the FP64 kernel's.  A column that holds an infinity or
// a NaN sends the whole call through FP64 additions (uniform branch), so
// non-finite values propagate as before.
//
// Layout: CTAs of 8 warps own R consecutive rows.  A warp sums its rows one
// by one, B/2 lanes per nonzero (16-byte gathers), and keeps each row's sum in
// the lanes of one slot, so that one epilogue with all lanes busy (an idle
// lane costs an FP64 slot too) scales 64/B rows.  Rows of more than kLong
// nonzeros are summed by the whole CTA afterwards.  R is the largest size
// that still gives every SM eight CTAs (short matrices take 4 rows a CTA).
// Four CTAs per SM (64 registers) beat three by 3-10 % and five by more; two
// index chunks in flight at 8 columns beat one (20 %) and four (30 %).
//
// Measured, Xᵀ / X pass with the FP64 kernel's best variant in brackets:
// 5,000 x 200,003, 2.1e7 nonzeros, 8 columns: 167 / 159 us (502 / 495); 2,000
// x 50,000, 3.1e6, 8 columns: 39 / 40 us (95 / 88); 20,000 x 300,000, 8.3e7:
// 4 columns 0.39 / 0.43 ms (0.97 / 0.74), 32 columns 1.39 / 1.85 ms (6.1 /
// 5.9), where the 256-byte rows arrive at 15 / 11 TB/s.  The gathers bind now.
#include "common.cuh"
#include "internal.h"

namespace sg {
namespace {

constexpr int kFxThreads = 256;
constexpr int kFxWarps = kFxThreads / 32;
constexpr int kLong = 512;         // nonzeros above which a row is shared by the CTA's warps
constexpr int kHeadBytes = 256;    // per-column maxima in front of the integers
constexpr unsigned kNonFinite = 0x7ff00000u;

// scale exponent of a column whose largest |x| has this high word: |x| 2^s < 2^62
__device__ __forceinline__ int fx_shift(unsigned maxhi) {
  const int ex = (int)(maxhi >> 20);
  return 1084 - (ex < 1 ? 1 : ex);
}

// x 2^s, -1083 <= s <= 1083 (a column near the bottom of the exponent range takes two steps)
__device__ __forceinline__ double scale2(double x, int s) {
  const int a = s < -1022 ? -1022 : (s > 1022 ? 1022 : s);
  x *= __longlong_as_double((long long)(a + 1023) << 52);
  if (a != s) x *= __longlong_as_double((long long)(s - a + 1023) << 52);
  return x;
}

// per-column maximum of the high words of |x| (ordered as the magnitudes are)
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
    a = max(a, (unsigned)__double2hiint(v.x) & 0x7fffffffu);
    b = max(b, (unsigned)__double2hiint(v.y) & 0x7fffffffu);
  }
  const int c = 2 * (threadIdx.x % (B / 2));
  atomicMax(&m[c], a);
  atomicMax(&m[c + 1], b);
  __syncthreads();
  if (threadIdx.x < B) atomicMax(head + threadIdx.x, m[threadIdx.x]);
}

// q = rint(x 2^s) + 2^63 (biased, so that the sums need no sign extension)
template <int B>
__global__ void __launch_bounds__(kFxThreads)
fx_quantize_kernel(int64_t nvec, const double2* __restrict__ in, const unsigned* __restrict__ head,
                   ulonglong2* __restrict__ q) {
  const int64_t stride = (int64_t)gridDim.x * kFxThreads;
  const int c = 2 * (threadIdx.x % (B / 2));
  const unsigned ha = head[c], hb = head[c + 1];
  if (ha >= kNonFinite || hb >= kNonFinite) return;  // the sums are taken in FP64 then
  const int sa = fx_shift(ha), sb = fx_shift(hb);
  for (int64_t i = blockIdx.x * (int64_t)kFxThreads + threadIdx.x; i < nvec; i += stride) {
    const double2 v = in[i];
    ulonglong2 o;
    o.x = (unsigned long long)__double2ll_rn(scale2(v.x, sa)) ^ (1ull << 63);
    o.y = (unsigned long long)__double2ll_rn(scale2(v.y, sb)) ^ (1ull << 63);
    q[i] = o;
  }
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

template <int B>
struct Acc {
  Sum96 a, b;  // the lane's two columns
  __device__ __forceinline__ void zero() { a = {0, 0, 0}; b = {0, 0, 0}; }
  __device__ __forceinline__ void add(const ulonglong2& g) {
    a.add((unsigned)g.x, (unsigned)(g.x >> 32));
    b.add((unsigned)g.y, (unsigned)(g.y >> 32));
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
    }
  }
};

// adds CH chunks of 32 nonzeros starting at k0 (entries at or past e are skipped)
template <int B, int CH>
__device__ __forceinline__ void fx_chunk(Acc<B>& acc, int64_t k0, int64_t e, const int32_t* __restrict__ idx,
                                         const ulonglong2* __restrict__ q, int lane) {
  constexpr int LPN = B / 2, NPS = 32 / LPN;
  constexpr int GB = LPN < 8 ? LPN : 8;  // gathers in flight per chunk
  const int sub = lane % LPN, slot = lane / LPN;
  int ci[CH];
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int64_t k = k0 + c * 32 + lane;
    ci[c] = k < e ? __ldg(idx + k) : -1;
  }
#pragma unroll
  for (int j0 = 0; j0 < LPN; j0 += GB) {
    ulonglong2 g[CH * GB];
#pragma unroll
    for (int c = 0; c < CH; ++c)
#pragma unroll
      for (int j = 0; j < GB; ++j) {
        const int col = __shfl_sync(0xffffffffu, ci[c], (j0 + j) * NPS + slot);
        g[c * GB + j] = col >= 0 ? __ldg(q + (int64_t)col * LPN + sub) : make_ulonglong2(0, 0);
      }
#pragma unroll
    for (int t = 0; t < CH * GB; ++t) acc.add(g[t]);
  }
}

// chunks k0, k0 + step, ... of a row
template <int B>
__device__ __forceinline__ void fx_row(Acc<B>& acc, int64_t k0, int64_t e, int64_t step,
                                       const int32_t* __restrict__ idx, const ulonglong2* __restrict__ q, int lane) {
  constexpr int CH = B == 4 ? 4 : (B == 8 ? 2 : 1);
  for (; k0 < e; k0 += step) {
    if (CH == 1 || k0 + 32 < e) fx_chunk<B, CH>(acc, k0, e, idx, q, lane);
    else fx_chunk<B, 1>(acc, k0, e, idx, q, lane);
  }
}

template <int B, bool SHIFT>
__device__ __forceinline__ void fx_store(int64_t r, int sub, double a, double b, double* __restrict__ out,
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
  *reinterpret_cast<double2*>(out + r * B + 2 * sub) = o;
}

template <int B, bool SHIFT>
__global__ void __launch_bounds__(kFxThreads, 4)
spmm_fx_kernel(int64_t rows, int R, const int64_t* __restrict__ ptr, const int32_t* __restrict__ idx,
               const double* __restrict__ in, const ulonglong2* __restrict__ q, const unsigned* __restrict__ head,
               double* __restrict__ out, const double* __restrict__ scale, const double* __restrict__ dshift,
               const double* __restrict__ y) {
  constexpr int LPN = B / 2, NPS = 32 / LPN;
  constexpr int CH = B == 4 ? 4 : (B == 8 ? 2 : 1);
  static_assert(NPS * kFxWarps <= kFxThreads, "one thread per row of the CTA");
  __shared__ int64_t s_ptr[kFxWarps * NPS + 1];
  __shared__ int s_long[kFxWarps * NPS];
  __shared__ int s_nlong;
  __shared__ unsigned s_part[2][kFxWarps][LPN][6];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = lane % LPN, slot = lane / LPN;
  const int64_t r0 = blockIdx.x * (int64_t)R;
  const int nr = (int)(rows - r0 < R ? rows - r0 : R);
  if (threadIdx.x == 0) s_nlong = 0;
  if (threadIdx.x <= nr) s_ptr[threadIdx.x] = ptr[r0 + threadIdx.x];
  const unsigned ha = head[2 * sub], hb = head[2 * sub + 1];
  const bool finite = __all_sync(0xffffffffu, ha < kNonFinite && hb < kNonFinite);  // the same in every warp
  __syncthreads();
  if (!finite) {  // FP64 additions, a warp per row
    for (int i = warp; i < nr; i += kFxWarps) {
      double2 acc = make_double2(0.0, 0.0);
      for (int64_t k = s_ptr[i] + slot; k < s_ptr[i + 1]; k += NPS)
        V16<double>::add(acc, *reinterpret_cast<const double2*>(in + (int64_t)idx[k] * B + 2 * sub));
      __syncwarp();
#pragma unroll
      for (int o = LPN; o < 32; o <<= 1) V16<double>::add(acc, V16<double>::shfl_xor(acc, o));
      if (slot == 0) fx_store<B, SHIFT>(r0 + i, sub, acc.x, acc.y, out, scale, dshift, y);
    }
    return;
  }
  const int sa = fx_shift(ha), sb = fx_shift(hb);
  if (threadIdx.x < nr && s_ptr[threadIdx.x + 1] - s_ptr[threadIdx.x] > kLong)
    s_long[atomicAdd(&s_nlong, 1)] = threadIdx.x;
  // rows of this warp, one after the other; row i of the warp ends up in slot i
  const int per = R < kFxWarps ? 1 : R / kFxWarps;  // <= NPS
  Acc<B> mine;
  mine.zero();
  unsigned mylen = 0;
  int myrow = -1;
  for (int i = 0; i < per; ++i) {
    const int t = warp * per + i;
    if (t >= nr) break;
    const int64_t s = s_ptr[t], e = s_ptr[t + 1];
    if (e - s > kLong) continue;
    Acc<B> acc;
    acc.zero();
    fx_row<B>(acc, s, e, 32 * CH, idx, q, lane);
    acc.fold();
    if (slot == i) {
      mine = acc;
      mylen = (unsigned)(e - s);
      myrow = t;
    }
  }
  if (myrow >= 0)
    fx_store<B, SHIFT>(r0 + myrow, sub, mine.a.value(mylen, sa), mine.b.value(mylen, sb), out, scale, dshift, y);
  __syncthreads();
  // long rows, by all warps; one barrier a row (the partial sums alternate between two buffers)
  const int nl = s_nlong;
  for (int l = 0; l < nl; ++l) {
    const int t = s_long[l];
    const int64_t s = s_ptr[t], e = s_ptr[t + 1];
    Acc<B> acc;
    acc.zero();
    fx_row<B>(acc, s + (int64_t)warp * 32 * CH, e, (int64_t)kFxWarps * 32 * CH, idx, q, lane);
    acc.fold();
    if (slot == 0) {
      unsigned* p = s_part[l & 1][warp][sub];
      p[0] = acc.a.lo; p[1] = acc.a.mid; p[2] = acc.a.hi;
      p[3] = acc.b.lo; p[4] = acc.b.mid; p[5] = acc.b.hi;
    }
    __syncthreads();
    if (warp == l % kFxWarps && slot == 0) {
      for (int w = 0; w < kFxWarps; ++w) {
        if (w == warp) continue;
        const unsigned* p = s_part[l & 1][w][sub];
        acc.a.add(p[0], p[1], p[2]);
        acc.b.add(p[3], p[4], p[5]);
      }
      const unsigned n = (unsigned)(e - s);
      fx_store<B, SHIFT>(r0 + t, sub, acc.a.value(n, sa), acc.b.value(n, sb), out, scale, dshift, y);
    }
  }
}

template <int B>
int launch_fx(int64_t rows, const int64_t* ptr, const int32_t* idx, int64_t in_rows, const double* in, double* out,
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
  int R = kFxWarps * (64 / B);
  while (R > 4 && (rows + R - 1) / R < 8 * (int64_t)sms) R >>= 1;
  const int64_t grid = (rows + R - 1) / R;
  if (grid > 0x7fffffffLL) return SG_ERR_ARG;
  if (dshift)
    spmm_fx_kernel<B, true><<<(unsigned)grid, kFxThreads, 0, s>>>(rows, R, ptr, idx, in, q, head, out, scale, dshift, y);
  else
    spmm_fx_kernel<B, false><<<(unsigned)grid, kFxThreads, 0, s>>>(rows, R, ptr, idx, in, q, head, out, scale, dshift,
                                                                   y);
  SG_CHECK_LAUNCH();
  return SG_OK;
}

}  // namespace
}  // namespace sg

using namespace sg;

extern "C" int64_t sg_spmm_fx_work_bytes(int block, int64_t in_rows) {
  if (in_rows < 0 || (block != 4 && block != 8 && block != 16 && block != 32)) return -1;
  return kHeadBytes + 8 * (int64_t)block * in_rows;
}

extern "C" int sg_spmm_fx(int block, int64_t rows, const int64_t* ptr, const int32_t* idx, int64_t in_rows,
                          const double* in, double* out, const double* scale, const double* dshift, const double* y,
                          void* work, int64_t work_bytes, void* stream) {
  const int64_t need = sg_spmm_fx_work_bytes(block, in_rows);
  if (rows < 0 || need < 0 || !scale || (dshift && !y)) return SG_ERR_ARG;
  if (rows == 0) return SG_OK;
  if (!work || work_bytes < need) return SG_ERR_CAP;
  if (((uintptr_t)work | (uintptr_t)in | (uintptr_t)out | (uintptr_t)y) & 15u) return SG_ERR_ARG;
  cudaStream_t s = as_stream(stream);
  char* w = reinterpret_cast<char*>(work);
  switch (block) {
    case 4: return launch_fx<4>(rows, ptr, idx, in_rows, in, out, scale, dshift, y, w, s);
    case 8: return launch_fx<8>(rows, ptr, idx, in_rows, in, out, scale, dshift, y, w, s);
    case 16: return launch_fx<16>(rows, ptr, idx, in_rows, in, out, scale, dshift, y, w, s);
    default: return launch_fx<32>(rows, ptr, idx, in_rows, in, out, scale, dshift, y, w, s);
  }
}
