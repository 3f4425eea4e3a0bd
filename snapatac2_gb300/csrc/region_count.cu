// Cell-by-region counts (peak matrix): fragments -> CSR of region hit
// counts, the arithmetic of RegionCounter::insert_fragment
// (snapatac2-core/src/feature_count/counter.rs:117-146) over the fragments
// that pair_to_fragments / single_to_fragments rebuild
// (snapatac2-core/src/feature_count/data_iter.rs:27-117), driven by
// create_peak_matrix (snapatac2-core/src/feature_count/matrix.rs:95-170).
//
// Regions are given per chromosome, sorted by start, with the running
// maximum of their ends: the regions that overlap [qs, qe) are those from the
// last start < qe backwards, until the running maximum end falls to qs or
// below.  A bucket index over the genome (sg_region_index: the first region
// that starts at or after every 2^shift-th base) narrows the search for that
// start to the regions of one bucket; without it the search is a binary one
// over the chromosome (18 dependent loads at 200,000 regions).
//
// Same phases as the tile matrix: plan counts the region hits ("keys") per
// cell and marks the fragments that have any; run collects the marked
// fragments' hits, sorts them (CTA radix sort over the bits the row spans)
// and run-length encodes them into (region, count) pairs; sg_tile_emit
// compacts the pairs into the CSR arrays (same scratch layout).
//
// Measured, 5,000 cells, 6.1e7 fragments, 200,000 peaks of 500 bp,
// paired-insertion: the call took 11.65 ms with the binary searches (plan
// 2.3 ms; run 8.7 ms, twice per fragment at one CTA of 512 threads per SM) and
// takes 2.44 ms.  What is left is the plan's two lookups per fragment, at the
// rate of L2 sector reads.
#include <algorithm>

#include "common.cuh"
#include "internal.h"

namespace sg {
namespace {

constexpr int kPlanBlock = 256;
constexpr int kRunBlock = 512;
constexpr int kSmemKeys = 24576;   // region_long_kernel: one CTA per SM
constexpr int kShortKeys = 4096;    // region_short_kernel: four CTAs per SM

struct RegionSet {
  const uint64_t* __restrict__ chrom_end;  // cumulative chromosome lengths
  const uint8_t* __restrict__ excl;
  int n_chrom;
  const int64_t* __restrict__ rptr;   // regions of chromosome c: [rptr[c], rptr[c + 1])
  const uint64_t* __restrict__ rs;    // start (0-based, chromosome coordinates)
  const uint64_t* __restrict__ re;    // end (exclusive)
  const uint64_t* __restrict__ rmax;  // running max of re within the chromosome
  const uint32_t* __restrict__ rid;   // feature index
};

struct RFilter {
  int strategy;
  int64_t min_len, max_len;
};

struct Index {
  const int32_t* __restrict__ first;  // first region starting at or after base b << shift; nullptr: no index
  int shift;
};

// The chromosome of the last fragment a thread looked up (sorted fragments
// stay on it), with its regions.
struct Chrom {
  uint64_t start = 1, end = 0;  // empty
  int64_t lo = 0, hi = 0;
  bool skip = false;
};

// regions overlapping [qs, qe) of the chromosome; `skip` drops those that
// also contain the point skip_at (the paired-insertion union)
template <class F>
__device__ __forceinline__ void visit(const RegionSet& R, const Index& ix, const Chrom& ch, uint64_t qs, uint64_t qe,
                                      bool skip, uint64_t skip_at, F&& f) {
  int64_t a = ch.lo, b = ch.hi;  // first region with start >= qe
  if (ix.first && qe < ch.end - ch.start) {
    const int64_t k = (int64_t)((ch.start + qe) >> ix.shift);
    a = max(a, (int64_t)__ldg(ix.first + k));
    b = min(b, (int64_t)__ldg(ix.first + k + 1));
  }
  while (a < b) {
    const int64_t m = (a + b) >> 1;
    if (__ldg(R.rs + m) < qe) a = m + 1;
    else b = m;
  }
  for (int64_t j = a - 1; j >= ch.lo; --j) {
    if (__ldg(R.rmax + j) <= qs) break;
    const uint64_t e = __ldg(R.re + j);
    if (e > qs) {
      if (skip && __ldg(R.rs + j) <= skip_at && e > skip_at) continue;
      f(__ldg(R.rid + j));
    }
  }
}

// Hits of one fragment: returns their number (calling f for each), or -1
// when the position lies outside the genome.
template <class F>
__device__ __forceinline__ int fragment_hits(const RegionSet& R, const Index& ix, const RFilter& flt, Chrom& ch,
                                             uint64_t pos, uint32_t len, F&& f) {
  if (pos < ch.start || pos >= ch.end) {
    int a = 0, b = R.n_chrom;  // first chromosome with end > pos
    while (a < b) {
      const int m = (a + b) >> 1;
      if (__ldg(R.chrom_end + m) <= pos) a = m + 1;
      else b = m;
    }
    if (a >= R.n_chrom) return -1;
    ch.start = a ? __ldg(R.chrom_end + a - 1) : 0ull;
    ch.end = __ldg(R.chrom_end + a);
    ch.lo = __ldg(R.rptr + a);
    ch.hi = __ldg(R.rptr + a + 1);
    ch.skip = __ldg(R.excl + a) != 0;
  }
  if (ch.skip) return 0;
  const uint64_t s = pos - ch.start;
  int n = 0;
  auto g = [&](uint32_t k) {
    ++n;
    f(k);
  };
  if (flt.strategy == SG_COUNT_SINGLE) {
    visit(R, ix, ch, s, s + 1, false, 0, g);
    return n;
  }
  const uint64_t size = len;
  if (flt.min_len >= 0 && size < (uint64_t)flt.min_len) return 0;
  if (flt.max_len >= 0 && size > (uint64_t)flt.max_len) return 0;
  const uint64_t e = s + size, e1 = e - 1ull;  // wraps like the reference's u64
  switch (flt.strategy) {
    case SG_COUNT_FRAGMENT: visit(R, ix, ch, s, e, false, 0, g); break;
    case SG_COUNT_INSERTION:
      visit(R, ix, ch, s, s + 1, false, 0, g);
      visit(R, ix, ch, e1, e1 + 1, false, 0, g);
      break;
    default:  // paired-insertion: each region hit by either insertion once
      visit(R, ix, ch, s, s + 1, false, 0, g);
      visit(R, ix, ch, e1, e1 + 1, true, s, g);
      break;
  }
  return n;
}

// ---- the bucket index --------------------------------------------------------
// genome coordinate of each region's start (at most its chromosome's end, so
// that the coordinates ascend)
__global__ void region_gstart(int64_t n_regions, int n_chrom, const uint64_t* __restrict__ chrom_end,
                              const int64_t* __restrict__ rptr, const uint64_t* __restrict__ rs,
                              uint64_t* __restrict__ gstart) {
  const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (j >= n_regions) return;
  int a = 0, b = n_chrom - 1;  // last chromosome whose regions start at or before j and end after it
  while (a < b) {
    const int m = (a + b) >> 1;
    if (rptr[m + 1] <= j) a = m + 1;
    else b = m;
  }
  const uint64_t c0 = a ? chrom_end[a - 1] : 0ull, c1 = chrom_end[a], s = rs[j];
  gstart[j] = s < c1 - c0 ? c0 + s : c1;
}

__global__ void region_buckets(int64_t n_regions, const uint64_t* __restrict__ gstart, int64_t n_buckets, int shift,
                               int32_t* __restrict__ first) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= n_buckets) return;
  const uint64_t x = (uint64_t)k << shift;
  int64_t a = 0, b = n_regions;
  while (a < b) {
    const int64_t m = (a + b) >> 1;
    if (gstart[m] < x) a = m + 1;
    else b = m;
  }
  first[k] = (int32_t)a;
}

// About four buckets per region, and at least 4,096: a bucket then holds a
// region or none, and at 200,000 regions the index is 3 MB (it stays in L2).
int index_shift(uint64_t genome, int64_t n_regions) {
  const uint64_t most = 4 * (uint64_t)std::max<int64_t>(n_regions, 1024);
  int shift = 0;
  while ((genome >> shift) > most) ++shift;
  return shift;
}

__global__ void __launch_bounds__(kPlanBlock)
region_plan_kernel(const int64_t* __restrict__ cell_ptr, int64_t n_cells, int64_t n_frags,
                   const uint64_t* __restrict__ pos, const uint32_t* __restrict__ len, RegionSet R, Index ix,
                   RFilter flt, uint32_t* __restrict__ mask, int64_t* __restrict__ key_ptr, int* status,
                   unsigned long long* bad) {
  __shared__ long long ws[kPlanBlock / 32];
  const int64_t c = blockIdx.x;
  if (c >= n_cells) return;
  int64_t a = cell_ptr[c], b = cell_ptr[c + 1];
  if (a < 0 || b < a || b > n_frags) {  // malformed row pointer: no access
    if (threadIdx.x == 0) report_error(status, nullptr, SG_ERR_ARG, 0);
    a = b = 0;
  }
  long long cnt = 0;
  Chrom ch;
  for (int64_t w0 = a & ~31LL; w0 < b; w0 += kPlanBlock) {  // warps aligned to the words of the mask
    const int64_t k = w0 + threadIdx.x;
    int r = 0;
    if (k >= a && k < b) {
      r = fragment_hits(R, ix, flt, ch, __ldg(pos + k), len ? __ldg(len + k) : 0u, [](uint32_t) {});
      if (r < 0) report_error(status, bad, SG_ERR_RANGE, (unsigned long long)k);
      else cnt += r;
    }
    if (mask) {
      const unsigned m = __ballot_sync(0xffffffffu, r > 0);
      if (m && (threadIdx.x & 31) == 0) atomicOr(mask + (k >> 5), m);  // a word may span two cells
    }
  }
  cnt = block_sum_ll<kPlanBlock>(cnt, ws);
  if (threadIdx.x == 0) {
    key_ptr[c + 1] = cnt;
    if (c == 0) key_ptr[0] = 0;
  }
}

struct RunSmem {
  SortSmem<kRunBlock> sort;
  unsigned kmin_ws[kRunBlock / 32];
  int scan_ws[kRunBlock / 32 + 1];
  int fill;
  int left[kRunBlock];  // cells of this CTA's stride that region_short_kernel left
  int n_left;
};

struct RunArgs {
  const int64_t* __restrict__ cell_ptr;
  int64_t n_cells, n_frags;
  const uint64_t* __restrict__ pos;
  const uint32_t* __restrict__ len;
  const uint32_t* __restrict__ mask;  // fragments with hits; nullptr: not known
  const int64_t* __restrict__ key_ptr;
  int64_t key_cap;
  uint32_t* __restrict__ gkeys;
  uint32_t* __restrict__ gtmp;
  int32_t* __restrict__ pair_idx;
  uint32_t* __restrict__ pair_cnt;
  int64_t* __restrict__ cell_nnz;
  int* status;
};

// One cell by the whole CTA; rows of more than smem_keys keys use global
// scratch, or (global == false) are left alone with cell_nnz = -1.
__device__ void region_cell(const RunArgs& A_, const RegionSet& R, const Index& ix, const RFilter& flt, int64_t c,
                            RunSmem& sm, uint32_t* skeys, int smem_keys, bool global) {
  const int64_t* __restrict__ cell_ptr = A_.cell_ptr;
  const int64_t* __restrict__ key_ptr = A_.key_ptr;
  const int64_t n_frags = A_.n_frags, key_cap = A_.key_cap;
  const uint64_t* __restrict__ pos = A_.pos;
  const uint32_t* __restrict__ len = A_.len;
  int64_t* __restrict__ cell_nnz = A_.cell_nnz;
  int* status = A_.status;
  const int tid = threadIdx.x;
  const int64_t kbase = key_ptr[c];
  const int64_t K64 = key_ptr[c + 1] - kbase;
  const int64_t fa = cell_ptr[c], fb = cell_ptr[c + 1];
  if (K64 <= 0 || kbase < 0 || kbase + K64 > key_cap || K64 > 0x7fffffffLL || fa < 0 || fb < fa ||
      fb > n_frags) {
    if (tid == 0) {
      cell_nnz[c + 1] = 0;
      if (K64 != 0) report_error(status, nullptr, K64 < 0 ? SG_ERR_ARG : SG_ERR_CAP, 0);
    }
    return;
  }
  const int K = (int)K64;
  const bool in_smem = K <= smem_keys;
  if (!in_smem && !global) {
    if (tid == 0) cell_nnz[c + 1] = -1;
    return;
  }
  uint32_t* A = in_smem ? skeys : A_.gkeys + kbase;
  uint32_t* B = in_smem ? skeys + smem_keys : A_.gtmp + kbase;

  // 1. the cell's region hits (order is irrelevant before sorting)
  if (tid == 0) sm.fill = 0;
  __syncthreads();
  unsigned kmin = 0xffffffffu, kmax = 0u;
  Chrom ch;
  auto collect = [&](int64_t k) {
    fragment_hits(R, ix, flt, ch, __ldg(pos + k), len ? __ldg(len + k) : 0u, [&](uint32_t key) {
      const int o = atomicAdd(&sm.fill, 1);
      if (o < K) A[o] = key;
      kmin = min(kmin, key);
      kmax = max(kmax, key);
    });
  };
  if (A_.mask) {  // thread per word of the mask
    for (int64_t w = (fa >> 5) + tid; w * 32 < fb; w += kRunBlock) {
      uint32_t m = A_.mask[w];
      if (w * 32 < fa) m &= ~0u << (fa & 31);
      if (w * 32 + 32 > fb) m &= (1u << (fb & 31)) - 1u;  // fb & 31 > 0 here
      for (; m; m &= m - 1) collect(w * 32 + __ffs(m) - 1);
    }
  } else {
    for (int64_t k = fa + tid; k < fb; k += kRunBlock) collect(k);
  }
  __syncthreads();
  if (sm.fill != K) {  // plan and run disagree: inputs changed in between
    if (tid == 0) {
      cell_nnz[c + 1] = 0;
      report_error(status, nullptr, SG_ERR_ARG, 0);
    }
    return;
  }
  kmin = block_min_u32<kRunBlock>(kmin, sm.kmin_ws);
  kmax = block_max_u32<kRunBlock>(kmax, sm.kmin_ws);
  const unsigned span = kmax - kmin;
  const int nbits = span ? 32 - __clz(span) : 0;

  // 2. sort, 3. run-length encode: H[u] = start of the u-th distinct region
  uint32_t* S = cta_radix_sort<kRunBlock>(A, B, K, kmin, nbits, sm.sort);
  uint32_t* H = (S == A) ? B : A;
  int U = 0;
  for (int base = 0; base < K; base += kRunBlock) {
    const int i = base + tid;
    int head = 0;
    if (i < K) head = (i == 0) || (S[i] != S[i - 1]);
    int tot;
    const int p = block_exscan<kRunBlock>(head, sm.scan_ws, tot);
    if (head) H[U + p] = (uint32_t)i;
    U += tot;
  }
  __syncthreads();
  int32_t* pi = A_.pair_idx + kbase;
  uint32_t* pc = A_.pair_cnt + kbase;
  for (int u = tid; u < U; u += kRunBlock) {
    const uint32_t s0 = H[u];
    const uint32_t s1 = (u + 1 < U) ? H[u + 1] : (uint32_t)K;
    pi[u] = (int32_t)S[s0];
    pc[u] = s1 - s0;
  }
  if (tid == 0) cell_nnz[c + 1] = U;
}

// Rows of up to kShortKeys keys, one CTA per cell in 52 KB of shared memory.
__global__ void __launch_bounds__(kRunBlock) region_short_kernel(RunArgs a, RegionSet R, Index ix, RFilter flt) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  RunSmem& sm = *reinterpret_cast<RunSmem*>(smem_raw);
  region_cell(a, R, ix, flt, blockIdx.x, sm, reinterpret_cast<uint32_t*>(smem_raw + sizeof(RunSmem)), kShortKeys,
              false);
}

// The longer rows, on a grid of one CTA per SM: when there are none the launch
// ends after one look at the flags.
__global__ void __launch_bounds__(kRunBlock) region_long_kernel(RunArgs a, RegionSet R, Index ix, RFilter flt) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  RunSmem& sm = *reinterpret_cast<RunSmem*>(smem_raw);
  uint32_t* skeys = reinterpret_cast<uint32_t*>(smem_raw + sizeof(RunSmem));
  for (int64_t c0 = blockIdx.x; c0 < a.n_cells; c0 += (int64_t)gridDim.x * kRunBlock) {
    if (threadIdx.x == 0) sm.n_left = 0;
    __syncthreads();
    const int64_t mine = c0 + (int64_t)threadIdx.x * gridDim.x;
    if (mine < a.n_cells && a.cell_nnz[mine + 1] < 0) sm.left[atomicAdd(&sm.n_left, 1)] = threadIdx.x;
    __syncthreads();
    const int n = sm.n_left;
    for (int i = 0; i < n; ++i) {
      region_cell(a, R, ix, flt, c0 + (int64_t)sm.left[i] * gridDim.x, sm, skeys, kSmemKeys, true);
      __syncthreads();
    }
  }
}

__global__ void zero_first_r(int64_t* p) { p[0] = 0; }

int check_region_args(int64_t n_cells, int n_chrom, int strategy, int64_t n_features) {
  if (n_cells < 0 || n_cells > 0x7fffffffLL || n_chrom <= 0) return SG_ERR_ARG;
  if (strategy < SG_COUNT_INSERTION || strategy > SG_COUNT_SINGLE) return SG_ERR_ARG;
  if (n_features < 0 || n_features > 0x7fffffffLL) return SG_ERR_ARG;
  return SG_OK;
}

}  // namespace
}  // namespace sg

using namespace sg;

extern "C" int sg_region_index_shift(uint64_t genome, int64_t n_regions) {
  return genome >= (1ull << 62) || n_regions < 0 ? -1 : index_shift(genome, n_regions);
}

extern "C" int64_t sg_region_index_bytes(uint64_t genome, int64_t n_regions) {
  const int shift = sg_region_index_shift(genome, n_regions);
  if (shift < 0) return -1;
  return 8 * n_regions + 4 * (int64_t)((genome >> shift) + 2);
}

extern "C" int sg_region_index(uint64_t genome, const uint64_t* chrom_end, int n_chrom, const int64_t* region_ptr,
                               const uint64_t* region_start, int64_t n_regions, void* index, int64_t index_bytes,
                               void* stream) {
  const int64_t need = sg_region_index_bytes(genome, n_regions);
  if (need < 0 || n_chrom <= 0 || n_regions > 0x7fffffffLL || ((uintptr_t)index & 7u)) return SG_ERR_ARG;
  if (!index || index_bytes < need) return SG_ERR_CAP;
  cudaStream_t s = as_stream(stream);
  const int shift = index_shift(genome, n_regions);
  uint64_t* gstart = reinterpret_cast<uint64_t*>(index);
  int32_t* first = reinterpret_cast<int32_t*>(gstart + n_regions);
  const int64_t nb = (int64_t)(genome >> shift) + 2;
  if (n_regions > 0)
    region_gstart<<<(unsigned)((n_regions + 255) / 256), 256, 0, s>>>(n_regions, n_chrom, chrom_end, region_ptr,
                                                                      region_start, gstart);
  region_buckets<<<(unsigned)((nb + 255) / 256), 256, 0, s>>>(n_regions, gstart, nb, shift, first);
  SG_CHECK_LAUNCH();
  return SG_OK;
}

// the table of an index built by sg_region_index (nullptr: none)
static Index index_of(const void* index, uint64_t genome, int64_t n_regions) {
  if (!index) return {nullptr, 0};
  return {reinterpret_cast<const int32_t*>(reinterpret_cast<const uint64_t*>(index) + n_regions),
          index_shift(genome, n_regions)};
}

extern "C" int sg_region_plan(const int64_t* cell_ptr, int64_t n_cells, int64_t n_frags, const uint64_t* frag_pos,
                              const uint32_t* frag_len, const uint64_t* chrom_end, const uint8_t* chrom_excl,
                              int n_chrom, const int64_t* region_ptr, const uint64_t* region_start,
                              const uint64_t* region_end, const uint64_t* region_maxend, const uint32_t* region_id,
                              int64_t n_features, int strategy, int64_t min_len, int64_t max_len, int64_t* key_ptr,
                              void* scan_scratch, int* status, unsigned long long* bad, void* stream) {
  return sg_region_plan_indexed(cell_ptr, n_cells, n_frags, frag_pos, frag_len, chrom_end, chrom_excl, n_chrom,
                                region_ptr, region_start, region_end, region_maxend, region_id, n_features, strategy,
                                min_len, max_len, nullptr, 0, 0, nullptr, key_ptr, scan_scratch, status, bad, stream);
}

extern "C" int sg_region_plan_indexed(const int64_t* cell_ptr, int64_t n_cells, int64_t n_frags, const uint64_t* frag_pos,
                              const uint32_t* frag_len, const uint64_t* chrom_end, const uint8_t* chrom_excl,
                              int n_chrom, const int64_t* region_ptr, const uint64_t* region_start,
                              const uint64_t* region_end, const uint64_t* region_maxend, const uint32_t* region_id,
                              int64_t n_features, int strategy, int64_t min_len, int64_t max_len,
                                      const void* index, uint64_t genome, int64_t n_regions, uint32_t* frag_mask,
                                      int64_t* key_ptr, void* scan_scratch, int* status, unsigned long long* bad,
                                      void* stream) {
  const int e = check_region_args(n_cells, n_chrom, strategy, n_features);
  if (e) return e;
  if (strategy != SG_COUNT_SINGLE && !frag_len && n_frags > 0) return SG_ERR_ARG;
  cudaStream_t s = as_stream(stream);
  if (n_cells == 0) {
    zero_first_r<<<1, 1, 0, s>>>(key_ptr);
    SG_CHECK_LAUNCH();
    return SG_OK;
  }
  RegionSet R{chrom_end, chrom_excl, n_chrom, region_ptr, region_start, region_end, region_maxend, region_id};
  RFilter f{strategy, min_len, max_len};
  if (frag_mask && cudaMemsetAsync(frag_mask, 0, (size_t)((n_frags + 31) / 32) * 4, s) != cudaSuccess)
    return SG_ERR_CUDA;
  region_plan_kernel<<<(unsigned)n_cells, kPlanBlock, 0, s>>>(
      cell_ptr, n_cells, n_frags, frag_pos, strategy == SG_COUNT_SINGLE ? nullptr : frag_len, R,
      index_of(index, genome, n_regions), f, frag_mask, key_ptr, status, bad);
  SG_CHECK_LAUNCH();
  if (inclusive_scan_i64(key_ptr + 1, n_cells, scan_scratch, s) != cudaSuccess) return SG_ERR_CUDA;
  return SG_OK;
}

extern "C" int sg_region_run(const int64_t* cell_ptr, int64_t n_cells, int64_t n_frags, const uint64_t* frag_pos,
                             const uint32_t* frag_len, const uint64_t* chrom_end, const uint8_t* chrom_excl,
                             int n_chrom, const int64_t* region_ptr, const uint64_t* region_start,
                             const uint64_t* region_end, const uint64_t* region_maxend, const uint32_t* region_id,
                             int64_t n_features, int strategy, int64_t min_len, int64_t max_len,
                             const int64_t* key_ptr, void* scratch, int64_t scratch_bytes, int64_t* out_indptr,
                             void* scan_scratch, int* status, unsigned long long* bad, void* stream) {
  return sg_region_run_indexed(cell_ptr, n_cells, n_frags, frag_pos, frag_len, chrom_end, chrom_excl, n_chrom,
                               region_ptr, region_start, region_end, region_maxend, region_id, n_features, strategy,
                               min_len, max_len, nullptr, 0, 0, nullptr, key_ptr, scratch, scratch_bytes, out_indptr,
                               scan_scratch, status, bad, stream);
}

extern "C" int sg_region_run_indexed(const int64_t* cell_ptr, int64_t n_cells, int64_t n_frags, const uint64_t* frag_pos,
                             const uint32_t* frag_len, const uint64_t* chrom_end, const uint8_t* chrom_excl,
                             int n_chrom, const int64_t* region_ptr, const uint64_t* region_start,
                             const uint64_t* region_end, const uint64_t* region_maxend, const uint32_t* region_id,
                             int64_t n_features, int strategy, int64_t min_len, int64_t max_len,
                             const void* index, uint64_t genome, int64_t n_regions,
                             const uint32_t* frag_mask, const int64_t* key_ptr, void* scratch, int64_t scratch_bytes, int64_t* out_indptr,
                             void* scan_scratch, int* status, unsigned long long* bad, void* stream) {
  (void)bad;
  const int e = check_region_args(n_cells, n_chrom, strategy, n_features);
  if (e) return e;
  if (strategy != SG_COUNT_SINGLE && !frag_len && n_frags > 0) return SG_ERR_ARG;
  if (((uintptr_t)scratch & 15u) != 0) return SG_ERR_ARG;
  cudaStream_t s = as_stream(stream);
  if (n_cells == 0) {
    zero_first_r<<<1, 1, 0, s>>>(out_indptr);
    SG_CHECK_LAUNCH();
    return SG_OK;
  }
  // same sub-buffer split as sg_tile_run, so that sg_tile_emit reads the pairs
  const int64_t k4 = (scratch_bytes - 16) / (4 * (int64_t)sizeof(uint32_t));
  if (k4 < 0) return SG_ERR_CAP;
  uint32_t* base = reinterpret_cast<uint32_t*>(scratch);
  RegionSet R{chrom_end, chrom_excl, n_chrom, region_ptr, region_start, region_end, region_maxend, region_id};
  RFilter f{strategy, min_len, max_len};
  const size_t smem_short = sizeof(RunSmem) + 2 * (size_t)kShortKeys * sizeof(uint32_t);
  const size_t smem_long = sizeof(RunSmem) + 2 * (size_t)kSmemKeys * sizeof(uint32_t);
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (sms < 1 ||
      cudaFuncSetAttribute(region_short_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_short) !=
          cudaSuccess ||
      cudaFuncSetAttribute(region_long_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_long) !=
          cudaSuccess)
    return SG_ERR_CUDA;
  const Index ix = index_of(index, genome, n_regions);
  const RunArgs a{cell_ptr, n_cells, n_frags, frag_pos, strategy == SG_COUNT_SINGLE ? nullptr : frag_len, frag_mask,
                  key_ptr, k4, base, base + k4, reinterpret_cast<int32_t*>(base + 2 * k4), base + 3 * k4, out_indptr,
                  status};
  if (cudaMemsetAsync(out_indptr, 0, sizeof(int64_t), s) != cudaSuccess) return SG_ERR_CUDA;
  region_short_kernel<<<(unsigned)n_cells, kRunBlock, smem_short, s>>>(a, R, ix, f);
  SG_CHECK_LAUNCH();
  region_long_kernel<<<(unsigned)std::min<int64_t>(n_cells, sms), kRunBlock, smem_long, s>>>(a, R, ix, f);
  SG_CHECK_LAUNCH();
  if (inclusive_scan_i64(out_indptr + 1, n_cells, scan_scratch, s) != cudaSuccess) return SG_ERR_CUDA;
  return SG_OK;
}
