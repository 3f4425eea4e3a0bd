// Tile binning: fragments -> cell x tile count CSR, bit-exact with the
// reference's gen_mat_pair / gen_mat_single
// (snapatac2-core/src/feature_count/data_iter.rs:313-415).
//
// Design (one CTA per cell):
//   bound: key_ptr from the row pointers alone, two tile hits ("keys") per
//          fragment at most (one for single-end reads): no fragment is read.
//   plan : for the fragment strategy, whose hits per fragment are unbounded,
//          the exact number of keys per cell, prefix-summed into key_ptr.
//   run  : every fragment is located on the genome (binary search of the
//          cumulative chromosome lengths, genome.rs:419-434), filtered
//          (excluded chromosome, size bounds) and checked (end past the
//          chromosome -> SG_ERR_RANGE, the reference's panic in
//          get_position_rev, genome.rs:397-399).  A cell whose fragments are sorted by start (how import_fragments
//          and the reference store them) is counted without a sort
//          (stream_kernel below); any other cell has its keys
//          gathered in shared memory (global scratch above kSmemKeys),
//          sorted with a stable LSD radix sort over the bits they span and
//          run-length encoded into (tile, count) pairs (sort_kernel).  The
//          per-cell unique counts are prefix-summed into out_indptr.
//   emit : pairs are compacted from the key_ptr layout into the CSR arrays.
// The BTreeMap of the reference yields tiles in increasing order with their
// hit counts; both forms yield exactly the same rows.
#include <algorithm>

#include "common.cuh"
#include "internal.h"

namespace sg {
namespace {

constexpr int kPlanBlock = 256;
constexpr int kRunBlock = 512;
constexpr int kSmemKeys = 24576;  // keys per cell sorted in shared memory

struct Genome {
  const uint64_t* __restrict__ end;  // cumulative base lengths
  const uint64_t* __restrict__ bin_off;
  const uint8_t* __restrict__ excl;
  int n;
  uint32_t bin;
  uint64_t magic;  // floor(2^64 / bin) + 1 (bin > 1)

  // x / bin for 32-bit x: the high word of magic * x (Lemire, Kaser and Kurz,
  // "Faster remainder by direct computation", 2019)
  __device__ __forceinline__ uint32_t div(uint32_t x) const {
    return bin == 1 ? x : (uint32_t)__umul64hi(magic, x);
  }
};

Genome make_genome(const uint64_t* end, const uint64_t* off, const uint8_t* excl, int n, uint32_t bin) {
  return {end, off, excl, n, bin, bin > 1 ? ~0ull / bin + 1 : 0ull};
}

// The chromosome of the last fragment a thread looked up: fragments arrive
// sorted, so the next one is nearly always on the same chromosome and the
// binary search (five dependent loads at 24 chromosomes) is left out.
struct Chrom {
  uint64_t start = 1, end = 0, off = 0;  // empty
  bool skip = false;
};

struct Filter {
  int strategy;
  int64_t min_len, max_len;
};

// Fragment -> [lo, hi] tile range plus the number of keys it emits.
// Returns 0 (skipped), the key count, or -1 on a range error.
__device__ __forceinline__ int frag_keys(const Genome& g, const Filter& f, Chrom& ch, uint64_t pos, uint32_t len,
                                         uint32_t& lo, uint32_t& hi) {
  if (pos < ch.start || pos >= ch.end) {
    int a = 0, b = g.n;  // first chromosome with end > pos
    while (a < b) {
      int m = (a + b) >> 1;
      if (__ldg(g.end + m) <= pos) a = m + 1; else b = m;
    }
    if (a >= g.n) return -1;
    ch.start = a ? __ldg(g.end + a - 1) : 0ull;
    ch.end = __ldg(g.end + a);
    ch.off = __ldg(g.bin_off + a);
    ch.skip = __ldg(g.excl + a) != 0;
  }
  if (ch.skip) return 0;
  const uint64_t start = pos - ch.start;
  if (f.strategy == SG_COUNT_SINGLE) {
    lo = hi = (uint32_t)ch.off + g.div((uint32_t)start);
    return 1;
  }
  const uint64_t fs = len;
  const uint64_t end = start + fs - 1ull;  // wraps like the reference's u64
  if (f.min_len >= 0 && fs < (uint64_t)f.min_len) return 0;
  if (f.max_len >= 0 && fs > (uint64_t)f.max_len) return 0;
  if (end >= ch.end - ch.start) return -1;
  lo = (uint32_t)ch.off + g.div((uint32_t)start);
  hi = (uint32_t)ch.off + g.div((uint32_t)end);
  switch (f.strategy) {
    case SG_COUNT_INSERTION: return 2;
    case SG_COUNT_PIC: return hi != lo ? 2 : 1;
    default: return hi >= lo ? (int)(hi - lo + 1u) : 0;  // fragment
  }
}

__global__ void __launch_bounds__(kPlanBlock)
plan_kernel(const int64_t* __restrict__ cell_ptr, int64_t n_cells, int64_t n_frags,
            const uint64_t* __restrict__ pos, const uint32_t* __restrict__ len, Genome g, Filter f,
            int64_t* __restrict__ key_ptr, int* status, unsigned long long* bad) {
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
  for (int64_t k0 = a + threadIdx.x; k0 < b; k0 += 4 * kPlanBlock) {  // four loads in flight
    uint64_t p[4];
    uint32_t l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int64_t k = k0 + i * kPlanBlock;
      p[i] = k < b ? __ldg(pos + k) : 0ull;
      l[i] = k < b ? __ldg(len + k) : 0u;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int64_t k = k0 + i * kPlanBlock;
      if (k >= b) break;
      uint32_t lo, hi;
      const int r = frag_keys(g, f, ch, p[i], l[i], lo, hi);
      if (r < 0) report_error(status, bad, SG_ERR_RANGE, (unsigned long long)k);
      else cnt += r;
    }
  }
  cnt = block_sum_ll<kPlanBlock>(cnt, ws);
  if (threadIdx.x == 0) {
    key_ptr[c + 1] = cnt;
    if (c == 0) key_ptr[0] = 0;
  }
}

// key_ptr of a bound: rate keys per fragment
__global__ void bound_kernel(int64_t n_cells, const int64_t* __restrict__ cell_ptr, int64_t rate,
                             int64_t* __restrict__ key_ptr) {
  const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c <= n_cells) key_ptr[c] = rate * (cell_ptr[c] - cell_ptr[0]);
}

// a row's key and fragment ranges lie inside their arrays (false for an empty row too)
__device__ __forceinline__ bool row_ok(int64_t K, int64_t kbase, int64_t key_cap, int64_t fa, int64_t fb,
                                       int64_t n_frags) {
  return K > 0 && kbase >= 0 && kbase + K <= key_cap && K <= 0x7fffffffLL && fa >= 0 && fb >= fa && fb <= n_frags;
}

// ---------------------------------------------------------------------------
// Counting of sorted fragments, one CTA per cell, kChunk fragments at a time.
//
// With starts ascending, the first tiles `lo` ascend too, and the tiles that
// the fragments seen so far can still touch form one open run ending at the
// running maximum of the last tiles.  So every tile of the union of the
// fragments' ranges gets a counter slot in ascending order: with C_k the
// number of tiles covered by fragments 0..k and P_k the running maximum of
// the last tiles, tile t of fragment k has slot C_k - 1 - (P_k - t).  A max
// scan and a sum scan give every slot, the hits are shared-memory atomics,
// and the slots are already in output order.  At the end of a chunk the slots
// below the last fragment's first tile are final and written out; the rest
// (one or two) move to the front.
//
// The radix sort it replaces moved every key through shared memory in three
// passes of six barriers per 512 keys, at one CTA per SM (200 KB), and
// through L2 for the third of the cells above 24,576 keys: 4.87 ms for 5,000
// cells and 6.1e7 fragments, 0.7 ms here (1.0 TB/s of fragments in, at four
// CTAs of 64 registers per SM; instruction issue and barriers bind).  The call
// went from 6.07 to 1.06 ms with the pass that planned it left out (0.53 ms)
// and one read back instead of five.  Cells that break
// the assumptions (unsorted or zero-length fragments, or a chunk that covers
// more tiles than there are slots) are left to sort_kernel: cell_nnz = -1.
// ---------------------------------------------------------------------------
constexpr int kStreamThreads = 256;
constexpr int kItems = 4;
constexpr int kChunk = kStreamThreads * kItems;
constexpr int kSlots = 4096;  // 32 KB of counters and tile ids
constexpr int kStreamWarps = kStreamThreads / 32;

// *flag = 1 unless the tile indices ascend with the chromosomes (0 else); one
// CTA.  Looked at once per call: with every cell's CTA reading the whole table
// for itself a call over 3,000 cells of 500 fragments on 100,000 contigs took
// 746 us, now 468 (24 chromosomes, 5,000 cells: 1,094 -> 1,042).
__global__ void __launch_bounds__(1024) layout_kernel(Genome g, int64_t* __restrict__ flag) {
  bool odd = false;
  for (int i = 1 + threadIdx.x; i < g.n; i += 1024) {
    const uint64_t n0 = __ldg(g.end + i - 1) - (i > 1 ? __ldg(g.end + i - 2) : 0ull);
    const uint64_t w = __ldg(g.excl + i - 1) || n0 == 0 ? 0ull : g.div((uint32_t)(n0 - 1));
    odd |= __ldg(g.bin_off + i) < __ldg(g.bin_off + i - 1) + w;
  }
  odd = __syncthreads_or(odd);
  if (threadIdx.x == 0) *flag = odd;
}

__global__ void __launch_bounds__(kStreamThreads)
stream_kernel(const int64_t* __restrict__ cell_ptr, int64_t n_cells, int64_t n_frags,
              const uint64_t* __restrict__ pos, const uint32_t* __restrict__ len, Genome g, Filter f,
              const int64_t* __restrict__ key_ptr, int64_t key_cap, int32_t* __restrict__ pair_idx,
              uint32_t* __restrict__ pair_cnt, int64_t* __restrict__ cell_nnz, int* status,
              unsigned long long* bad) {
  __shared__ uint32_t cnt[kSlots], tile[kSlots];
  __shared__ uint32_t ws_max[kStreamWarps], ws_lo[kStreamWarps], ws_sum[kStreamWarps], ws_out[kStreamWarps];
  const int64_t c = blockIdx.x;
  if (c >= n_cells) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t kbase = key_ptr[c];
  const int64_t K = key_ptr[c + 1] - kbase;
  const int64_t fa = cell_ptr[c], fb = cell_ptr[c + 1];
  if (!row_ok(K, kbase, key_cap, fa, fb, n_frags)) {
    if (tid == 0) {
      cell_nnz[c + 1] = 0;
      if (fa < 0 || fb < fa || fb > n_frags || K < 0) report_error(status, nullptr, SG_ERR_ARG, 0);
      else if (K > 0) report_error(status, nullptr, SG_ERR_CAP, 0);
    }
    return;
  }
  for (int i = tid; i < kSlots; i += kStreamThreads) cnt[i] = 0;
  uint32_t pm = 0;    // 1 + largest tile so far
  uint32_t cov = 0;   // slots carried over from the previous chunk
  int64_t U = 0;      // pairs written
  bool odd = cell_nnz[0] != 0;  // layout_kernel; then: a fragment out of order or of zero length
  Chrom ch;
  uint64_t p[kItems];
  uint32_t l[kItems];
  auto load = [&](int64_t base) {
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      const int64_t k = base + kItems * tid + i;
      p[i] = k < fb ? __ldg(pos + k) : 0ull;
      l[i] = k < fb ? __ldg(len + k) : 0u;
    }
  };
  load(fa);
  for (int64_t base = fa; base < fb; base += kChunk) {
    uint32_t lo[kItems], hi[kItems];
    int r[kItems];
    uint32_t b1 = 0, l1 = 0;  // 1 + largest last / first tile of this thread's fragments
    const int64_t k0 = base + kItems * tid;
    uint64_t prev = k0 > fa && k0 < fb ? __ldg(pos + k0 - 1) : 0ull;
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      r[i] = 0;
      if (k0 + i < fb) {
        odd |= p[i] < prev;
        prev = p[i];
        r[i] = frag_keys(g, f, ch, p[i], l[i], lo[i], hi[i]);
        if (r[i] < 0) report_error(status, bad, SG_ERR_RANGE, (unsigned long long)(k0 + i));
        if (r[i] > 0) {
          odd |= hi[i] < lo[i];
          b1 = max(b1, hi[i] + 1);
          l1 = max(l1, lo[i] + 1);
        }
      }
    }
    if (base + kChunk < fb) load(base + kChunk);  // in flight during the scans
    // running maximum of the last tiles over the threads before this one
    uint32_t x = b1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x = max(x, y);
    }
    const uint32_t wl = __reduce_max_sync(0xffffffffu, l1);
    if (lane == 31) {
      ws_max[warp] = x;
      ws_lo[warp] = wl;
    }
    uint32_t run = __shfl_up_sync(0xffffffffu, x, 1);
    if (lane == 0) run = 0;
    __syncthreads();
    uint32_t last1 = 0, pm_new = pm;
    run = max(run, pm);
#pragma unroll
    for (int w = 0; w < kStreamWarps; ++w) {
      if (w < warp) run = max(run, ws_max[w]);
      pm_new = max(pm_new, ws_max[w]);
      last1 = max(last1, ws_lo[w]);
    }
    // tiles that each fragment adds to the union (saturated: more than kSlots never fits)
    uint32_t add[kItems], q = run, mine = 0;
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      add[i] = 0;
      if (r[i] > 0) {
        if (hi[i] + 1 > q) add[i] = min(hi[i] + 1 - max(q, lo[i]), (uint32_t)kSlots + 1);
        q = max(q, hi[i] + 1);
      }
      mine += add[i];
    }
    x = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) ws_sum[warp] = x;
    const bool bail = __syncthreads_or(odd);
    uint32_t C = cov + x - mine, total = cov;
#pragma unroll
    for (int w = 0; w < kStreamWarps; ++w) {
      if (w < warp) C += ws_sum[w];
      total += ws_sum[w];
    }
    const bool end = base + kChunk >= fb;
    // the open run [first tile of the last fragment, running maximum]; a chunk without keys keeps the old one
    const uint32_t open = end ? 0u : (last1 ? pm_new - (last1 - 1) : cov);
    if (bail || total > kSlots || open > kStreamThreads) {  // uniform
      if (tid == 0) cell_nnz[c + 1] = -1;
      return;
    }
    q = run;
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      C += add[i];
      if (r[i] > 0) {
        q = max(q, hi[i] + 1);
        const uint32_t z = C - q;  // slot = z + tile
        if (f.strategy == SG_COUNT_FRAGMENT) {
          for (uint32_t t = lo[i]; t <= hi[i]; ++t) {
            atomicAdd(&cnt[z + t], 1u);
            tile[z + t] = t;
          }
        } else {
          const bool twice = f.strategy == SG_COUNT_INSERTION && lo[i] == hi[i];
          atomicAdd(&cnt[z + lo[i]], twice ? 2u : 1u);
          tile[z + lo[i]] = lo[i];
          if (lo[i] != hi[i]) {
            atomicAdd(&cnt[z + hi[i]], 1u);
            tile[z + hi[i]] = hi[i];
          }
        }
      }
    }
    __syncthreads();
    // write the final slots [0, E), a contiguous share per warp
    const int E = (int)(total - open);
    const int share = ((E + kStreamWarps - 1) / kStreamWarps + 31) & ~31;
    const int s0 = warp * share, s1 = min(s0 + share, E);
    int n = 0;
    for (int i = s0 + lane; i - lane < s1; i += 32) n += __popc(__ballot_sync(0xffffffffu, i < s1 && cnt[i] != 0));
    if (lane == 0) ws_out[warp] = n;
    uint32_t oc = 0, ot = 0;
    if (tid < (int)open) {
      oc = cnt[E + tid];
      ot = tile[E + tid];
    }
    __syncthreads();
    int64_t o = U;
#pragma unroll
    for (int w = 0; w < kStreamWarps; ++w) {
      if (w < warp) o += ws_out[w];
      U += ws_out[w];
    }
    if (U > K) {  // plan and run disagree: inputs changed in between
      if (tid == 0) {
        cell_nnz[c + 1] = 0;
        report_error(status, nullptr, SG_ERR_ARG, 0);
      }
      return;
    }
    for (int i = s0 + lane; i - lane < s1; i += 32) {
      const uint32_t v = i < s1 ? cnt[i] : 0u;
      const unsigned m = __ballot_sync(0xffffffffu, v != 0);
      if (v) {
        const int64_t d = kbase + o + __popc(m & lanemask_lt());
        pair_idx[d] = (int32_t)tile[i];
        pair_cnt[d] = v;
        cnt[i] = 0;
      }
      o += __popc(m);
    }
    if (tid < (int)open) cnt[E + tid] = 0;
    __syncthreads();
    if (tid < (int)open) {
      cnt[tid] = oc;
      tile[tid] = ot;
    }
    cov = open;
    pm = pm_new;
  }
  if (tid == 0) cell_nnz[c + 1] = U;
}

struct RunSmem {
  SortSmem<kRunBlock> sort;
  unsigned kmin_ws[kRunBlock / 32];
  int scan_ws[kRunBlock / 32 + 1];
  int fill;
  int left[kRunBlock];  // cells of this CTA's stride that stream_kernel left
  int n_left, first, mine;
};

// One cell by radix sort and run-length encoding, by the whole CTA.
__device__ void sort_cell(int64_t c, RunSmem& sm, uint32_t* skeys, const int64_t* __restrict__ cell_ptr,
                          int64_t n_frags, const uint64_t* __restrict__ pos, const uint32_t* __restrict__ len,
                          const Genome& g, const Filter& f, const int64_t* __restrict__ key_ptr, int64_t key_cap,
                          uint32_t* __restrict__ gkeys, uint32_t* __restrict__ gtmp, int32_t* __restrict__ pair_idx,
                          uint32_t* __restrict__ pair_cnt, int64_t* __restrict__ cell_nnz, int* status,
                          unsigned long long* bad) {
  const int tid = threadIdx.x, lane = tid & 31;
  const int64_t kbase = key_ptr[c];
  const int64_t cap = key_ptr[c + 1] - kbase;  // stream_kernel checked the row
  const int64_t fa = cell_ptr[c], fb = cell_ptr[c + 1];
  const bool in_smem = cap <= kSmemKeys;
  uint32_t* A = in_smem ? skeys : gkeys + kbase;
  uint32_t* B = in_smem ? skeys + kSmemKeys : gtmp + kbase;

  // 1. regenerate the cell's tile hits; order is irrelevant before sorting
  if (tid == 0) sm.fill = 0;
  __syncthreads();
  unsigned kmin = 0xffffffffu, kmax = 0u;
  Chrom ch;
  for (int64_t k0 = fa; k0 < fb; k0 += kRunBlock) {
    const int64_t k = k0 + tid;
    uint32_t lo = 0, hi = 0;
    int r = 0;
    if (k < fb) {
      r = frag_keys(g, f, ch, pos[k], len[k], lo, hi);
      if (r < 0) {
        report_error(status, bad, SG_ERR_RANGE, (unsigned long long)k);
        r = 0;
      }
    }
    // warp-aggregated slot reservation
    int x = r;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    int wbase = 0;
    if (lane == 31) wbase = atomicAdd(&sm.fill, x);
    wbase = __shfl_sync(0xffffffffu, wbase, 31);
    int o = wbase + x - r;
    if (r > 0 && o + r <= cap) {
      if (f.strategy == SG_COUNT_FRAGMENT) {
        for (uint32_t t = lo; t <= hi; ++t) A[o++] = t;
      } else if (f.strategy == SG_COUNT_INSERTION) {
        A[o] = lo;
        A[o + 1] = hi;
      } else {
        A[o] = lo;
        if (r == 2) A[o + 1] = hi;
      }
      // a zero-length fragment has hi = lo - 1 (end = start - 1)
      kmin = min(kmin, min(lo, hi));
      kmax = max(kmax, max(lo, hi));
    }
  }
  __syncthreads();
  const int K = sm.fill;
  if (K > cap || K <= 0) {  // more keys than planned: inputs changed in between
    if (tid == 0) {
      cell_nnz[c + 1] = 0;
      if (K) report_error(status, nullptr, SG_ERR_ARG, 0);
    }
    return;
  }
  kmin = block_min_u32<kRunBlock>(kmin, sm.kmin_ws);
  kmax = block_max_u32<kRunBlock>(kmax, sm.kmin_ws);
  const unsigned span = kmax - kmin;
  const int nbits = span ? 32 - __clz(span) : 0;

  // 2. sort
  uint32_t* S = cta_radix_sort<kRunBlock>(A, B, K, kmin, nbits, sm.sort);
  uint32_t* H = (S == A) ? B : A;  // free buffer: run starts

  // 3. run-length encode: H[u] = start of the u-th distinct tile
  int U = 0;
  for (int base = 0; base < K; base += kRunBlock) {
    const int i = base + tid;
    int head = 0;
    if (i < K) head = (i == 0) || (S[i] != S[i - 1]);
    int tot;
    int p = block_exscan<kRunBlock>(head, sm.scan_ws, tot);
    if (head) H[U + p] = (uint32_t)i;
    U += tot;
  }
  __syncthreads();
  int32_t* pi = pair_idx + kbase;
  uint32_t* pc = pair_cnt + kbase;
  for (int u = tid; u < U; u += kRunBlock) {
    const uint32_t s0 = H[u];
    const uint32_t s1 = (u + 1 < U) ? H[u + 1] : (uint32_t)K;
    pi[u] = (int32_t)S[s0];
    pc[u] = s1 - s0;
  }
  if (tid == 0) cell_nnz[c + 1] = U;
}

// The cells that stream_kernel left (cell_nnz = -1), on a grid of one CTA per
// SM: when there are none the launch ends after one look at the flags.  A CTA
// takes the cells of its stride, then what is left of the others' (a cell is
// taken by changing its flag to -2): with strides alone the longest of the 152
// sums of 13 cells was 1.4 times their mean (2,000 unsorted cells of 12,000
// fragments: a call took 4.04 ms, now 2.79).
__global__ void __launch_bounds__(kRunBlock)
sort_kernel(const int64_t* __restrict__ cell_ptr, int64_t n_cells, int64_t n_frags, const uint64_t* __restrict__ pos,
            const uint32_t* __restrict__ len, Genome g, Filter f, const int64_t* __restrict__ key_ptr,
            int64_t key_cap, uint32_t* __restrict__ gkeys, uint32_t* __restrict__ gtmp,
            int32_t* __restrict__ pair_idx, uint32_t* __restrict__ pair_cnt, int64_t* cell_nnz,
            int* status, unsigned long long* bad) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  RunSmem& sm = *reinterpret_cast<RunSmem*>(smem_raw);
  uint32_t* skeys = reinterpret_cast<uint32_t*>(smem_raw + sizeof(RunSmem));
  if (blockIdx.x == 0 && threadIdx.x == 0) cell_nnz[0] = 0;  // layout_kernel's flag, read by stream_kernel
  auto left = [&](int64_t c) { return *(volatile int64_t*)(cell_nnz + c + 1) == -1; };
  auto take = [&](int64_t c) {  // by the whole CTA
    __syncthreads();
    if (threadIdx.x == 0)
      sm.mine = atomicCAS(reinterpret_cast<unsigned long long*>(cell_nnz + c + 1), (unsigned long long)-1LL,
                          (unsigned long long)-2LL) == (unsigned long long)-1LL;
    __syncthreads();
    if (sm.mine)
      sort_cell(c, sm, skeys, cell_ptr, n_frags, pos, len, g, f, key_ptr, key_cap, gkeys, gtmp, pair_idx, pair_cnt,
                cell_nnz, status, bad);
  };
  bool any = false;
  for (int64_t c0 = blockIdx.x; c0 < n_cells; c0 += (int64_t)gridDim.x * kRunBlock) {
    __syncthreads();
    if (threadIdx.x == 0) sm.n_left = 0;
    __syncthreads();
    const int64_t mine = c0 + (int64_t)threadIdx.x * gridDim.x;
    if (mine < n_cells && left(mine)) sm.left[atomicAdd(&sm.n_left, 1)] = threadIdx.x;
    __syncthreads();
    const int n = sm.n_left;
    any |= n > 0;
    for (int i = 0; i < n; ++i) take(c0 + (int64_t)sm.left[i] * gridDim.x);
  }
  if (!any) return;
  const int64_t from = n_cells * blockIdx.x / gridDim.x;
  for (int64_t k0 = 0; k0 < n_cells;) {  // flags never turn -1 again: every look takes a cell or moves on
    auto cell = [&](int64_t k) { return from + k < n_cells ? from + k : from + k - n_cells; };
    __syncthreads();
    if (threadIdx.x == 0) sm.first = kRunBlock;
    __syncthreads();
    const int64_t k = k0 + threadIdx.x;
    if (k < n_cells && left(cell(k))) atomicMin(&sm.first, (int)threadIdx.x);
    __syncthreads();
    const int at = sm.first;
    if (at < kRunBlock) take(cell(k0 + at));
    k0 += at;
  }
}

__global__ void emit_kernel(int64_t n_cells, const int64_t* __restrict__ key_ptr, int64_t key_cap,
                            const int32_t* __restrict__ pair_idx, const uint32_t* __restrict__ pair_cnt,
                            const int64_t* __restrict__ out_indptr, int32_t* __restrict__ out_idx,
                            uint32_t* __restrict__ out_cnt, int64_t cap, int* status) {
  const int64_t c = blockIdx.x;
  if (c >= n_cells) return;
  const int64_t src = key_ptr[c], dst = out_indptr[c], n = out_indptr[c + 1] - dst;
  if (dst < 0 || n < 0 || dst + n > cap || src < 0 || src + n > key_cap) {
    if (threadIdx.x == 0) report_error(status, nullptr, SG_ERR_CAP, 0);
    return;
  }
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
    out_idx[dst + i] = pair_idx[src + i];
    out_cnt[dst + i] = pair_cnt[src + i];
  }
}

__global__ void zero_first(int64_t* p) { p[0] = 0; }

}  // namespace
}  // namespace sg

using namespace sg;

static int check_common(int64_t n_cells, int n_chrom, uint32_t bin_size, int strategy) {
  if (n_cells < 0 || n_cells > 0x7fffffffLL || n_chrom <= 0 || bin_size == 0) return SG_ERR_ARG;
  if (strategy < SG_COUNT_INSERTION || strategy > SG_COUNT_SINGLE) return SG_ERR_ARG;
  return SG_OK;
}

extern "C" int64_t sg_scan_scratch_bytes(int64_t n) { return sg::scan_scratch_bytes(n); }

extern "C" int64_t sg_tile_scratch_bytes(int64_t total_keys) {
  if (total_keys < 0) return -1;
  // gkeys + gtmp (uint32) + pair_idx (int32) + pair_cnt (uint32) + cell_nnz scan
  // area is separate (out_indptr); 16-byte aligned sub-buffers.
  int64_t k = (total_keys + 3) / 4 * 4;
  return 4 * k * (int64_t)sizeof(uint32_t) + 16;
}

extern "C" int sg_tile_plan(const int64_t* cell_ptr, int64_t n_cells, int64_t n_frags, const uint64_t* frag_pos,
                            const uint32_t* frag_len, const uint64_t* chrom_end, const uint64_t* bin_off,
                            const uint8_t* chrom_excl, int n_chrom, uint32_t bin_size, int strategy,
                            int64_t min_len, int64_t max_len, int64_t* key_ptr, void* scan_scratch,
                            int* status, unsigned long long* bad, void* stream) {
  int e = check_common(n_cells, n_chrom, bin_size, strategy);
  if (e) return e;
  cudaStream_t s = as_stream(stream);
  if (n_cells == 0) {
    zero_first<<<1, 1, 0, s>>>(key_ptr);
    SG_CHECK_LAUNCH();
    return SG_OK;
  }
  const Genome g = make_genome(chrom_end, bin_off, chrom_excl, n_chrom, bin_size);
  Filter f{strategy, min_len, max_len};
  plan_kernel<<<(unsigned)n_cells, kPlanBlock, 0, s>>>(cell_ptr, n_cells, n_frags, frag_pos, frag_len,
                                                       g, f, key_ptr, status, bad);
  SG_CHECK_LAUNCH();
  if (inclusive_scan_i64(key_ptr + 1, n_cells, scan_scratch, s) != cudaSuccess) return SG_ERR_CUDA;
  return SG_OK;
}

extern "C" int sg_tile_bound(const int64_t* cell_ptr, int64_t n_cells, int strategy, int64_t* key_ptr, void* stream) {
  if (n_cells < 0 || n_cells > 0x7fffffffLL || strategy < SG_COUNT_INSERTION || strategy > SG_COUNT_SINGLE ||
      strategy == SG_COUNT_FRAGMENT)
    return SG_ERR_ARG;
  bound_kernel<<<(unsigned)(n_cells / 256 + 1), 256, 0, as_stream(stream)>>>(
      n_cells, cell_ptr, strategy == SG_COUNT_SINGLE ? 1 : 2, key_ptr);
  SG_CHECK_LAUNCH();
  return SG_OK;
}

extern "C" int sg_tile_run(const int64_t* cell_ptr, int64_t n_cells, int64_t n_frags, const uint64_t* frag_pos,
                           const uint32_t* frag_len, const uint64_t* chrom_end, const uint64_t* bin_off,
                           const uint8_t* chrom_excl, int n_chrom, uint32_t bin_size, int strategy,
                           int64_t min_len, int64_t max_len, const int64_t* key_ptr, void* scratch,
                           int64_t scratch_bytes, int64_t* out_indptr, void* scan_scratch, int* status,
                           unsigned long long* bad, void* stream) {
  int e = check_common(n_cells, n_chrom, bin_size, strategy);
  if (e) return e;
  if (((uintptr_t)scratch & 15u) != 0) return SG_ERR_ARG;
  cudaStream_t s = as_stream(stream);
  if (n_cells == 0) {
    zero_first<<<1, 1, 0, s>>>(out_indptr);
    SG_CHECK_LAUNCH();
    return SG_OK;
  }
  // The caller sized scratch from key_ptr[n_cells]; the sub-buffer split uses
  // that same total, recovered from the byte count.
  const int64_t k4 = (scratch_bytes - 16) / (4 * (int64_t)sizeof(uint32_t));
  if (k4 < 0) return SG_ERR_CAP;
  uint32_t* base = reinterpret_cast<uint32_t*>(scratch);
  uint32_t* gkeys = base;
  uint32_t* gtmp = base + k4;
  int32_t* pidx = reinterpret_cast<int32_t*>(base + 2 * k4);
  uint32_t* pcnt = base + 3 * k4;
  const Genome g = make_genome(chrom_end, bin_off, chrom_excl, n_chrom, bin_size);
  Filter f{strategy, min_len, max_len};
  const size_t smem = sizeof(RunSmem) + 2 * (size_t)kSmemKeys * sizeof(uint32_t);
  // per function and device; cheap enough to set on every call
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (sms < 1 || cudaFuncSetAttribute(sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
                     cudaSuccess)
    return SG_ERR_CUDA;
  layout_kernel<<<1, 1024, 0, s>>>(g, out_indptr);  // the flag in out_indptr[0] until sort_kernel clears it
  SG_CHECK_LAUNCH();
  stream_kernel<<<(unsigned)n_cells, kStreamThreads, 0, s>>>(cell_ptr, n_cells, n_frags, frag_pos, frag_len, g, f,
                                                             key_ptr, k4, pidx, pcnt, out_indptr, status, bad);
  SG_CHECK_LAUNCH();
  sort_kernel<<<(unsigned)std::min<int64_t>(n_cells, sms), kRunBlock, smem, s>>>(
      cell_ptr, n_cells, n_frags, frag_pos, frag_len, g, f, key_ptr, k4, gkeys, gtmp, pidx, pcnt, out_indptr, status,
      bad);
  SG_CHECK_LAUNCH();
  if (inclusive_scan_i64(out_indptr + 1, n_cells, scan_scratch, s) != cudaSuccess) return SG_ERR_CUDA;
  return SG_OK;
}

extern "C" int sg_tile_emit(int64_t n_cells, const int64_t* key_ptr, const void* scratch,
                            int64_t scratch_bytes, const int64_t* out_indptr, int32_t* out_idx,
                            uint32_t* out_cnt, int64_t cap, int* status, void* stream) {
  if (n_cells < 0) return SG_ERR_ARG;
  if (n_cells == 0) return SG_OK;
  const int64_t k4 = (scratch_bytes - 16) / (4 * (int64_t)sizeof(uint32_t));
  if (k4 < 0) return SG_ERR_CAP;
  const uint32_t* base = reinterpret_cast<const uint32_t*>(scratch);
  emit_kernel<<<(unsigned)n_cells, 256, 0, as_stream(stream)>>>(
      n_cells, key_ptr, k4, reinterpret_cast<const int32_t*>(base + 2 * k4), base + 3 * k4, out_indptr,
      out_idx, out_cnt, cap, status);
  SG_CHECK_LAUNCH();
  return SG_OK;
}
