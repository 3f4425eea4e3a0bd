// Exact Euclidean k-nearest-neighbour graph, replacing the reference's
// kd-tree search (snapatac2-core/src/utils/knn.rs:9-31: squared Euclidean in
// FP64, self removed by index, first k kept, value = sqrt(distance); rows of
// the CSR sorted by column index, to_csr_matrix 58-78).
//
// Pipeline (no host synchronisation):
//  1. prep    X (n x d FP64) -> zero-padded FP32 and FP64 copies (n x DP),
//             max row norm.  From kOrderMin points on, the FP32 copy is in a
//             space-filling order (point_order), so that tiles are compact.
//  2. scan    tiled brute force in FP32, filter then verify: a CTA owns 32
//             queries and streams 128-candidate tiles (stored tile-transposed,
//             so a tile is one coalesced 16 KB copy) through shared memory.
//             Filter: every thread computes 4 queries x 4 candidates in the
//             expanded form |q|^2 + |c|^2 - 2 q.c (one FFMA per dimension and
//             pair) and keeps the pairs that pass the current K'-th distance
//             tau widened by a bound on the FP32 error of that form (so no
//             pair whose exact-order difference-form distance is below tau is
//             dropped).  Verify: the warp recomputes the kept pairs in the
//             difference form sum (q_t - c_t)^2 (the FP32 arithmetic the
//             certificate below is stated for) and appends those below tau to
//             the query's list, shrunk to K' when it overflows.  On ordered
//             points of up to 32 dimensions the dot products come from the
//             tensor cores and far tiles are left out (tc_filter_kernel).
//  3. rerank  FP64 distances of the K' candidates, sort by (distance, index),
//             keep k.  Certificate: every point outside the list has FP32
//             distance >= tau (the K'-th), hence FP64 distance >= tau - delta
//             with delta a bound on the FP32 error; if tau - delta > the k-th
//             FP64 distance the FP64 top-k is exact, otherwise the query is
//             queued for
//  4. exact   the same scan in FP64 for the queued queries only.
//  5. rows sorted by column index, distances sqrt'ed.
// Ties are broken by the smaller index.
#include <cuda_bf16.h>
#include <float.h>
#include <stdlib.h>
#include <string.h>

#include <type_traits>

#include "common.cuh"
#include "internal.h"

namespace sg {
namespace {

constexpr int kQT = 32;    // queries per CTA (one per lane)
constexpr int kCT = 128;   // candidates per shared-memory tile
constexpr int kLW = 8;     // warps per CTA
constexpr int kList = 256; // per-query list + append buffer
constexpr int kMaxKp = 128;

template <typename K>
__device__ __forceinline__ bool lex_gt(K a, int ia, K b, int ib) {
  return a > b || (a == b && ia > ib);
}

// Ascending bitonic sort of N = 2^p (key, idx) pairs in shared memory by one warp.
template <typename K>
__device__ void warp_bitonic(K* key, int* idx, int N) {
  const int lane = threadIdx.x & 31;
  for (int size = 2; size <= N; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int t = lane; t < (N >> 1); t += 32) {
        const int i = 2 * t - (t & (stride - 1));
        const int j = i + stride;
        const bool asc = (i & size) == 0;
        const K ki = key[i], kj = key[j];
        const int ii = idx[i], ij = idx[j];
        if (lex_gt(ki, ii, kj, ij) == asc) {
          key[i] = kj; key[j] = ki;
          idx[i] = ij; idx[j] = ii;
        }
      }
      __syncwarp();
    }
  }
}

template <typename K> __device__ __forceinline__ K kinf();
template <> __device__ __forceinline__ double kinf<double>() { return DBL_MAX; }

template <typename TD, int DP>
struct ScanSmem {
  TD cv[kCT][DP];          // candidate tile
  TD dist[kQT][kCT + 1];   // distance tile
  TD lk[kQT][kList];       // per-query list keys
  int li[kQT][kList];      // per-query list indices
  int cnt[kQT];
  TD tau[kQT];
};

// Sort query q's list (warp), keep Kp, update tau.
template <typename TD, int DP>
__device__ void merge_list(ScanSmem<TD, DP>& sm, int q, int Kp) {
  const int lane = threadIdx.x & 31;
  const int c = sm.cnt[q];
  for (int t = c + lane; t < kList; t += 32) {
    sm.lk[q][t] = kinf<TD>();
    sm.li[q][t] = 0x7fffffff;
  }
  __syncwarp();
  warp_bitonic<TD>(sm.lk[q], sm.li[q], kList);
  __syncwarp();
  if (lane == 0) {
    const int keep = c < Kp ? c : Kp;
    sm.cnt[q] = keep;
    sm.tau[q] = keep == Kp ? sm.lk[q][Kp - 1] : kinf<TD>();
  }
  __syncwarp();
}

// Scan all n points for queries qlist[blockIdx.x*32 + lane] (or the identity
// when qlist == nullptr).  Writes per query the Kp best (distance, index)
// sorted ascending, and tau = Kp-th distance (inf if fewer).
template <typename TD, int DP>
__global__ void __launch_bounds__(kLW * 32)
scan_kernel(const TD* __restrict__ Xp, int64_t n, const int* __restrict__ qlist, const int* __restrict__ qcount,
            int Kp, int* __restrict__ cand, TD* __restrict__ cand_d, TD* __restrict__ tau_out) {
  extern __shared__ __align__(128) unsigned char sraw[];
  ScanSmem<TD, DP>& sm = *reinterpret_cast<ScanSmem<TD, DP>*>(sraw);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t nq = qcount ? (int64_t)*qcount : n;
  const int64_t qbase = (int64_t)blockIdx.x * kQT;
  if (qbase >= nq) return;  // uniform across the CTA
  const int64_t qslot = qbase + lane;
  const bool qvalid = qslot < nq;
  const int64_t qid = qvalid ? (qlist ? (int64_t)qlist[qslot] : qslot) : -1;

  using V = typename std::conditional<sizeof(TD) == 4, float4, double2>::type;
  constexpr int VW = 16 / sizeof(TD);
  TD qr[DP];
#pragma unroll
  for (int t = 0; t < DP; t += VW) {
    V v;
    if (qvalid) v = *reinterpret_cast<const V*>(Xp + qid * DP + t);
    else memset(&v, 0, sizeof(v));
    const TD* pv = reinterpret_cast<const TD*>(&v);
#pragma unroll
    for (int s = 0; s < VW; ++s) qr[t + s] = pv[s];
  }
  if (threadIdx.x < kQT) {
    sm.cnt[threadIdx.x] = 0;
    sm.tau[threadIdx.x] = kinf<TD>();
  }
  for (int64_t c0 = 0; c0 < n; c0 += kCT) {
    __syncthreads();
    // load candidate tile
    const int nct = (n - c0) < kCT ? (int)(n - c0) : kCT;
    for (int t = threadIdx.x; t < kCT * DP / VW; t += kLW * 32) {
      const int r = t / (DP / VW), v = t % (DP / VW);
      V val;
      if (r < nct) val = *reinterpret_cast<const V*>(Xp + (c0 + r) * DP + v * VW);
      else memset(&val, 0, sizeof(val));
      *reinterpret_cast<V*>(&sm.cv[r][v * VW]) = val;
    }
    __syncthreads();
    // distances: lane = query, warp covers candidates wid, wid+8, ...
#pragma unroll 2
    for (int j = 0; j < kCT / kLW; ++j) {
      const int c = wid + j * kLW;
      TD acc = TD(0);
#pragma unroll
      for (int t = 0; t < DP; t += VW) {
        const V v = *reinterpret_cast<const V*>(&sm.cv[c][t]);
        const TD* pv = reinterpret_cast<const TD*>(&v);
#pragma unroll
        for (int s = 0; s < VW; ++s) {
          if (sizeof(TD) == 8) {  // FP64 pass: the reference's unfused arithmetic
            const double df = __dsub_rn((double)qr[t + s], (double)pv[s]);
            acc = (TD)__dadd_rn((double)acc, __dmul_rn(df, df));
          } else {
            const TD df = qr[t + s] - pv[s];
            acc = fma(df, df, acc);
          }
        }
      }
      const int64_t cg = c0 + c;
      if (c >= nct || cg == qid || !qvalid) acc = kinf<TD>();
      sm.dist[lane][c] = acc;
    }
    __syncthreads();
    // fused selection: warp wid owns queries 4*wid .. 4*wid+3
    for (int qq = 0; qq < kQT / kLW; ++qq) {
      const int q = wid * (kQT / kLW) + qq;
      const TD th = sm.tau[q];
      int base = sm.cnt[q];
#pragma unroll
      for (int j = 0; j < kCT / 32; ++j) {
        const int c = lane + 32 * j;
        const TD dv = sm.dist[q][c];
        const bool take = dv < th;
        const unsigned bal = __ballot_sync(0xffffffffu, take);
        if (take) {
          const int p = base + __popc(bal & lanemask_lt());
          sm.lk[q][p] = dv;
          sm.li[q][p] = (int)(c0 + c);
        }
        base += __popc(bal);
      }
      __syncwarp();
      if (lane == 0) sm.cnt[q] = base;
      __syncwarp();
      if (base > kList - kCT) merge_list<TD, DP>(sm, q, Kp);
    }
  }
  __syncthreads();
  for (int qq = 0; qq < kQT / kLW; ++qq) {
    const int q = wid * (kQT / kLW) + qq;
    merge_list<TD, DP>(sm, q, Kp);
    const int64_t qs = qbase + q;
    if (qs < nq) {
      const int c = sm.cnt[q];
      for (int t = lane; t < Kp; t += 32) {
        cand[qs * Kp + t] = t < c ? sm.li[q][t] : -1;
        if (cand_d) cand_d[qs * Kp + t] = t < c ? sm.lk[q][t] : kinf<TD>();
      }
      if (lane == 0 && tau_out) tau_out[qs] = sm.tau[q];
    }
  }
}

// ---------------------------------------------------------------------------
// FP32 filter-verify scan (step 2).  XT holds the centred FP32 points tile-
// transposed: tile t (points 128t .. 128t+127) at XT + t*DP*128, coordinate
// (dim, j) at [dim*128 + j], zero beyond n; nrm[i] = FP32 of |x_i - mean|^2.
// ---------------------------------------------------------------------------
constexpr int kFQ = 32;          // queries per CTA
constexpr int kFC = 128;         // candidates per tile
constexpr int kFW = 8;           // warps per CTA (warp w owns queries 4w .. 4w+3)
constexpr int kFBuf = 3;         // candidate tiles in flight (ring)

// LIST entries per query: the kept Kp plus one verify batch of 32 (a list is
// re-sorted before a batch that would not fit), so LIST >= Kp + 32.
template <int DP, int LIST>
struct FilterSmem {
  uint64_t full[kFBuf];                      // tile k landed in buffer k % kFBuf
  uint64_t empty[kFBuf];                     // every warp is done with that buffer
  __align__(16) float cT[kFBuf][DP][kFC];    // candidate tiles (bulk copies of XT)
  __align__(16) float cn[kFBuf][kFC];        // their squared norms (bulk copies of nrm)
  __align__(16) float qT[DP][kFQ];
  float lk[kFQ][LIST];
  int li[kFQ][LIST];
  int cnt[kFQ];
  float tau[kFQ];
  unsigned queue[kFW][kFC];                  // one query's filtered candidates of a tile
  int nqueue[kFW];
};

// Shrink the lists of R queries (warp) to their Kp smallest distances and
// update tau, the bound that every point outside a list is at or above.  The
// lists are held in registers and the Kp-th distance found bit by bit
// (distances are not negative, so their bits order as integers), one
// warp-wide count per bit; the counts of the R lists are independent and
// overlap.  Unless `exact`, a bound that keeps up to `slack` entries more ends
// the search early (8 to 10 counts instead of some 25).  A bitonic sort of
// each list in shared memory did this before, in 28 dependent rounds of
// shared loads and stores (3,500 clocks a list).
template <int LIST, int R>
__device__ void shrink_lists(const int (&row)[R], float (*lk)[LIST], int (*li)[LIST], int* cnt, float* tau, int Kp,
                             int slack, bool exact) {
  constexpr int E = LIST / 32;
  const int lane = threadIdx.x & 31;
  unsigned key[R][E], lo[R];
  int id[R][E], hb[R];
  bool live[R], strict[R];  // warp-uniform
  int top = -1;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int c = row[i] >= 0 ? cnt[row[i]] : 0;
    live[i] = c >= Kp;  // else everything is kept and tau stays open
    unsigned mn = 0xffffffffu, mx = 0u;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int t = e * 32 + lane;
      const bool in = live[i] && t < c;
      key[i][e] = in ? __float_as_uint(lk[row[i]][t]) : 0xffffffffu;
      id[i][e] = in ? li[row[i]][t] : 0;
      mn = min(mn, key[i][e]);
      if (in) mx = max(mx, key[i][e]);
    }
    mn = __reduce_min_sync(0xffffffffu, mn);
    mx = __reduce_max_sync(0xffffffffu, mx);
    // the largest lo with fewer than Kp keys below it is the Kp-th key
    hb[i] = !live[i] || mn == mx ? -1 : 31 - __clz(mn ^ mx);
    lo[i] = hb[i] < 0 ? mn : mn & ~((2u << hb[i]) - 1u);
    strict[i] = false;
    top = max(top, hb[i]);
  }
  auto below = [&](int i, unsigned t) {
    int n = 0;
#pragma unroll
    for (int e = 0; e < E; ++e) n += key[i][e] < t;
    return __reduce_add_sync(0xffffffffu, n);
  };
  for (int bit = top; bit >= 0; --bit) {
    bool going = false;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const unsigned t = lo[i] | (1u << bit);
      const int n = below(i, t);
      if (bit <= hb[i] && !strict[i]) {
        if (n < Kp) lo[i] = t;
        else if (!exact && n <= Kp + slack) {
          lo[i] = t;
          strict[i] = true;
        }
      }
      going |= !strict[i] && hb[i] >= 0;
    }
    if (!going) break;
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < R; ++i) {
    if (!live[i]) continue;
    int more = strict[i] ? 0 : Kp - below(i, lo[i]);  // equal keys that still fit
    int at = 0;
    float* k = lk[row[i]];
    int* v = li[row[i]];
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const bool eq = !strict[i] && key[i][e] == lo[i];
      const unsigned be = __ballot_sync(0xffffffffu, eq);
      const bool take = key[i][e] < lo[i] || (eq && __popc(be & lanemask_lt()) < more);
      more -= min(more, __popc(be));
      const unsigned bt = __ballot_sync(0xffffffffu, take);
      if (take) {
        const int p = at + __popc(bt & lanemask_lt());
        k[p] = __uint_as_float(key[i][e]);
        v[p] = id[i][e];
      }
      at += __popc(bt);
    }
    if (lane == 0) {
      cnt[row[i]] = at;
      tau[row[i]] = __uint_as_float(lo[i]);
    }
  }
  __syncwarp();
}

// Warps advance through the tiles on their own: a tile is consumed once its
// copy lands (full barrier), and its buffer is refilled only after all
// warps arrived on its empty barrier, so a warp busy re-sorting a list holds
// up the others only once they run a whole ring ahead.  Thread 0 produces.
template <int DP, int LIST>
__global__ void __launch_bounds__(kFW * 32, 2)
filter_scan_kernel(const float* __restrict__ XT, const float* __restrict__ nrm, int64_t n, int d, int Kp,
                   const int* __restrict__ perm, int* __restrict__ cand, float* __restrict__ tau_out) {
  extern __shared__ __align__(128) unsigned char sraw[];
  FilterSmem<DP, LIST>& sm = *reinterpret_cast<FilterSmem<DP, LIST>*>(sraw);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t qbase = (int64_t)blockIdx.x * kFQ;
  const int64_t ntiles = (n + kFC - 1) / kFC;
  constexpr uint32_t kTileBytes = DP * kFC * 4, kNormBytes = kFC * 4;
  const int slack = min(8, LIST - 32 - Kp);
  // the k-th tile taken: the queries' own, then outwards (in an ordered copy
  // near points sit in near tiles, and tau is tight after the first few)
  const int64_t own = qbase / kFC;
  auto tile_of = [&](int64_t k) {
    int64_t t = own + ((k & 1) ? (k + 1) / 2 : -(k / 2));
    if (t < 0) t += ntiles;
    if (t >= ntiles) t -= ntiles;
    return t;
  };
  auto issue = [&](int64_t k) {
    const int b = (int)(k % kFBuf);
    const int64_t t = tile_of(k);
    mbar_expect_tx(&sm.full[b], kTileBytes + kNormBytes);
    bulk_copy(&sm.cT[b][0][0], XT + t * DP * kFC, kTileBytes, &sm.full[b]);
    bulk_copy(&sm.cn[b][0], nrm + t * kFC, kNormBytes, &sm.full[b]);
  };
  if (threadIdx.x == 0) {
    for (int b = 0; b < kFBuf; ++b) {
      mbar_init(&sm.full[b], 1);
      mbar_init(&sm.empty[b], kFW);
    }
    fence_barrier_init();
    fence_proxy_async();
    for (int64_t k = 0; k < kFBuf - 1 && k < ntiles; ++k) issue(k);
  }
  {
    const float* src = XT + (qbase / kFC) * DP * kFC + (qbase % kFC);
    for (int e = threadIdx.x; e < DP * kFQ; e += blockDim.x) sm.qT[e / kFQ][e % kFQ] = src[(e / kFQ) * kFC + e % kFQ];
  }
  if (threadIdx.x < kFQ) {
    sm.cnt[threadIdx.x] = 0;
    sm.tau[threadIdx.x] = FLT_MAX;
  }
  if (lane == 0) sm.nqueue[wid] = 0;
  float qn[4];
  int64_t qid[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    qid[i] = qbase + 4 * wid + i;
    qn[i] = qid[i] < n ? nrm[qid[i]] : 0.f;
  }
  __syncthreads();
  // Filter bound.  With u = 2^-24, s the FP32 dot product (FMA chain over DP
  // terms), nq, nc the FP32 squared norms and D^ the exact squared distance
  // of the FP32 points: |(nq + nc - 2 s) - D^| <= (DP + 3) u (nq + nc) + u D^,
  // and the difference-form FP32 distance d32 obeys |d32 - D^| <= (d + 3) u D^.
  // So d32 < tau implies nq + nc - 2 s < tau + Ku (nq + nc) + Tu tau with
  // K = 2 DP + 16, T = 4 (d + 4) (twice the derived constants, which also
  // covers the rounding of the test itself), written as
  // nc (1 - Ku) - 2 s < tau (1 + Tu) + Ku nq - nq.
  const float u = 5.9604644775390625e-08f;
  const float Ku = (float)(2 * DP + 16) * u, Tu = (float)(4 * (d + 4)) * u;
  const float kInf = __int_as_float(0x7f800000);
  bool failed = false;
  int64_t issued = kFBuf - 1 < ntiles ? kFBuf - 1 : ntiles;  // tiles handed to the copy engine (thread 0)
  for (int64_t k = 0; k < ntiles; ++k) {
    const int b = (int)(k % kFBuf);
    bool pfail = false;
    if (threadIdx.x == 0 && k + kFBuf - 1 < ntiles) {
      // refill the buffer tile k - 1 used, once every warp is done with it
      const int64_t kn = k + kFBuf - 1;
      const bool ok = kn < kFBuf || mbar_wait(&sm.empty[kn % kFBuf], (uint32_t)(((kn / kFBuf) - 1) & 1));
      if (ok) {
        fence_proxy_async();
        issue(kn);
        issued = kn + 1;
      } else {
        pfail = true;
      }
    }
    const bool got = !pfail && mbar_wait(&sm.full[b], (uint32_t)((k / kFBuf) & 1));
    if (!__all_sync(0xffffffffu, got)) {
      failed = true;  // a tile never landed: leave this warp's queries to the exact rescan
      break;
    }
    const int64_t c0 = tile_of(k) * kFC;
    float T[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float tq = sm.tau[4 * wid + i];
      T[i] = qid[i] >= n ? -kInf : (tq >= FLT_MAX ? kInf : (tq + Tu * tq) + (Ku * qn[i] - qn[i]));
    }
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
#pragma unroll 8
    for (int t = 0; t < DP; ++t) {
      const float4 qv = *reinterpret_cast<const float4*>(&sm.qT[t][4 * wid]);
      const float4 cv = *reinterpret_cast<const float4*>(&sm.cT[b][t][4 * lane]);
      const float qa[4] = {qv.x, qv.y, qv.z, qv.w}, ca[4] = {cv.x, cv.y, cv.z, cv.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(qa[i], ca[j], acc[i][j]);
    }
    const float4 cn4 = *reinterpret_cast<const float4*>(&sm.cn[b][4 * lane]);
    const float cadj[4] = {cn4.x * (1.0f - Ku), cn4.y * (1.0f - Ku), cn4.z * (1.0f - Ku), cn4.w * (1.0f - Ku)};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int q = 4 * wid + i;
      const int64_t so = qid[i] - c0;  // the query's own column in this tile, if any
      const int self = (so >= 0 && so < kFC) ? (int)so : -1;
      bool keep[4];
      bool any = false;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        keep[j] = fmaf(-2.0f, acc[i][j], cadj[j]) < T[i] && 4 * lane + j != self;
        any |= keep[j];
      }
      if (!__any_sync(0xffffffffu, any)) continue;  // nothing of this query passed the filter
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (keep[j]) sm.queue[wid][atomicAdd(&sm.nqueue[wid], 1)] = (unsigned)(4 * lane + j);
      __syncwarp();
      // verify in the difference form; append (ballot order) those below tau,
      // re-sorting the list first when the batch would not fit
      const int nk = sm.nqueue[wid];
      int cq = sm.cnt[q];
      for (int e0 = 0; e0 < nk; e0 += 32) {
        const int e = e0 + lane;
        int c = 0;
        float dd = kInf;
        if (e < nk) {
          c = (int)sm.queue[wid][e];
          dd = 0.f;
#pragma unroll
          for (int t = 0; t < DP; ++t) {
            const float df = sm.qT[t][q] - sm.cT[b][t][c];
            dd = fmaf(df, df, dd);
          }
        }
        bool pass = dd < sm.tau[q];
        unsigned bal = __ballot_sync(0xffffffffu, pass);
        if (cq + __popc(bal) > LIST) {
          if (lane == 0) sm.cnt[q] = cq;
          __syncwarp();
          shrink_lists<LIST, 1>({q}, sm.lk, sm.li, sm.cnt, sm.tau, Kp, slack, false);
          cq = sm.cnt[q];
          pass = dd < sm.tau[q];
          bal = __ballot_sync(0xffffffffu, pass);
        }
        if (pass) {
          const int p = cq + __popc(bal & lanemask_lt());
          sm.lk[q][p] = dd;
          sm.li[q][p] = (int)(c0 + c);
        }
        cq += __popc(bal);
      }
      if (lane == 0) {
        sm.cnt[q] = cq;
        sm.nqueue[wid] = 0;
      }
      __syncwarp();
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&sm.empty[b]);  // this warp is done with buffer b
  }
  failed = __any_sync(0xffffffffu, failed);
  if (!failed) {
    shrink_lists<LIST, 2>({4 * wid, 4 * wid + 1}, sm.lk, sm.li, sm.cnt, sm.tau, Kp, 0, true);
    shrink_lists<LIST, 2>({4 * wid + 2, 4 * wid + 3}, sm.lk, sm.li, sm.cnt, sm.tau, Kp, 0, true);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int q = 4 * wid + i;
    if (qid[i] < n) {
      const int64_t qo = perm ? perm[qid[i]] : qid[i];
      const int c = failed ? 0 : sm.cnt[q];
      for (int t = lane; t < Kp; t += 32) cand[qo * Kp + t] = t < c ? (perm ? perm[sm.li[q][t]] : sm.li[q][t]) : -1;
      if (lane == 0) tau_out[qo] = failed ? -1.0f : sm.tau[q];  // negative tau: certificate fails
    }
  }
  // no copy may still be landing in this CTA's shared memory when it exits:
  // after a failure, wait (bounded) for the last tiles thread 0 issued
  if (threadIdx.x == 0 && failed)
    for (int64_t t = issued - kFBuf < 0 ? 0 : issued - kFBuf; t < issued; ++t)
      mbar_wait(&sm.full[t % kFBuf], (uint32_t)((t / kFBuf) & 1));
}

// ---------------------------------------------------------------------------
// Tensor-core filter (d <= 32).  The filter's dot products q.c come from
// tcgen05.mma: the centred FP32 coordinates are split into bf16 hi + lo and
// q.c ~= qh.ch + qh.cl + ql.ch (three K = 32 products per 128 x 128 tile,
// FP32 accumulation in TMEM).  Dropped terms and accumulation stay below
// 6e-5 sum|q_t c_t|; the filter is widened by KTC = 2^-12 of nq + nc (four
// times that), so, as in the FP32 filter, no pair whose difference-form
// distance is below tau is dropped; the verify, the lists and the output are
// those of filter_scan_kernel.
//
// TC layout (prep): per 128-point tile, [hi 8 KB][lo 8 KB][FP32 16 KB]
// [nc (1 - K) 512 B].  hi = RN(v) and lo = RN(v - hi) are bf16 in the
// no-swizzle K-major core-matrix layout: element (row r, dim t) at byte
// (r/8)*512 + (t/8)*128 + (r%8)*16 + (t%8)*2.  The FP32 rows (for the verify)
// have their 16-byte parts permuted by part ^ (r % 8), so that lanes that read
// the same part of different rows spread over the banks.
// ---------------------------------------------------------------------------
constexpr int kTQ = 128;                  // queries per CTA (MMA M)
constexpr int kTC = 128;                  // candidates per tile (MMA N)
constexpr int kTDim = 32;                 // K (padded dimensions)
constexpr int kTMat = kTQ * kTDim * 2;    // one bf16 operand: 8 KB
constexpr int kTRows = 2 * kTMat;         // byte offset of the FP32 rows
constexpr int kTNorm = kTRows + kTC * kTDim * 4;  // of the scaled norms
constexpr int kTTile = kTNorm + kTC * 4;
constexpr int kTBufMax = 4;               // tile buffers: as many as the heaps leave room for, two at least
constexpr int kTAcc = 4;                  // TMEM accumulators of 128 columns
constexpr int kTConsumers = 4;            // warps 0..3 read TMEM lanes 32w..32w+31
constexpr int kTThreads = (kTConsumers + 1) * 32;  // + one producer warp
constexpr float kTcK = 2.44140625e-4f + 8.0f * 5.9604644775390625e-08f;  // 2^-12 + rounding of the test

struct TcSmem {
  uint64_t full[kTBufMax];  // tile landed
  uint64_t sfree[kTBufMax]; // tile consumed: MMA done (commit) + 4 consumer warps
  uint64_t mdone[kTAcc];    // accumulator x holds tile k (commit)
  uint64_t tfree[kTAcc];    // accumulator x read by the 4 consumer warps
  uint64_t aful;            // query operands landed
  uint64_t drain;           // failure path: every MMA issued so far has completed (commit)
  uint32_t tmem_slot;
  int failed;
  int seq[kTBufMax];        // tile in each buffer, -1: no more tiles
  float qlo[kTDim], qhi[kTDim];  // bounding box of the queries
  float tau[kTQ];
  __align__(128) unsigned char A[2 * kTMat];
  // followed by the tile buffers and the heaps: distances, then indices, [warp][entry][lane]
};
static_assert(sizeof(TcSmem) % 128 == 0, "the tile buffers follow on a 128-byte boundary");

// entries of a heap of Kp: whole groups of eight children below the root
__host__ __device__ constexpr int heap_entries(int Kp) { return Kp <= 1 ? 1 : 1 + (Kp - 1 + 7) / 8 * 8; }
constexpr size_t kTSmemMax = 232448;  // shared memory of a CTA
constexpr size_t tc_smem_bytes(int Kp, int nbuf) {
  return sizeof(TcSmem) + (size_t)nbuf * kTTile + (size_t)heap_entries(Kp) * kTQ * 8;
}
constexpr int tc_buffers(int Kp) {
  return tc_smem_bytes(Kp, 4) <= kTSmemMax ? 4 : (tc_smem_bytes(Kp, 3) <= kTSmemMax ? 3 : 2);
}
static_assert(tc_smem_bytes(kMaxKp, tc_buffers(kMaxKp)) <= kTSmemMax, "tensor-core filter shared memory");

__device__ __forceinline__ uint32_t tc_off(int r, int t) {
  return (uint32_t)((r >> 3) * 512 + (t >> 3) * 128 + (r & 7) * 16 + (t & 7) * 2);
}

// TC layout from the tile-transposed FP32 copy (XT) and the norms.
__global__ void tc_prep_kernel(const float* __restrict__ XT, const float* __restrict__ nrm, int64_t n,
                               unsigned char* __restrict__ TC) {
  const int64_t npad = (n + kFC - 1) / kFC * kFC;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < npad; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t k = i / kFC;
    const int r = (int)(i % kFC);
    unsigned char* tile = TC + k * kTTile;
    const float* src = XT + k * 32 * kFC + r;
#pragma unroll 2
    for (int t0 = 0; t0 < kTDim; t0 += 8) {
      float v[8];
      __nv_bfloat162 h[4], l[4];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = src[(t0 + j) * kFC];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        h[j] = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
        l[j] = __floats2bfloat162_rn(v[2 * j] - __low2float(h[j]), v[2 * j + 1] - __high2float(h[j]));
      }
      *reinterpret_cast<uint4*>(tile + tc_off(r, t0)) = *reinterpret_cast<const uint4*>(h);
      *reinterpret_cast<uint4*>(tile + kTMat + tc_off(r, t0)) = *reinterpret_cast<const uint4*>(l);
      float4* x = reinterpret_cast<float4*>(tile + kTRows) + r * (kTDim / 4);
      x[(t0 / 4) ^ (r & 7)] = make_float4(v[0], v[1], v[2], v[3]);
      x[(t0 / 4 + 1) ^ (r & 7)] = make_float4(v[4], v[5], v[6], v[7]);
    }
    reinterpret_cast<float*>(tile + kTNorm)[r] = nrm[i] * (1.0f - kTcK);  // the filter's nc (1 - K)
  }
}

// Bounding boxes of the tiles, 32 tiles to a group: lo then hi, [dim][tile]
// within a group (a lane per tile reads them coalesced); tiles past the end
// get an empty box, at infinite distance from every other.
__global__ void __launch_bounds__(128)
tile_box_kernel(const float* __restrict__ XT, int64_t n, int64_t ntiles, float* __restrict__ box) {
  const int64_t k = blockIdx.x;  // tiles, up to whole groups
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const float inf = __int_as_float(0x7f800000);
  float* lo = box + (k >> 5) * 2 * kTDim * 32 + (k & 31);
  float* hi = lo + kTDim * 32;
  for (int t = w; t < kTDim; t += 4) {
    float a = inf, b = -inf;
    if (k < ntiles)
      for (int j = lane; j < kFC; j += 32)
        if (k * kFC + j < n) {
          const float v = XT[(k * 32 + t) * kFC + j];
          a = fminf(a, v);
          b = fmaxf(b, v);
        }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      a = fminf(a, __shfl_xor_sync(0xffffffffu, a, o));
      b = fmaxf(b, __shfl_xor_sync(0xffffffffu, b, o));
    }
    if (lane == 0) {
      lo[t * 32] = a;
      hi[t * 32] = b;
    }
  }
}

// Tiles are taken from the queries' own outwards, 32 at a time and nearest
// box first, and a tile whose box is further from the queries' box than the
// largest tau of the CTA is left out: no pair of it can be below any tau.
// With the points in the order of point_order (below) a third to a half of
// the tiles fall to that test, and the first tiles bring tau close to its
// final value, so that few later pairs reach the verify step.
//
// A consumer lane owns one query from end to end: its coordinates are in
// registers, the pairs of its acceptance mask are verified one after another
// from the tile in shared memory, and its Kp smallest distances are an 8-ary
// max-heap in shared memory whose root is tau (two levels at 66).  The
// heaps of a warp are interleaved ([entry][lane]), so a lane's accesses stay
// in its own bank whatever the others do.  Lists that were sorted by the whole
// warp when they overflowed, fed by a queue of pairs, took four fifths of the
// time.  100,000 points in 30 dimensions, k = 50: 21.0 ms in input order with
// those lists, 8.1 ms in the point order, 5.5 ms with heaps.  Now the three
// phases of a tile (waiting for the slowest warp, the filter, verify and
// insertion) cost about a quarter, a quarter and a half; one warp per
// scheduler leaves each of them bound by latency.
template <int NB>  // tile buffers
__global__ void __launch_bounds__(kTThreads)
tc_filter_kernel(const unsigned char* __restrict__ TC, const float* __restrict__ nrm,
                 const float* __restrict__ box, int64_t n, int d, int Kp,
                 const int* __restrict__ perm, int* __restrict__ cand, float* __restrict__ tau_out) {
  extern __shared__ __align__(128) unsigned char sraw[];
  TcSmem& sm = *reinterpret_cast<TcSmem*>(sraw);
  unsigned char* tiles = sraw + sizeof(TcSmem);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t qbase = (int64_t)blockIdx.x * kTQ;
  const int64_t ntiles = (n + kTC - 1) / kTC;
  if (wid == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&sm.tmem_slot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (threadIdx.x == 0) {
    for (int b = 0; b < NB; ++b) {
      mbar_init(&sm.full[b], 1);
      mbar_init(&sm.sfree[b], 1 + kTConsumers);
    }
    for (int x = 0; x < kTAcc; ++x) {
      mbar_init(&sm.mdone[x], 1);
      mbar_init(&sm.tfree[x], kTConsumers);
    }
    mbar_init(&sm.aful, 1);
    mbar_init(&sm.drain, 1);
    sm.failed = 0;
    fence_barrier_init();
  }
  if (wid < kTConsumers) {
    sm.tau[wid * 32 + lane] = qbase + wid * 32 + lane < n ? FLT_MAX : 0.f;
  } else {
    const float* b = box + (blockIdx.x >> 5) * 2 * kTDim * 32 + (blockIdx.x & 31);
    sm.qlo[lane] = b[lane * 32];
    sm.qhi[lane] = b[(kTDim + lane) * 32];
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm.tmem_slot;
  const uint32_t idesc = umma_idesc_bf16(kTQ, kTC);
  bool failed = false;

  if (wid == kTConsumers) {
    // -------- producer warp: choice of tiles; lane 0: copies and MMAs ------
    const int64_t ngroups = (ntiles + 31) / 32, own_group = (int64_t)blockIdx.x >> 5;
    const int64_t reach = own_group > ngroups - 1 - own_group ? own_group : ngroups - 1 - own_group;
    int64_t step = -1, group = 0;  // groups own, own + 1, own - 1, own + 2, ...
    unsigned pend = 0;             // tiles of the group not taken or left out yet
    float lb = 0.f;                // this lane's tile: squared distance of the boxes
    auto next_tile = [&]() -> int {  // warp-uniform; -1: none is left
      while (true) {
        if (!pend) {
          do {
            if (++step > 2 * reach) return -1;
            group = own_group + ((step & 1) ? (step + 1) / 2 : -(step / 2));
          } while (group < 0 || group >= ngroups);
          const float* b = box + group * 2 * kTDim * 32 + lane;
          lb = 0.f;
#pragma unroll 16
          for (int t = 0; t < kTDim; ++t) {
            const float gap = fmaxf(fmaxf(__ldg(b + t * 32) - sm.qhi[t], sm.qlo[t] - __ldg(b + (kTDim + t) * 32)), 0.f);
            lb = fmaf(gap, gap, lb);
          }
          lb *= 0.99999f;  // 168 u: above the rounding of lb and of the difference-form distances together
          pend = 0xffffffffu;
        }
        float mt = 0.f;
        for (int j = lane; j < kTQ; j += 32) mt = fmaxf(mt, *(volatile float*)&sm.tau[j]);
        const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(mt));
        const unsigned key = ((pend >> lane) & 1u) && lb <= __uint_as_float(m) ? __float_as_uint(lb) : 0xffffffffu;
        const unsigned best = __reduce_min_sync(0xffffffffu, key);
        if (best == 0xffffffffu) {  // tau only falls: the rest of the group stays out
          pend = 0;
          continue;
        }
        const unsigned same = __ballot_sync(0xffffffffu, key == best);
        int sel = __ffs(same) - 1;
        if (step == 0 && (pend >> (blockIdx.x & 31) & 1u) && (same >> (blockIdx.x & 31) & 1u)) sel = blockIdx.x & 31;
        pend &= ~(1u << sel);
        return (int)(group * 32 + sel);
      }
    };
    // tiles [waited, issued) have copies in flight, at most one per buffer
    int issued = 0, waited = 0, total = -1;
    auto issue = [&](int k) {  // the k-th tile taken, or the end mark, into buffer k % NB
      const int t = next_tile();
      const int b = (int)(k % NB);
      if (lane == 0) {
        *(volatile int*)&sm.seq[b] = t;
        if (t >= 0) {
          mbar_expect_tx(&sm.full[b], kTTile);
          bulk_copy(tiles + b * kTTile, TC + (int64_t)t * kTTile, kTTile, &sm.full[b]);
        } else {
          mbar_arrive(&sm.full[b]);
        }
      }
      if (t >= 0) issued = k + 1;
      else total = k;
    };
    if (lane == 0) {
      mbar_expect_tx(&sm.aful, 2 * kTMat);
      bulk_copy(sm.A, TC + (qbase / kFC) * kTTile, 2 * kTMat, &sm.aful);
    }
    for (int k = 0; k < NB && total < 0; ++k) issue(k);
    const bool a_ok = __all_sync(0xffffffffu, mbar_wait(&sm.aful, 0));
    bool ok = a_ok;
    const uint32_t a_hi = smem_u32(sm.A), a_lo = a_hi + kTMat;
    // tile k: MMA as soon as it landed and its accumulator buffer was read
    // out (tile k - kTAcc); then refill the buffer tile k - 1 used once the
    // consumers are done with tile k - 1: copies and tensor cores work on the
    // next tiles while the consumers filter tile k.
    for (int k = 0; ok && k != total; ++k) {
      const int b = (int)(k % NB), x = (int)(k % kTAcc);
      ok = __all_sync(0xffffffffu, mbar_wait(&sm.full[b], (uint32_t)((k / NB) & 1)));
      if (ok) waited = k + 1;
      if (ok && k >= kTAcc)
        ok = __all_sync(0xffffffffu, mbar_wait(&sm.tfree[x], (uint32_t)(((k / kTAcc) - 1) & 1)));
      if (!ok) break;
      tc_fence_after();
      if (lane == 0) {
        const uint32_t b_hi = smem_u32(tiles + b * kTTile), b_lo = b_hi + kTMat;
        const uint32_t dst = tmem + (uint32_t)(x * kTC);
        const uint32_t pa[3] = {a_hi, a_hi, a_lo}, pb[3] = {b_hi, b_lo, b_hi};
#pragma unroll
        for (int p = 0; p < 3; ++p)
#pragma unroll
          for (int ks = 0; ks < kTDim / 16; ++ks)
            umma_bf16(dst, umma_desc(pa[p] + ks * 256u, 128u, 512u), umma_desc(pb[p] + ks * 256u, 128u, 512u), idesc,
                      p > 0 || ks > 0);
        umma_commit(&sm.mdone[x]);
        umma_commit(&sm.sfree[b]);
      }
      __syncwarp();
      const int kt = k + NB - 1;  // into the buffer tile k - 1 used
      if (total < 0 && kt >= NB) {
        ok = __all_sync(0xffffffffu, mbar_wait(&sm.sfree[(k - 1) % NB], (uint32_t)(((k - 1) / NB) & 1)));
        if (!ok) break;
        fence_proxy_async();
        issue(kt);
      }
    }
    if (!ok && lane == 0) {
      atomicExch(&sm.failed, 1);
      // before the CTA frees TMEM and exits, let what is in flight land:
      // the query copy, every tile copy not yet waited for (one phase per
      // buffer, so each parity wait is unambiguous) and every committed
      // MMA (a last commit completes once all earlier ones have); each
      // wait is bounded like the others
      if (!a_ok) mbar_wait(&sm.aful, 0);
      for (int t = waited; t < issued; ++t) mbar_wait(&sm.full[t % NB], (uint32_t)((t / NB) & 1));
      umma_commit(&sm.drain);
      mbar_wait(&sm.drain, 0);
    }
    __syncwarp();
  } else {
    // ---------------- consumers: filter from TMEM, verify, heaps ----------
    const int row = wid * 32 + lane;
    const int64_t q = qbase + row;
    const float nq = q < n ? nrm[q] : 0.f;
    const float u = 5.9604644775390625e-08f;
    const float Tu = (float)(4 * (d + 4)) * u;
    const float kInf = __int_as_float(0x7f800000);
    const int entries = heap_entries(Kp);
    unsigned char* heaps = tiles + NB * kTTile;
    float* hd = reinterpret_cast<float*>(heaps) + wid * entries * 32 + lane;
    int* hi = reinterpret_cast<int*>(heaps + (size_t)entries * kTQ * 4) + wid * entries * 32 + lane;
    for (int e = 0; e < entries; ++e) {  // Kp open places; the padding is below every distance
      hd[e * 32] = e < Kp ? FLT_MAX : -1.f;
      hi[e * 32] = -1;
    }
    float tau = q < n ? FLT_MAX : 0.f;
    float4 qv[kTDim / 4];
#pragma unroll
    for (int g = 0; g < kTDim / 4; ++g)
      qv[g] = __ldg(reinterpret_cast<const float4*>(TC + (qbase / kTC) * kTTile + kTRows) + row * (kTDim / 4) +
                    (g ^ (row & 7)));
    for (int k = 0;; ++k) {
      const int b = (int)(k % NB), x = (int)(k % kTAcc);
      bool ok = mbar_wait(&sm.full[b], (uint32_t)((k / NB) & 1));  // the tile's number and norms
      const int tile = *(volatile int*)&sm.seq[b];
      if (__all_sync(0xffffffffu, ok) && tile < 0) break;
      ok = ok && mbar_wait(&sm.mdone[x], (uint32_t)((k / kTAcc) & 1));
      if (!__all_sync(0xffffffffu, ok)) {
        failed = true;
        break;
      }
      tc_fence_after();
      const int64_t c0 = (int64_t)tile * kTC;
      const float4* cadj4 = reinterpret_cast<const float4*>(tiles + b * kTTile + kTNorm);
      const float4* rows = reinterpret_cast<const float4*>(tiles + b * kTTile + kTRows);
      const float T = q >= n ? -kInf : (tau >= FLT_MAX ? kInf : (tau + Tu * tau) + (kTcK * nq - nq));
      // acceptance masks, 32 candidates (one TMEM load) at a time, built only
      // where the smallest of a lane's 32 passes for some lane of the warp
      uint32_t mw[4];
      const uint32_t tbase = tmem + ((uint32_t)(wid * 32) << 16) + (uint32_t)(x * kTC);
      uint32_t v[2][32];  // the next 32 columns land while these are filtered
      tmem_ld32(tbase, v[0]);
#pragma unroll
      for (int w4 = 0; w4 < 4; ++w4) {
        tmem_wait();
        tmem_landed(v[w4 & 1]);
        if (w4 < 3) tmem_ld32(tbase + 32 * (w4 + 1), v[(w4 + 1) & 1]);
        float f[32];
        float least = kInf;
#pragma unroll
        for (int j4 = 0; j4 < 8; ++j4) {
          const float4 c = cadj4[8 * w4 + j4];
          f[4 * j4 + 0] = fmaf(-2.0f, __uint_as_float(v[w4 & 1][4 * j4 + 0]), c.x);
          f[4 * j4 + 1] = fmaf(-2.0f, __uint_as_float(v[w4 & 1][4 * j4 + 1]), c.y);
          f[4 * j4 + 2] = fmaf(-2.0f, __uint_as_float(v[w4 & 1][4 * j4 + 2]), c.z);
          f[4 * j4 + 3] = fmaf(-2.0f, __uint_as_float(v[w4 & 1][4 * j4 + 3]), c.w);
          least = fminf(fminf(least, fminf(f[4 * j4 + 0], f[4 * j4 + 1])), fminf(f[4 * j4 + 2], f[4 * j4 + 3]));
        }
        uint32_t mm = 0;
        if (__any_sync(0xffffffffu, least < T)) {
#pragma unroll
          for (int j = 0; j < 32; ++j) mm |= (f[j] < T ? 1u : 0u) << j;
        }
        mw[w4] = mm;
      }
      if (c0 == qbase) {  // the query itself
#pragma unroll
        for (int w4 = 0; w4 < 4; ++w4)
          if (w4 == wid) mw[w4] &= ~(1u << lane);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.tfree[x]);  // accumulator x may be overwritten
      auto next = [&]() -> int {  // takes a pair off the mask, -1: none is left
        const bool e0 = mw[0] != 0, e1 = mw[1] != 0, e2 = mw[2] != 0;
        const uint32_t m = e0 ? mw[0] : (e1 ? mw[1] : (e2 ? mw[2] : mw[3]));
        const int j = (e0 ? 0 : (e1 ? 32 : (e2 ? 64 : 96))) + __ffs(m) - 1;
        const uint32_t rest = m & (m - 1);
        mw[0] = e0 ? rest : mw[0];
        mw[1] = !e0 && e1 ? rest : mw[1];
        mw[2] = !e0 && !e1 && e2 ? rest : mw[2];
        mw[3] = !e0 && !e1 && !e2 ? rest : mw[3];
        return m ? j : -1;
      };
      auto distance = [&](int j) -> float {
        float d0 = 0.f, d1 = 0.f;  // two chains: no further off than the one that the certificate allows for
        const int jj = j < 0 ? 0 : j;
#pragma unroll
        for (int g = 0; g < kTDim / 4; ++g) {
          const float4 c = rows[jj * (kTDim / 4) + (g ^ (jj & 7))];
          float df = qv[g].x - c.x;
          d0 = fmaf(df, df, d0);
          df = qv[g].y - c.y;
          d1 = fmaf(df, df, d1);
          df = qv[g].z - c.z;
          d0 = fmaf(df, df, d0);
          df = qv[g].w - c.w;
          d1 = fmaf(df, df, d1);
        }
        return j < 0 ? kInf : d0 + d1;
      };
      auto insert = [&](float dd, int j) {  // replace the root, sift down
        int at = 0;
        while (8 * at + 1 < Kp) {
          const int c = 8 * at + 1;
          float a[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) a[i] = hd[(c + i) * 32];
          const float m = fmaxf(fmaxf(fmaxf(a[0], a[1]), fmaxf(a[2], a[3])), fmaxf(fmaxf(a[4], a[5]), fmaxf(a[6], a[7])));
          if (at == 0) tau = fmaxf(m, dd);  // the root's new value
          if (m <= dd) break;
          int to = c;
#pragma unroll
          for (int i = 1; i < 8; ++i)
            if (a[i] == m) to = c + i;
          hd[at * 32] = m;
          hi[at * 32] = hi[to * 32];
          at = to;
        }
        hd[at * 32] = dd;
        hi[at * 32] = (int)(c0 + j);
        if (Kp == 1) tau = dd;
      };
      // two pairs a round: their reads and sums overlap
#pragma unroll 1
      while (__any_sync(0xffffffffu, (mw[0] | mw[1] | mw[2] | mw[3]) != 0)) {
        const int ja = next(), jb = next();
        const float da = distance(ja), db = distance(jb);
        if (da < tau) insert(da, ja);
        if (db < tau) insert(db, jb);
      }
      if (q < n) *(volatile float*)&sm.tau[row] = tau;
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.sfree[b]);  // done with this tile
    }
    failed = __any_sync(0xffffffffu, failed);
    if (q < n) {
      const int64_t qo = perm ? perm[q] : q;
      for (int e = 0; e < Kp; ++e) {
        const int c = failed ? -1 : hi[e * 32];
        cand[qo * Kp + e] = c >= 0 && perm ? perm[c] : c;
      }
      tau_out[qo] = failed ? -1.0f : tau;  // negative tau: certificate fails
    }
  }
  tc_fence_before();
  __syncthreads();
  // a producer failure leaves every consumer result to the exact rescan
  if (sm.failed && wid < kTConsumers) {
    const int64_t qq = qbase + wid * 32 + lane;
    if (qq < n) tau_out[perm ? perm[qq] : qq] = -1.0f;
  }
  tc_fence_after();
  if (wid == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
}

constexpr int kMeanParts = 256;

// Column means and spreads of X (n x d FP64), deterministic: per-CTA partial
// sums (four rows at a time, 64 columns), then a fixed-order reduction.  The
// FP32 copy is centred on the means, which removes the component every point
// shares and shrinks the FP32 rounding of distances; the spreads (second
// moments about the first row) pick the axes of point_order.
__global__ void __launch_bounds__(256)
mean_partial(const double* __restrict__ X, int64_t n, int d, double* __restrict__ part, float* __restrict__ part2) {
  __shared__ double s1[4][64];
  __shared__ float s2[4][64];
  const int b = blockIdx.x, nb = gridDim.x, t = threadIdx.x & 63, g = threadIdx.x >> 6;
  const int64_t r0 = n * b / nb, r1 = n * (b + 1) / nb;
  double s = 0.0;
  float v = 0.f;
  if (t < d) {
    const double x0 = X[t];
#pragma unroll 4
    for (int64_t i = r0 + g; i < r1; i += 4) {
      const double x = X[i * d + t];
      s += x;
      const float c = (float)(x - x0);
      v = fmaf(c, c, v);
    }
  }
  s1[g][t] = s;
  s2[g][t] = v;
  __syncthreads();
  if (g == 0 && t < d) {
    part[b * 64 + t] = ((s1[0][t] + s1[1][t]) + s1[2][t]) + s1[3][t];
    part2[b * 64 + t] = ((s2[0][t] + s2[1][t]) + s2[2][t]) + s2[3][t];
  }
}

// The axes of the point order: cell = floor((x - lo) * inv), 256 cells over
// five standard deviations (the rest clamped).
struct Axes {
  int t[3];
  float inv[3];
  double lo[3];
};

__global__ void __launch_bounds__(1024)
mean_reduce(const double* __restrict__ part, const float* __restrict__ part2, int nparts, int64_t n, int d,
            const double* __restrict__ X, double* __restrict__ mean, Axes* __restrict__ axes) {
  __shared__ double s1[16][64];
  __shared__ float s2[16][64];
  const int t = threadIdx.x & 63, g = threadIdx.x >> 6;
  double s = 0.0;
  float v = 0.f;
  if (t < d)
    for (int b = g; b < nparts; b += 16) {
      s += part[b * 64 + t];
      v += part2[b * 64 + t];
    }
  s1[g][t] = s;
  s2[g][t] = v;
  __syncthreads();
  if (g == 0) {
    for (int i = 1; i < 16; ++i) {
      s += s1[i][t];
      v += s2[i][t];
    }
    s = t < d ? s / (double)n : 0.0;
    mean[t] = s;
    s1[0][t] = s;
    const float c = t < d ? (float)(s - X[t]) : 0.f;
    s2[0][t] = t < d ? fmaxf(v / (float)n - c * c, 0.f) : -1.f;  // variance
  }
  __syncthreads();
  if (threadIdx.x == 0 && axes) {
    for (int a = 0; a < 3; ++a) {
      int best = -1;
      for (int j = 0; j < d; ++j)
        if (s2[0][j] >= 0.f && (best < 0 || s2[0][j] > s2[0][best])) best = j;
      const float sd = best < 0 ? 0.f : sqrtf(s2[0][best]);
      axes->t[a] = best < 0 ? 0 : best;
      axes->lo[a] = best < 0 ? 0.0 : s1[0][best] - 2.5 * (double)sd;
      axes->inv[a] = sd > 0.f ? 256.f / (5.f * sd) : 0.f;
      if (best >= 0) s2[0][best] = -1.f;
    }
  }
}

// ---- point order ---------------------------------------------------------------
// A Morton code of the three axes of largest spread, eight bits each: points
// that follow one another are near in those axes, so that a 128-point tile
// has a tight box in them.  Of 100,000 clustered points in 30 dimensions half
// of the tile pairs can then be left out at the final tau, against none in
// input order; more axes make looser boxes (four: 64 % stay, a cut at the
// median of the widest axis: 56 %).
__device__ __forceinline__ uint32_t spread3(uint32_t x) {  // bits of an 8-bit value to every third place
  uint32_t r = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) r |= ((x >> i) & 1u) << (3 * i);
  return r;
}

__global__ void order_codes(const double* __restrict__ X, int64_t n, int d, const Axes* __restrict__ axes,
                            uint64_t* __restrict__ keys, uint64_t* __restrict__ vals) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t code = 0;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float c = (float)(X[i * d + axes->t[a]] - axes->lo[a]) * axes->inv[a];
    code |= spread3((uint32_t)fminf(fmaxf(c, 0.f), 255.f)) << (2 - a);
  }
  keys[i] = code;
  vals[i] = (uint64_t)i;
}

__global__ void order_perm(int64_t n, const uint64_t* __restrict__ vals, int* __restrict__ perm) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) perm[i] = (int)vals[i];
}

// X -> centred FP32 copy, tile-transposed for the filter scan (XT, zero
// beyond n up to the tile boundary), its FP32 squared norms, the padded FP64
// copy (uncentred: the re-rank uses the reference's arithmetic on the
// original coordinates) and the max centred row norm (float bits, rounded up).
// With `perm`, position i of XT and nrm holds point perm[i]; the FP64 copy
// stays in input order.
template <int DP>
__global__ void prep_kernel(const double* __restrict__ X, int64_t n, int d, const double* __restrict__ mean,
                            const int* __restrict__ perm, float* __restrict__ XT, float* __restrict__ nrm, double* __restrict__ X64,
                            unsigned* __restrict__ maxnorm_bits) {
  float mx = 0.f;
  const int64_t npad = (n + kFC - 1) / kFC * kFC;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < npad; i += (int64_t)gridDim.x * blockDim.x) {
    float* dst = XT + (i / kFC) * DP * kFC + (i % kFC);
    if (i >= n) {
      for (int t = 0; t < DP; ++t) dst[t * kFC] = 0.f;
      nrm[i] = __int_as_float(0x7f800000);  // never passes the filter
      continue;
    }
    const int64_t p = perm ? perm[i] : i;
    double s = 0.0, s32 = 0.0;
#pragma unroll 4
    for (int t = 0; t < DP; ++t) {
      const double v = t < d ? X[p * d + t] : 0.0;
      const double c = t < d ? v - mean[t] : 0.0;
      const float c32 = (float)c;
      dst[t * kFC] = c32;
      X64[p * DP + t] = v;
      s += c * c;
      s32 += (double)c32 * (double)c32;
    }
    nrm[i] = (float)s32;
    mx = fmaxf(mx, (float)sqrt(s) * 1.0000002f);
  }
  for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0) atomicMax(maxnorm_bits, __float_as_uint(mx));
}

// Write row q: the k (distance, index) pairs in kd[0..k) / ki[0..k) (any
// order) sorted by column index, distances sqrt'ed.  Uses kk/ks scratch.
__device__ void emit_row(int64_t q, int k, const double* kd, const int* kidx, double* kk, int* ks,
                         int64_t* __restrict__ nbr, double* __restrict__ dist) {
  const int lane = threadIdx.x & 31;
  for (int s = lane; s < kMaxKp; s += 32) {
    kk[s] = s < k ? (double)kidx[s] : DBL_MAX;
    ks[s] = s < k ? s : 0x7fffffff;
  }
  __syncwarp();
  warp_bitonic<double>(kk, ks, kMaxKp);
  for (int t = lane; t < k; t += 32) {
    nbr[q * k + t] = (int64_t)kk[t];
    dist[q * k + t] = sqrt(kd[ks[t]]);
  }
  __syncwarp();
}

// FP64 re-rank of the Kp FP32 candidates, eight queries per CTA.
//
// What bounds it is the FP64 pipe (two lanes per clock and SM, idle lanes
// included): 3 d instructions per candidate.  So the candidates of all eight
// queries are dealt over the threads together (66 per query fill 17 warps
// instead of 24), the certificate of all queries is one warp's work, square
// roots are taken by full warps, and everything else is integer: the order by
// (distance, index) is found by counting, on the distances' bits (they are
// not negative), instead of two bitonic sorts whose FP64 compares cost more
// than the distances.  100,000 queries of 66 candidates in 30 dimensions:
// 3.8 -> 1.34 ms, of which the distances cannot take less than 0.97.
constexpr int kRQ = 8;  // queries (and warps) per CTA
template <int DP>
__global__ void __launch_bounds__(256)
rerank_kernel(const double* __restrict__ X64, int64_t n, int d, const double* __restrict__ mean,
              const int* __restrict__ cand, int Kp, const float* __restrict__ tau32, int k,
              const unsigned* __restrict__ maxnorm_bits, int64_t* __restrict__ nbr, double* __restrict__ dist,
              int* __restrict__ flagged, int* __restrict__ nflag) {
  __shared__ __align__(16) double xq[kRQ][DP];
  __shared__ unsigned long long kd[kRQ][kMaxKp];  // distance bits
  __shared__ int kc[kRQ][kMaxKp];                 // index (0x7fffffff: none)
  __shared__ int pick[kRQ][kMaxKp];               // the k nearest, by rank
  __shared__ double qn2[kRQ], dk[kRQ];
  __shared__ int ok[kRQ];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t q0 = (int64_t)blockIdx.x * kRQ;
  const int nq = (int)(n - q0 < kRQ ? n - q0 : kRQ);
  for (int e = threadIdx.x; e < nq * DP; e += 256) xq[e / DP][e % DP] = X64[q0 * DP + e];
  __syncthreads();
  const unsigned long long none = ~0ull;
  for (int e = threadIdx.x; e < nq * Kp; e += 256) {
    const int q = e / Kp, s = e - q * Kp;
    const int c = cand[q0 * Kp + e];
    unsigned long long key = none;
    if (c >= 0) {
      const double2* xc = reinterpret_cast<const double2*>(X64 + (int64_t)c * DP);
      const double2* x = reinterpret_cast<const double2*>(xq[q]);
      // sequential, unfused sum of squares: the reference's squared_euclidean
      double dd = 0.0;
#pragma unroll 4
      for (int t = 0; t < (d >> 1); ++t) {
        const double2 a = x[t], b = __ldg(xc + t);
        const double df = __dsub_rn(a.x, b.x), dg = __dsub_rn(a.y, b.y);
        dd = __dadd_rn(dd, __dmul_rn(df, df));
        dd = __dadd_rn(dd, __dmul_rn(dg, dg));
      }
      if (d & 1) {
        const double df = __dsub_rn(xq[q][d - 1], X64[(int64_t)c * DP + d - 1]);
        dd = __dadd_rn(dd, __dmul_rn(df, df));
      }
      key = (unsigned long long)__double_as_longlong(dd);
    }
    kd[q][s] = key;
    kc[q][s] = c >= 0 ? c : 0x7fffffff;
  }
  if (w < nq) {  // squared centred norm of the warp's query
    double c = 0.0;
    for (int t = lane; t < d; t += 32) {
      const double v = xq[w][t] - mean[t];
      c = fma(v, v, c);
    }
    for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if (lane == 0) {
      qn2[w] = c;
      ok[w] = 0;
    }
  }
  __syncthreads();
  constexpr int E = kMaxKp / 32;
  unsigned long long key[E];
  int id[E], rank[E], pos[E];
  if (w < nq) {
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int s = e * 32 + lane;
      key[e] = s < Kp ? kd[w][s] : none;
      id[e] = s < Kp ? kc[w][s] : 0x7fffffff;
      rank[e] = pos[e] = 0;
    }
    const int used = (Kp + 31) / 32;
    for (int j = 0; j < Kp; ++j) {
      const unsigned long long kj = kd[w][j];
      const int ij = kc[w][j];
#pragma unroll
      for (int e = 0; e < E; ++e)
        if (e < used) rank[e] += kj < key[e] || (kj == key[e] && ij < id[e]);
    }
#pragma unroll
    for (int e = 0; e < E; ++e) {
      if (rank[e] < k && id[e] != 0x7fffffff) {
        pick[w][rank[e]] = id[e];
        if (rank[e] == k - 1) {  // one candidate: ranks of real candidates differ
          dk[w] = __longlong_as_double((long long)key[e]);
          ok[w] = 1;
        }
      }
    }
  }
  __syncthreads();
  // Certificate.  Every point j outside the list has FP32 distance
  // d32(j) >= tau32.  With u = 2^-24, N = |x_q - mean| + max_j |x_j - mean|
  // and D the exact squared distance, rounding the centred coordinates to FP32
  // and the FP32 fused sum of squares give
  //   |d32 - D| <= 4.1 u N sqrt(D) + (d+1) u D + 5 u^2 N^2,
  // so every outside point has D >= L, the positive root bound of
  //   (1 + (d+1)u) s^2 + 4.1 u N s - (tau32 - 5 u^2 N^2) >= 0,  D = s^2.
  // If L exceeds the k-th FP64 distance among the candidates, the FP64 top-k
  // is exact.
  if (threadIdx.x < nq && ok[threadIdx.x]) {
    const int64_t q = q0 + threadIdx.x;
    const double u = 5.9604644775390625e-08;
    const double N = sqrt(qn2[threadIdx.x]) + (double)__uint_as_float(*maxnorm_bits);
    const double t32 = (double)tau32[q];
    const double qa = 1.0 + (double)(d + 1) * u, qb = 4.1 * u * N, qc = t32 - 5.0 * u * u * N * N;
    const double sroot = qc > 0.0 ? (-qb + sqrt(qb * qb + 4.0 * qa * qc)) / (2.0 * qa) : 0.0;
    const double lower = sroot * sroot * (1.0 - 4.0 * u);  // absorb the rounding of this bound itself
    const bool all_seen = t32 >= 3.0e38;  // fewer than Kp points: every point is a candidate
    if (!(all_seen || lower > dk[threadIdx.x])) ok[threadIdx.x] = 0;
  }
  __syncthreads();
  if (threadIdx.x < nq && !ok[threadIdx.x]) flagged[atomicAdd(nflag, 1)] = (int)(q0 + threadIdx.x);
  // rows by column index: a picked candidate's place is the number of picked ones below it
  if (w < nq && ok[w]) {
    for (int j = 0; j < k; ++j) {
      const int ij = pick[w][j];
#pragma unroll
      for (int e = 0; e < E; ++e) pos[e] += ij < id[e];
    }
  }
  __syncthreads();
  if (w < nq && ok[w]) {
#pragma unroll
    for (int e = 0; e < E; ++e)
      if (rank[e] < k && id[e] != 0x7fffffff) {
        kd[w][pos[e]] = key[e];
        kc[w][pos[e]] = id[e];
      }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < nq * k; e += 256) {
    const int q = e / k, t = e - q * k;
    if (!ok[q]) continue;
    nbr[q0 * k + e] = kc[q][t];
    dist[q0 * k + e] = sqrt(__longlong_as_double((long long)kd[q][t]));
  }
}

// Rows of the queries that the certificate rejected, from the exact FP64 scan.
__global__ void __launch_bounds__(256)
finalize_kernel(const int* __restrict__ flagged, const int* __restrict__ nflag, const int* __restrict__ cand,
                const double* __restrict__ cand_d, int k, int64_t* __restrict__ nbr, double* __restrict__ dist) {
  __shared__ double kd[8][kMaxKp];
  __shared__ int kc[8][kMaxKp];
  __shared__ double tk[8][kMaxKp];
  __shared__ int ts[8][kMaxKp];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t slot = (int64_t)blockIdx.x * 8 + w;
  if (slot >= *nflag) return;
  const int64_t q = flagged[slot];
  for (int s = lane; s < k; s += 32) {
    kd[w][s] = cand_d[slot * k + s];
    kc[w][s] = cand[slot * k + s];
  }
  __syncwarp();
  emit_row(q, k, kd[w], kc[w], tk[w], ts[w], nbr, dist);
}

__global__ void zero_int(int* p, unsigned* u) {
  *p = 0;
  *u = 0u;
}

struct KnnScratch {
  double* mpart;
  double* mean;
  float* XT;
  float* nrm;
  unsigned char* TC;  // tensor-core operand tiles (ordered, DP == 32)
  double* X64;
  int* cand;
  float* tau32;
  int* flagged;
  int* fcand;
  double* fcand_d;
  int* nflag;
  unsigned* maxnorm;
  float* mpart2;
  Axes* axes;
  // point order and tile boxes (nullptr below kOrderMin points)
  int* perm;
  uint64_t *keys, *vals, *keys_alt, *vals_alt;
  void* radix;
  float* box;
  int64_t bytes;
};

// Points from which the filter works on an ordered copy (and, up to 32
// dimensions, on the tensor cores with 128 queries per CTA).  Below, such CTAs
// are too few for the 152 SMs and 32 queries per CTA in input order are
// faster: 16,000 points 1.57 ms, 12,000 1.10, 5,000 0.44, 2,500 0.25, where
// the tensor-core filter took 1.04 for its one wave of 20 CTAs; 20,000 points
// take 1.40 ms on the tensor cores and 1.68 without.
constexpr int64_t kOrderMin = 16385;

constexpr int64_t align256(int64_t x) { return (x + 255) / 256 * 256; }

// Byte offsets of the scratch regions (each 256-byte aligned) and the total;
// constexpr so that the allocation-free entry point can size its fixed array
// from the same arithmetic.
struct KnnOffsets {
  int64_t mp, mean, XT, nrm, TC, X64, cand, tau, flagged, fcand, fcand_d, counters, mp2, axes, perm, sort, radix, box,
      bytes;
};

// `radix` = radix_scratch_bytes(n) where the points are ordered (n >= kOrderMin)
constexpr KnnOffsets knn_offsets(int64_t n, int DP, int k, int Kp, int64_t radix) {
  KnnOffsets o{};
  int64_t at = 0;
  const int64_t npad = (n + kFC - 1) / kFC * kFC;
  o.mp = at; at += align256((int64_t)kMeanParts * 64 * 8);
  o.mean = at; at += align256(64 * 8);
  o.XT = at; at += align256(npad * DP * 4);
  o.nrm = at; at += align256(npad * 4);
  const bool ordered = n >= kOrderMin;
  o.TC = at; at += DP == 32 && ordered ? align256(npad / kFC * kTTile) : 0;
  o.X64 = at; at += align256(n * DP * 8);
  o.cand = at; at += align256(n * (int64_t)Kp * 4);
  o.tau = at; at += align256(n * 4);
  o.flagged = at; at += align256(n * 4);
  o.fcand = at; at += align256(n * (int64_t)k * 4);
  o.fcand_d = at; at += align256(n * (int64_t)k * 8);
  o.counters = at; at += align256(16);
  o.mp2 = at; at += align256((int64_t)kMeanParts * 64 * 4);
  o.axes = at; at += align256(sizeof(Axes));
  o.perm = at; at += ordered ? align256(n * 4) : 0;
  o.sort = at; at += ordered ? 4 * align256(n * 8) : 0;
  o.radix = at; at += ordered ? align256(radix) : 0;
  o.box = at; at += DP == 32 && ordered ? (npad / kFC + 31) / 32 * 2 * kTDim * 32 * 4 : 0;
  o.bytes = at;
  return o;
}

KnnScratch knn_layout(char* base, int64_t n, int DP, int k, int Kp) {
  const bool ordered = n >= kOrderMin;
  const KnnOffsets o = knn_offsets(n, DP, k, Kp, ordered ? radix_scratch_bytes(n) : 0);
  KnnScratch s{};
  if (base) {
    s.mpart = (double*)(base + o.mp);
    s.mean = (double*)(base + o.mean);
    s.XT = (float*)(base + o.XT);
    s.nrm = (float*)(base + o.nrm);
    s.TC = DP == 32 && ordered ? (unsigned char*)(base + o.TC) : nullptr;
    s.X64 = (double*)(base + o.X64);
    s.cand = (int*)(base + o.cand);
    s.tau32 = (float*)(base + o.tau);
    s.flagged = (int*)(base + o.flagged);
    s.fcand = (int*)(base + o.fcand);
    s.fcand_d = (double*)(base + o.fcand_d);
    s.nflag = (int*)(base + o.counters);
    s.maxnorm = (unsigned*)(base + o.counters + 8);
    s.mpart2 = (float*)(base + o.mp2);
    s.axes = (Axes*)(base + o.axes);
    if (ordered) {
      const int64_t b = align256(n * 8);
      s.perm = (int*)(base + o.perm);
      s.keys = (uint64_t*)(base + o.sort);
      s.vals = (uint64_t*)(base + o.sort + b);
      s.keys_alt = (uint64_t*)(base + o.sort + 2 * b);
      s.vals_alt = (uint64_t*)(base + o.sort + 3 * b);
      s.radix = base + o.radix;
      s.box = DP == 32 ? (float*)(base + o.box) : nullptr;
    }
  }
  s.bytes = o.bytes;
  return s;
}

// 16 dimensions are padded to the 32 of the tensor-core filter where that one runs
inline int pad_dim(int d, int64_t n) { return d <= 16 && n < kOrderMin ? 16 : (d <= 32 ? 32 : 64); }

template <typename TD, int DP>
int launch_scan(const TD* Xp, int64_t n, const int* qlist, const int* qcount, int Kp, int* cand, TD* cand_d,
                TD* tau, cudaStream_t s) {
  const size_t smem = sizeof(ScanSmem<TD, DP>);
  if (cudaFuncSetAttribute(scan_kernel<TD, DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
      cudaSuccess)
    return SG_ERR_CUDA;
  const int64_t grid = (n + kQT - 1) / kQT;
  scan_kernel<TD, DP><<<(unsigned)grid, kLW * 32, smem, s>>>(Xp, n, qlist, qcount, Kp, cand, cand_d, tau);
  return cudaGetLastError() == cudaSuccess ? SG_OK : SG_ERR_CUDA;
}

template <int DP, int LIST>
int launch_filter_scan_l(const float* XT, const float* nrm, int64_t n, int d, int Kp, const int* perm, int* cand,
                         float* tau, cudaStream_t s) {
  const size_t smem = sizeof(FilterSmem<DP, LIST>);
  if (cudaFuncSetAttribute(filter_scan_kernel<DP, LIST>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
      cudaSuccess)
    return SG_ERR_CUDA;
  const int64_t grid = (n + kFQ - 1) / kFQ;
  filter_scan_kernel<DP, LIST><<<(unsigned)grid, kFW * 32, smem, s>>>(XT, nrm, n, d, Kp, perm, cand, tau);
  return cudaGetLastError() == cudaSuccess ? SG_OK : SG_ERR_CUDA;
}

template <int DP>
int launch_filter_scan(const float* XT, const float* nrm, int64_t n, int d, int Kp, const int* perm, int* cand,
                       float* tau, cudaStream_t s) {
  if (Kp + 32 <= 128) return launch_filter_scan_l<DP, 128>(XT, nrm, n, d, Kp, perm, cand, tau, s);
  return launch_filter_scan_l<DP, 256>(XT, nrm, n, d, Kp, perm, cand, tau, s);
}

// The tensor-core filter serves up to 32 dimensions and matrices that give
// every SM a CTA of 128 queries (kOrderMin);
// SNAPGB300_KNN_FILTER=simt selects the FP32 filter (both give the same
// candidate lists).
bool use_tensor_filter(int DP, int64_t n) {
  if (DP != 32 || n < kOrderMin) return false;
  const char* e = getenv("SNAPGB300_KNN_FILTER");
  return !(e && strcmp(e, "simt") == 0);
}

int launch_tc_filter(const unsigned char* TC, const float* nrm, const float* box, int64_t n, int d,
                     int Kp, const int* perm, int* cand, float* tau, cudaStream_t s) {
  // the cap is set to its largest value: calls of other sizes may run concurrently
  const int nbuf = tc_buffers(Kp);
  const auto kern = nbuf == 4 ? tc_filter_kernel<4> : (nbuf == 3 ? tc_filter_kernel<3> : tc_filter_kernel<2>);
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTSmemMax) != cudaSuccess)
    return SG_ERR_CUDA;
  const size_t smem = tc_smem_bytes(Kp, nbuf);
  const int64_t grid = (n + kTQ - 1) / kTQ;
  kern<<<(unsigned)grid, kTThreads, smem, s>>>(TC, nrm, box, n, d, Kp, perm, cand, tau);
  return cudaGetLastError() == cudaSuccess ? SG_OK : SG_ERR_CUDA;
}

template <int DP>
int knn_run(const double* X, int64_t n, int d, int k, int Kp, const KnnScratch& w, int64_t* nbr, double* dist,
            cudaStream_t s) {
  zero_int<<<1, 1, 0, s>>>(w.nflag, w.maxnorm);
  mean_partial<<<kMeanParts, 256, 0, s>>>(X, n, d, w.mpart, w.mpart2);
  mean_reduce<<<1, 1024, 0, s>>>(w.mpart, w.mpart2, kMeanParts, n, d, X, w.mean, w.axes);
  SG_CHECK_LAUNCH();
  if (w.perm) {
    const unsigned g = (unsigned)((n + 255) / 256);
    order_codes<<<g, 256, 0, s>>>(X, n, d, w.axes, w.keys, w.vals);
    SG_CHECK_LAUNCH();
    bool alt = false;
    if (radix_sort_u64(n, w.keys, w.vals, w.keys_alt, w.vals_alt, 0, 24, w.radix, s, &alt) != cudaSuccess)
      return SG_ERR_CUDA;
    order_perm<<<g, 256, 0, s>>>(n, alt ? w.vals_alt : w.vals, w.perm);
    SG_CHECK_LAUNCH();
  }
  prep_kernel<DP><<<grid_for(n, 256, 4096), 256, 0, s>>>(X, n, d, w.mean, w.perm, w.XT, w.nrm, w.X64, w.maxnorm);
  SG_CHECK_LAUNCH();
  int e;
  if (use_tensor_filter(DP, n)) {
    const int64_t ntiles = (n + kFC - 1) / kFC;
    tc_prep_kernel<<<grid_for(n, 256, 4096), 256, 0, s>>>(w.XT, w.nrm, n, w.TC);
    tile_box_kernel<<<(unsigned)((ntiles + 31) / 32 * 32), 128, 0, s>>>(w.XT, n, ntiles, w.box);
    SG_CHECK_LAUNCH();
    e = launch_tc_filter(w.TC, w.nrm, w.box, n, d, Kp, w.perm, w.cand, w.tau32, s);
  } else {
    e = launch_filter_scan<DP>(w.XT, w.nrm, n, d, Kp, w.perm, w.cand, w.tau32, s);
  }
  if (e) return e;
  rerank_kernel<DP><<<(unsigned)((n + kRQ - 1) / kRQ), 256, 0, s>>>(w.X64, n, d, w.mean, w.cand, Kp, w.tau32, k,
                                                            w.maxnorm, nbr, dist, w.flagged, w.nflag);
  SG_CHECK_LAUNCH();
  // exact FP64 scan of the rejected queries (CTAs past the count exit at once)
  e = launch_scan<double, DP>(w.X64, n, w.flagged, w.nflag, k, w.fcand, w.fcand_d, nullptr, s);
  if (e) return e;
  finalize_kernel<<<(unsigned)((n + 7) / 8), 256, 0, s>>>(w.flagged, w.nflag, w.fcand, w.fcand_d, k, nbr, dist);
  SG_CHECK_LAUNCH();
  return SG_OK;
}

}  // namespace
}  // namespace sg

using namespace sg;

extern "C" int64_t sg_knn_scratch_bytes(int64_t n, int d, int k, int margin) {
  if (n <= 0 || d <= 0 || d > 64 || k <= 0 || margin < 0) return -1;
  const int Kp = k + margin;
  return knn_layout(nullptr, n, pad_dim(d, n), k, Kp).bytes;
}

extern "C" int sg_knn(const double* X, int64_t n, int d, int k, int margin, int64_t* nbr, double* dist,
                      void* scratch, int64_t scratch_bytes, int* n_fallback, void* stream) {
  if (n < 2 || d <= 0 || d > 64 || k <= 0 || k > n - 1 || margin < 0 || n > 0x7fffffffLL) return SG_ERR_ARG;
  int Kp = k + margin;
  if (Kp > kMaxKp) Kp = kMaxKp;
  if (Kp > n - 1) Kp = (int)(n - 1);
  if (k > Kp) return SG_ERR_ARG;
  if (((uintptr_t)scratch & 255u) != 0) return SG_ERR_ARG;
  const int DP = pad_dim(d, n);
  KnnScratch w = knn_layout((char*)scratch, n, DP, k, k + margin);
  if (scratch_bytes < w.bytes) return SG_ERR_CAP;
  cudaStream_t s = as_stream(stream);
  int e;
  if (DP == 16) e = knn_run<16>(X, n, d, k, Kp, w, nbr, dist, s);
  else if (DP == 32) e = knn_run<32>(X, n, d, k, Kp, w, nbr, dist, s);
  else e = knn_run<64>(X, n, d, k, Kp, w, nbr, dist, s);
  if (e) return e;
  if (n_fallback &&
      cudaMemcpyAsync(n_fallback, w.nflag, sizeof(int), cudaMemcpyDeviceToDevice, s) != cudaSuccess)
    return SG_ERR_CUDA;
  return SG_OK;
}

// ---------------------------------------------------------------------------
// Allocation-free variant of sg_knn.
//
// Some callers cannot allocate device memory for the scratch sg_knn needs:
// an application whose device memory is owned by its own pool or framework
// (raw cudaMalloc is not allowed there), or a latency-bound caller for whom
// cudaMalloc, which may synchronise the whole device and is slow, is not an
// option.  For them the scratch lives in the fixed array below, which is part
// of this library's device image: every GPU that loads the library holds it
// (about 33 MB) until the process exits.
// ---------------------------------------------------------------------------
namespace sg {
namespace {

constexpr int64_t kNoAllocMaxN = 16384;  // points
constexpr int kNoAllocMaxDim = 32;       // dimensions
constexpr int kNoAllocMaxK = 100;        // neighbours
// sized by the scratch layout of the largest accepted problem: 16,384
// points (whole 128-point tiles), 32 dimensions (the tensor-core operand
// tiles are included), k = 100, candidate lists of kMaxKp
static_assert(kNoAllocMaxN < kOrderMin, "the point order needs scratch that the fixed array does not hold");
static_assert(kNoAllocMaxN % kFC == 0, "no-alloc capacity must be whole tiles");
constexpr int64_t kNoAllocBytes = knn_offsets(kNoAllocMaxN, kNoAllocMaxDim, kNoAllocMaxK, kMaxKp, 0).bytes;

static __device__ __align__(256) unsigned char g_knn_scratch[kNoAllocBytes];

// Device address of g_knn_scratch on the current device.  In host code the
// name g_knn_scratch is only a host-side stand-in, so the address is looked
// up with the device current and the return code checked.  The lookup is
// repeated on every call (it is a table lookup in the CUDA runtime): a cached
// address would go stale when the device's context is destroyed and made
// again (cudaDeviceReset), which reloads the module at a new address.  The
// first lookup on a device loads the module that holds the array (CUDA's
// lazy module loading).
int knn_scratch_address(void** out) {
  void* p = nullptr;
  if (cudaGetSymbolAddress(&p, g_knn_scratch) != cudaSuccess || !p) return SG_ERR_CUDA;
  *out = p;
  return SG_OK;
}

}  // namespace
}  // namespace sg

extern "C" int sg_knn_noalloc(const double* X, int64_t n, int d, int k, int margin, int64_t* nbr, double* dist,
                              int* n_fallback, void* stream) {
  if (n < 2 || d <= 0 || k <= 0 || k > n - 1 || margin < 0) return SG_ERR_ARG;
  if (n > kNoAllocMaxN || d > kNoAllocMaxDim || k > kNoAllocMaxK) return SG_ERR_CAP;
  if (k + margin > kMaxKp) margin = kMaxKp - k;
  int Kp = k + margin;
  if (Kp > n - 1) Kp = (int)(n - 1);
  void* base = nullptr;
  int e = knn_scratch_address(&base);
  if (e) return e;
  const int DP = pad_dim(d, n);
  KnnScratch w = knn_layout((char*)base, n, DP, k, k + margin);
  if (w.bytes > kNoAllocBytes) return SG_ERR_CAP;
  cudaStream_t s = as_stream(stream);
  // knn_run clears the two counters it accumulates into (fallback count,
  // max norm) before use; every other scratch byte is written before read.
  e = DP == 16 ? knn_run<16>(X, n, d, k, Kp, w, nbr, dist, s) : knn_run<32>(X, n, d, k, Kp, w, nbr, dist, s);
  if (e) return e;
  if (n_fallback &&
      cudaMemcpyAsync(n_fallback, w.nflag, sizeof(int), cudaMemcpyDeviceToDevice, s) != cudaSuccess)
    return SG_ERR_CUDA;
  return SG_OK;
}
