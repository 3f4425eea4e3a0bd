// Fragment-file import (snap.pp.import_fragments) on the GPU.
//
// Input: the decompressed text of a fragment file in device memory.  Output:
// the per-cell fragment matrix of the reference (rows = cells, column = global
// base index of the fragment start, value = fragment size; signed size for
// single-end reads) plus the per-cell QC columns.  Reference:
// snapatac2-python/src/preprocessing.rs:87-184 (entry, shifts, unsorted
// input) and snapatac2-core/src/preprocessing/import.rs:31-210 (grouping,
// QC, per-cell sort), record syntax qc.rs:303-348.
//
// Pipeline (one CUDA stream; the host reads back a handful of sizes):
//   lines     newline count per 64 KB chunk, scan, line starts;
//   parse     thread per line: fields, saturating shifts, chromosome by
//             binary search over the sorted names, global position and
//             signed size, 64-bit barcode hash (SplitMix64 finaliser over
//             8-byte words), flags;
//   group     records with a barcode entered into a hash table (its size
//             grows until every barcode finds a place); every record's
//             barcode is compared byte for byte with that of its slot's first
//             record (a collision re-hashes with another seed), group ids by
//             a scan of the table, per-group counts by atomics;
//   decide    whitelist (hash + byte compare), the minimum-count whitelist
//             of unsorted input, the "sorted by barcode" check (a group's
//             records must be one run), position and size-conversion errors
//             of processed groups, the minimum-fragment filter;
//   order     kept groups by first appearance (sorted input) or by barcode
//             bytes: by counting up to kRankGroups groups of up to 64 bytes,
//             else by LSD radix (over length, then 8-byte big-endian words);
//   matrix    kept in-genome records keyed (cell, position, size), brought
//             into order (see order_matrix) and decoded into CSR order.
#include "common.cuh"
#include "internal.h"

#include <algorithm>

namespace sg {
namespace {

enum : uint16_t {
  F_REC = 1,        // a record (not a comment line)
  F_LEN = 2,        // end != start after the shifts
  F_GEN = 4,        // chromosome present in the genome
  F_MITO = 8,       // mitochondrial chromosome
  F_BC = 16,        // barcode present (not ".")
  F_REV = 32,       // strand "-"
  F_STRANDED = 64,  // strand column present and not "."
  F_POSERR = 128,   // position outside its chromosome
  F_FITU32 = 256,   // signed size in [0, 2^32)
  F_FITI32 = 512,   // signed size in [-2^31, 2^31)
};

constexpr int kThreads = 256;
constexpr int64_t kChunk = 64 * 1024;  // bytes of text per CTA in the line index

// ---- hashing ---------------------------------------------------------------
// SplitMix64 output function (Steele, Lea & Flood, "Fast splittable
// pseudorandom number generators", 2014), used as a 64-bit mixer.
__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}

struct Hasher {
  uint64_t h, w;
  int nb;
  int64_t len;
  __device__ explicit Hasher(uint64_t seed) : h(mix64(seed ^ 0x6a09e667f3bcc909ull)), w(0), nb(0), len(0) {}
  __device__ __forceinline__ void push(uint8_t b) {
    w |= (uint64_t)b << (8 * nb);
    ++len;
    if (++nb == 8) {
      h = mix64(h ^ w);
      w = 0;
      nb = 0;
    }
  }
  __device__ __forceinline__ uint64_t finish() {
    if (nb) h = mix64(h ^ w);
    return mix64(h ^ ((uint64_t)len * 0x9e3779b97f4a7c15ull));
  }
};

__device__ __forceinline__ uint64_t hash_bytes(const uint8_t* p, int64_t n, uint64_t seed) {
  Hasher hs(seed);
  for (int64_t i = 0; i < n; ++i) hs.push(p[i]);
  return hs.finish();
}

// barcode location: byte offset << 16 | length (length < 65536)
__device__ __forceinline__ int64_t loc_off(uint64_t l) { return (int64_t)(l >> 16); }
__device__ __forceinline__ int loc_len(uint64_t l) { return (int)(l & 0xFFFF); }

__device__ __forceinline__ bool bytes_equal(const uint8_t* a, const uint8_t* b, int n) {
  for (int i = 0; i < n; ++i)
    if (a[i] != b[i]) return false;
  return true;
}

__device__ __forceinline__ void set_error(int* status, unsigned long long* bad, int code, int64_t line) {
  atomicCAS(status, 0, code);
  atomicMin(bad, (unsigned long long)line);
}

// ---- line index ------------------------------------------------------------
__device__ __forceinline__ int nl_in_word(uint32_t x) { return __popc(__vcmpeq4(x, 0x0a0a0a0au)) >> 3; }

__global__ void __launch_bounds__(kThreads) line_count_kernel(const uint8_t* __restrict__ text, int64_t nbytes,
                                                              int64_t* __restrict__ counts) {
  const int64_t c = blockIdx.x, b0 = c * kChunk;
  const int64_t b1 = b0 + kChunk < nbytes ? b0 + kChunk : nbytes;
  int n = 0;
  const int64_t nvec = (b1 - b0) / 16;
  const uint4* v = reinterpret_cast<const uint4*>(text + b0);
  for (int64_t i = threadIdx.x; i < nvec; i += kThreads) {
    const uint4 q = __ldg(v + i);
    n += nl_in_word(q.x) + nl_in_word(q.y) + nl_in_word(q.z) + nl_in_word(q.w);
  }
  for (int64_t p = b0 + nvec * 16 + threadIdx.x; p < b1; p += kThreads) n += text[p] == '\n';
  __shared__ int ws[kThreads / 32];
#pragma unroll
  for (int o = 16; o; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = n;
  __syncthreads();
  if (threadIdx.x == 0) {
    int t = 0;
    for (int i = 0; i < kThreads / 32; ++i) t += ws[i];
    counts[1 + c] = t;
    if (c == 0) counts[0] = 0;
  }
}

// bit j: byte j of the 16 is a newline
__device__ __forceinline__ uint32_t nl_bits(const uint4& q) {
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
  uint32_t m = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) m |= (((__vcmpeq4(w[j], 0x0a0a0a0au) & 0x01010101u) * 0x01020408u) >> 24) << (4 * j);
  return m;
}

// line_start[k + 1] = 1 + position of the k-th newline; line_start[0] = 0.
// 64 bytes per thread and step as a bit mask of its newlines: of 45 bytes one
// is a newline, so there is next to nothing to do but the two reads of the
// text (0.83 GB: 0.13 ms to count, 0.15 here; a loop over the bytes took
// 0.46).
constexpr int kFillBytes = 64;

__global__ void __launch_bounds__(kThreads) line_fill_kernel(const uint8_t* __restrict__ text, int64_t nbytes,
                                                             const int64_t* __restrict__ before, int64_t n_lines,
                                                             int64_t* __restrict__ line_start) {
  const int64_t c = blockIdx.x, b0 = c * kChunk;
  const int64_t b1 = b0 + kChunk < nbytes ? b0 + kChunk : nbytes;
  __shared__ int wsum[2][kThreads / 32];
  int64_t base = before[c];  // newlines before this chunk
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const bool wide = ((uintptr_t)text & 15) == 0;  // p0 is a multiple of 16
  int turn = 0;
  for (int64_t r0 = b0; r0 < b1; r0 += kFillBytes * kThreads, turn ^= 1) {
    const int64_t p0 = r0 + kFillBytes * (int64_t)threadIdx.x;
    uint64_t m = 0;
    if (wide && p0 + kFillBytes <= b1) {
#pragma unroll
      for (int v = 0; v < kFillBytes / 16; ++v)
        m |= (uint64_t)nl_bits(__ldg(reinterpret_cast<const uint4*>(text + p0) + v)) << (16 * v);
    } else {
      for (int j = 0; j < kFillBytes && p0 + j < b1; ++j) m |= (uint64_t)(text[p0 + j] == '\n') << j;
    }
    const int n = __popcll(m);
    int x = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) wsum[turn][w] = x;
    __syncthreads();
    int off = 0, tot = 0;
#pragma unroll
    for (int i = 0; i < kThreads / 32; ++i) {
      off += i < w ? wsum[turn][i] : 0;
      tot += wsum[turn][i];
    }
    int64_t k = base + off + x - n;
    for (; m; m &= m - 1) line_start[1 + k++] = p0 + __ffsll((long long)m);
    base += tot;
  }
  if (c == 0 && threadIdx.x == 0) {
    line_start[0] = 0;
    // an unterminated last line ends at nbytes: its "next start" is nbytes + 1
    if (n_lines > 0 && text[nbytes - 1] != '\n') line_start[n_lines] = nbytes + 1;
  }
}

// ---- parse -----------------------------------------------------------------
struct ChromTable {
  const uint8_t* blob;    // names, concatenated, sorted by bytes
  const int64_t* off;     // n + 1 offsets into blob
  const uint64_t* size;   // chromosome length
  const uint64_t* base;   // cumulative length before the chromosome
  const uint8_t* mito;    // 1 for mitochondrial names
  const uint64_t* pk;     // first 8 bytes of each name, big-endian, zero padded
  int n;
};
constexpr int kMaxChroms = 1 << 16;

__global__ void chrom_pack(ChromTable ct, uint64_t* __restrict__ pk) {
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < ct.n; c += gridDim.x * blockDim.x) {
    const int64_t o = ct.off[c], n = ct.off[c + 1] - o;
    uint64_t k = 0;
    for (int j = 0; j < 8; ++j) k = (k << 8) | (j < n ? ct.blob[o + j] : 0u);
    pk[c] = k;
  }
}

// Chromosome of a name given as (first 8 bytes big-endian, length, bytes).
// Names compare by bytes; (packed prefix, length) orders them the same way
// unless both names are longer than 8 bytes and share the prefix, where the
// remaining bytes decide.
__device__ int find_chrom(const ChromTable& ct, uint64_t qk, int64_t qlen, const uint8_t* q) {
  int lo = 0, hi = ct.n - 1;
  while (lo <= hi) {
    const int mid = (lo + hi) >> 1;
    const uint64_t k = ct.pk[mid];
    const int64_t o = ct.off[mid], len = ct.off[mid + 1] - o;
    int c;
    if (qk != k) {
      c = qk < k ? -1 : 1;
    } else if (qlen > 8 && len > 8) {
      c = 0;
      const int64_t m = qlen < len ? qlen : len;
      for (int64_t j = 8; j < m && c == 0; ++j) {
        const uint8_t x = q[j], y = ct.blob[o + j];
        if (x != y) c = x < y ? -1 : 1;
      }
      if (c == 0) c = qlen < len ? -1 : (qlen > len ? 1 : 0);
    } else {
      c = qlen < len ? -1 : (qlen > len ? 1 : 0);
    }
    if (c == 0) return mid;
    if (c < 0) hi = mid - 1;
    else lo = mid + 1;
  }
  return -1;
}

__device__ __forceinline__ uint64_t sat_add(uint64_t x, int64_t s) {
  if (s >= 0) return x > UINT64_MAX - (uint64_t)s ? UINT64_MAX : x + (uint64_t)s;
  const uint64_t m = (uint64_t)(-(s + 1)) + 1;  // |s| without overflow
  return x < m ? 0 : x - m;
}

struct ParseOut {
  uint64_t* hash;
  uint64_t* loc;
  int64_t* pos;
  int64_t* val;
  uint32_t* cnt;
  uint16_t* flags;
};

// decimal digits into an unsigned accumulator; `ok` turns false on a
// non-digit or on overflow of 64 bits
__device__ __forceinline__ void push_digit(uint64_t& v, bool& ok, uint8_t c) {
  const uint32_t d = (uint32_t)c - '0';
  if (d > 9 || v > (UINT64_MAX - d) / 10) ok = false;
  else v = v * 10 + d;
}

// The fields of one line: chrom, start, end, barcode, count, strand.
struct Fields {
  int f;                        // tabs seen (6: the rest of the line is not looked at)
  uint64_t ck, start, end, cnt; // first bytes of the chromosome (big-endian), numbers
  int clen, len1, len2, len4, blen, slen;
  int bstart;               // offset of the barcode from the line's start
  bool ok1, ok2, ok4;           // the numbers are digits only and fit 64 bits
  uint8_t b0, c4, sc;           // first byte of barcode and count, last of the strand
  uint64_t h;                   // barcode hash
};

// byte by byte, from global memory (lines too long to be staged)
__device__ void fields_bytes(const uint8_t* __restrict__ text, int64_t s, int64_t e, uint64_t seed, Fields& r) {
  int f = 0;
  r.ck = r.start = r.end = r.cnt = 0;
  r.clen = r.len1 = r.len2 = r.len4 = r.blen = r.slen = r.bstart = 0;
  r.ok1 = r.ok2 = r.ok4 = true;
  r.b0 = r.c4 = r.sc = 0;
  Hasher hs(seed);
  for (int64_t p = s; p < e; ++p) {
    const uint8_t c = text[p];
    if (c == '\t') {
      if (++f == 6) break;
      if (f == 3) r.bstart = (int)(p + 1 - s);
      continue;
    }
    switch (f) {
      case 0:
        if (r.clen < 8) r.ck |= (uint64_t)c << (56 - 8 * r.clen);
        ++r.clen;
        break;
      case 1: ++r.len1; push_digit(r.start, r.ok1, c); break;
      case 2: ++r.len2; push_digit(r.end, r.ok2, c); break;
      case 3:
        if (r.blen == 0) r.b0 = c;
        hs.push(c);
        ++r.blen;
        break;
      case 4:
        if (r.len4 == 0) r.c4 = c;
        ++r.len4;
        push_digit(r.cnt, r.ok4, c);
        break;
      default:
        r.sc = c;
        ++r.slen;
        break;
    }
  }
  r.f = f;
  r.h = hs.finish();
}

// 4 and 8 bytes at any byte offset of the staged text (words past the line are
// inside the staging buffer)
__device__ __forceinline__ uint32_t staged4(const uint32_t* st, int o) {
  return __funnelshift_r(st[o >> 2], st[(o >> 2) + 1], 8 * (o & 3));
}
__device__ __forceinline__ uint64_t staged8(const uint32_t* st, int o) {
  const uint32_t a = st[o >> 2], b = st[(o >> 2) + 1], c = st[(o >> 2) + 2];
  const int sh = 8 * (o & 3);
  return (uint64_t)__funnelshift_r(a, b, sh) | ((uint64_t)__funnelshift_r(b, c, sh) << 32);
}

// a decimal number of n bytes; ok: digits only and below 2^64
__device__ __forceinline__ uint64_t staged_number(const uint32_t* st, int o, int n, bool& ok) {
  uint64_t v = 0;
  ok = true;
  if (n > 18) {  // could overflow: one digit at a time
    for (int i = 0; i < n; ++i) push_digit(v, ok, (uint8_t)(st[(o + i) >> 2] >> (8 * ((o + i) & 3))));
    return v;
  }
  for (int i = 0; i < n; i += 4) {  // four digits at a time: 1000 a + 100 b + 10 c + d
    const int k = n - i < 4 ? n - i : 4;
    uint32_t x = staged4(st, o + i);
    x = k == 4 ? x : (x << (32 - 8 * k)) | (0x30303030u >> (8 * k));  // leading zeros in front of a short piece
    const uint32_t d = x - 0x30303030u;
    // a byte below '0' borrows into its top bit (or its neighbour's); one above '9' carries past 0x7f with + 0x76
    ok = ok && ((x & 0xf0f0f0f0u) == 0x30303030u) && (((d + 0x76767676u) & 0x80808080u) == 0);
    const uint32_t lo = (d & 0xff) * 1000 + ((d >> 8) & 0xff) * 100 + ((d >> 16) & 0xff) * 10 + (d >> 24);
    v = v * (k == 4 ? 10000u : (k == 3 ? 1000u : (k == 2 ? 100u : 10u))) + lo;
  }
  return v;
}

// the same from the staged text, in words: tabs by a byte compare of four
// bytes at a time, numbers by four digits, the barcode's hash by eight bytes
__device__ __forceinline__ void fields_staged(const uint32_t* __restrict__ st, int s, int e, uint64_t h0,
                                              Fields& r) {
  int tab[6];
  int f = 0;
  const int o0 = s & ~3;
  if (e - o0 <= 64) {  // one bit per byte: the lanes of a warp stay together whatever their fields' lengths
    uint64_t m = 0;
    for (int o = o0; o < e; o += 4)
      m |= (uint64_t)(((__vcmpeq4(st[o >> 2], 0x09090909u) & 0x01010101u) * 0x01020408u) >> 24) << (o - o0);
    m &= ~0ull << (s - o0);
    if (e - o0 < 64) m &= (1ull << (e - o0)) - 1ull;
    f = min(__popcll(m), 6);
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      tab[i] = m ? o0 + __ffsll((long long)m) - 1 : e;
      m &= m - 1;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 6; ++i) tab[i] = e;
    for (int o = o0; o < e && f < 6; o += 4) {
      uint32_t m = __vcmpeq4(st[o >> 2], 0x09090909u) & 0x01010101u;
      if (o < s) m &= ~0u << (8 * (s - o));
      if (o + 4 > e) m &= (1u << (8 * (e - o))) - 1u;
      for (; m && f < 6; m &= m - 1) {
        const int at = o + ((__ffs(m) - 1) >> 3);
#pragma unroll
        for (int i = 0; i < 6; ++i)
          if (i == f) tab[i] = at;
        ++f;
      }
    }
  }
  r.f = f;
  r.clen = tab[0] - s;
  uint64_t c = staged8(st, s);
  if (r.clen < 8) c = r.clen ? c & (~0ull >> (64 - 8 * (int)r.clen)) : 0ull;
  r.ck = ((uint64_t)__byte_perm((uint32_t)c, 0, 0x0123) << 32) | __byte_perm((uint32_t)(c >> 32), 0, 0x0123);
  auto len = [&](int i) { return f > i ? tab[i + 1 > 5 ? 5 : i + 1] - tab[i] - 1 : 0; };
  r.len1 = len(0);
  r.len2 = len(1);
  r.blen = len(2);
  r.len4 = len(3);
  r.slen = len(4);
  r.start = staged_number(st, tab[0] + 1, (int)r.len1, r.ok1);
  r.end = staged_number(st, tab[1] + 1, (int)r.len2, r.ok2);
  r.cnt = staged_number(st, tab[3] + 1, (int)r.len4, r.ok4);
  r.bstart = f > 2 ? tab[2] + 1 - s : 0;
  auto byte = [&](int o) { return (uint8_t)(st[o >> 2] >> (8 * (o & 3))); };
  r.b0 = r.blen ? byte(tab[2] + 1) : 0;
  r.c4 = r.len4 ? byte(tab[3] + 1) : 0;
  r.sc = r.slen ? byte(tab[4] + (int)r.slen) : 0;
  uint64_t h = h0;  // as Hasher over the bytes, h0 = its start
  for (int i = 0; i < (int)r.blen; i += 8) {
    uint64_t w = staged8(st, tab[2] + 1 + i);
    if ((int)r.blen - i < 8) w &= ~0ull >> (64 - 8 * ((int)r.blen - i));
    h = mix64(h ^ w);
  }
  r.h = mix64(h ^ ((uint64_t)r.blen * 0x9e3779b97f4a7c15ull));
}

// Thread per line, 256 lines of a CTA at a time with their text staged in
// shared memory by 16-byte loads.  A loop over each line's bytes in global
// memory, with the lanes of a warp in different fields, took 1.65 ms for 1.8e7
// lines (0.83 GB); 0.97 now (some 1,000 instructions a line).  The kernel-wide first record, longest barcode
// and record count are reduced in registers and per warp before one atomic each.
constexpr int kStage = 20 * 1024;  // bytes of text staged per CTA

__global__ void __launch_bounds__(kThreads) parse_kernel(const uint8_t* __restrict__ text, int64_t nbytes,
                                                         const int64_t* __restrict__ line_start, int64_t n_lines,
                                                         ChromTable ct, int64_t shift_left, int64_t shift_right,
                                                         uint64_t seed, int bc_always, ParseOut o,
                                                         unsigned long long* first_rec,
                                                         unsigned long long* max_bc_len,
                                                         unsigned long long* n_rec, unsigned long long* bad,
                                                         int* status) {
  __shared__ __align__(16) uint32_t stage[kStage / 4 + 8];
  unsigned long long my_first = ~0ull, my_bc = 0;
  unsigned my_rec = 0;
  const uint64_t h0 = Hasher(seed).h;
  uint64_t last_ck = 0;  // the chromosome of this thread's line before (names of up to 8 bytes)
  int last_clen = -1, last_cid = -1;
  for (int64_t i0 = blockIdx.x * (int64_t)kThreads; i0 < n_lines; i0 += (int64_t)gridDim.x * kThreads) {
    const int64_t i = i0 + threadIdx.x, il = i0 + kThreads < n_lines ? i0 + kThreads : n_lines;
    const int64_t base = line_start[i0] & ~(int64_t)15;
    int64_t stop = line_start[il];
    if (stop > nbytes) stop = nbytes;
    const bool staged = stop - base <= kStage && ((uintptr_t)text & 15) == 0;  // uniform; 16-byte loads
    __syncthreads();
    if (staged) {
      for (int64_t p = base + 16 * threadIdx.x; p < stop; p += 16 * kThreads) {
        uint4 q;
        if (p + 16 <= nbytes) {
          q = __ldg(reinterpret_cast<const uint4*>(text + p));
        } else {
          uint32_t w[4] = {0, 0, 0, 0};
          for (int j = 0; j < 16 && p + j < nbytes; ++j) w[j >> 2] |= (uint32_t)text[p + j] << (8 * (j & 3));
          q = make_uint4(w[0], w[1], w[2], w[3]);
        }
        *reinterpret_cast<uint4*>(stage + (p - base) / 4) = q;
      }
    }
    __syncthreads();
    if (i >= n_lines) continue;  // the barriers above are reached by whole CTAs: i0 is uniform
    const int64_t s = line_start[i];
    int64_t e = line_start[i + 1] - 1;
    if (e > nbytes) e = nbytes;
    auto byte_at = [&](int64_t p) {
      return staged ? (uint8_t)(stage[(p - base) >> 2] >> (8 * ((p - base) & 3))) : text[p];
    };
    if (e < nbytes && e > s && byte_at(e - 1) == '\r') --e;  // CR of a CRLF line end
    if (e > s && byte_at(s) == '#') {
      o.flags[i] = 0;
      continue;
    }
    Fields r;
    if (staged) fields_staged(stage, (int)(s - base), (int)(e - base), h0, r);
    else fields_bytes(text, s, e, seed, r);
    const int f = r.f;
    uint64_t start = r.start, end = r.end;
    const uint64_t ck = r.ck, cntv = r.cnt;
    const int clen = r.clen, len1 = r.len1, len2 = r.len2, len4 = r.len4, blen = r.blen, slen = r.slen;
    const int64_t bstart = s + r.bstart;
    const bool ok1 = r.ok1, ok2 = r.ok2, ok4 = r.ok4;
    const uint8_t b0 = r.b0, c4 = r.c4, sc = r.sc;
    const int nf = f >= 6 ? 6 : f + 1;
    bool ok = nf >= 4 && ok1 && len1 > 0 && ok2 && len2 > 0;
    uint16_t fl = F_REC;
    uint64_t count = 1;
    if (ok && nf >= 5 && !(len4 == 1 && c4 == '.')) {   // "." = 1
      ok = ok4 && len4 > 0 && !(cntv >> 32);
      count = cntv;
    }
    if (ok && nf >= 6) {
      if (slen == 1 && sc == '+') fl |= F_STRANDED;
      else if (slen == 1 && sc == '-') fl |= F_STRANDED | F_REV;
      else if (!(slen == 1 && sc == '.')) ok = false;
    }
    const bool has_bc = ok && !(blen == 1 && b0 == '.');
    if (has_bc && blen > 0xFFFF) ok = false;
    // 2 line + (stranded): the smallest is the first record's (a malformed one ends the import)
    const unsigned long long me = 2ull * (unsigned long long)i + ((fl & F_STRANDED) ? 1ull : 0ull);
    my_first = my_first < me ? my_first : me;
    if (!ok) {
      o.flags[i] = 0;
      set_error(status, bad, SG_ERR_PARSE, i);
      continue;
    }
    // saturating shifts, preprocessing.rs:174-184
    const bool stranded = (fl & F_STRANDED) != 0;
    if (shift_left != 0) {
      start = sat_add(start, shift_left);
      if (stranded) end = sat_add(end, shift_left);
    }
    if (shift_right != 0 && !stranded) end = sat_add(end, shift_right);
    if (start != end) fl |= F_LEN;
    uint64_t h = 0, loc = 0;
    if (has_bc) {
      fl |= F_BC;
      h = r.h;
      loc = ((uint64_t)bstart << 16) | (uint64_t)blen;
      my_bc = my_bc > (unsigned long long)blen ? my_bc : (unsigned long long)blen;
      ++my_rec;
    } else if ((fl & F_LEN) || bc_always) {
      o.flags[i] = 0;
      set_error(status, bad, SG_ERR_PARSE, i);  // a fragment without a barcode
      continue;
    }
    int64_t gpos = -1, v = 0;
    if (ck != last_ck || clen != last_clen) {
      last_cid = find_chrom(ct, ck, clen, text + s);
      last_ck = ck;
      last_clen = clen <= 8 ? clen : -1;
    }
    const int cid = last_cid;
    if (cid >= 0) {
      fl |= F_GEN;
      if (ct.mito[cid]) fl |= F_MITO;
      // import.rs:176-204 with i64 arithmetic that wraps like the release build
      const uint64_t size = end - start;
      uint64_t pp;
      if (fl & F_REV) {
        pp = end - 1;
        v = (int64_t)(0 - size);
      } else {
        pp = start;
        v = (int64_t)size;
      }
      if (pp >= ct.size[cid]) fl |= F_POSERR;
      else gpos = (int64_t)(ct.base[cid] + pp);
      if (v >= 0 && v <= (int64_t)UINT32_MAX) fl |= F_FITU32;
      if (v >= (int64_t)INT32_MIN && v <= (int64_t)INT32_MAX) fl |= F_FITI32;
    }
    o.hash[i] = h;
    o.loc[i] = loc;
    o.pos[i] = gpos;
    o.val[i] = v;
    o.cnt[i] = (uint32_t)count;
    o.flags[i] = fl;
  }
#pragma unroll
  for (int off = 16; off; off >>= 1) {
    const unsigned long long a = __shfl_xor_sync(0xffffffffu, my_first, off);
    const unsigned long long b = __shfl_xor_sync(0xffffffffu, my_bc, off);
    my_first = a < my_first ? a : my_first;
    my_bc = b > my_bc ? b : my_bc;
  }
  my_rec = __reduce_add_sync(0xffffffffu, my_rec);
  if ((threadIdx.x & 31) == 0) {
    if (my_rec) atomicAdd(n_rec, (unsigned long long)my_rec);
    if (my_first != ~0ull) atomicMin(first_rec, my_first);
    if (my_bc) atomicMax(max_bc_len, my_bc);
  }
}

// ---- grouping ----------------------------------------------------------------
__device__ __forceinline__ bool is_record(uint16_t f) { return (f & (F_REC | F_BC)) == (F_REC | F_BC); }

// 1 for records with end != start (their ranks decide whether sorted input is)
__global__ void mark_len(int64_t n, const uint16_t* __restrict__ flags, int64_t* __restrict__ b) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    b[i] = is_record(flags[i]) && (flags[i] & F_LEN);
}

__global__ void rehash_records(int64_t n, const uint16_t* __restrict__ flags, const uint64_t* __restrict__ loc,
                               const uint8_t* __restrict__ text, uint64_t seed, uint64_t* __restrict__ hash) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    if (is_record(flags[i])) hash[i] = hash_bytes(text + loc_off(loc[i]), loc_len(loc[i]), seed);
}

// The barcode table: open addressing by hash, linear probing; key 0 = empty
// (a hash of 0 is stored as 1: a clash of the two is found by the byte
// comparison like any other).  first[s] = earliest line of slot s.  A slot is
// settled by one atomicCAS and read by plain loads from then on.
constexpr int kProbe = 64;  // probes before a table is given up for a larger one

__global__ void __launch_bounds__(kThreads) table_insert(int64_t n, const uint16_t* __restrict__ flags,
                                                         const uint64_t* __restrict__ hash, uint64_t mask,
                                                         int64_t most_probes, unsigned long long* __restrict__ table,
                                                         unsigned long long* __restrict__ first,
                                                         uint32_t* __restrict__ slot, int* __restrict__ full) {
  for (int64_t i = blockIdx.x * (int64_t)kThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kThreads) {
    if (!is_record(flags[i])) continue;
    const unsigned long long h = hash[i] ? hash[i] : 1ull;
    uint64_t t = h & mask;
    bool found = false;
    for (int64_t p = 0; p < most_probes; ++p, t = (t + 1) & mask) {
      unsigned long long k = *(volatile unsigned long long*)(table + t);
      if (k == 0) k = atomicCAS(table + t, 0ull, h);
      if (k == 0 || k == h) {
        found = true;
        break;
      }
    }
    if (!found) {
      *full = 1;
      continue;
    }
    slot[i] = (uint32_t)t;
    if (*(volatile unsigned long long*)(first + t) > (unsigned long long)i) atomicMin(first + t, (unsigned long long)i);
  }
}

__global__ void table_used(int64_t n, const unsigned long long* __restrict__ table, int64_t* __restrict__ used) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x)
    used[t] = table[t] != 0;
}

// Barcodes of the groups' first lines, 32 bytes each: up to 31 bytes (zero
// padded) and their number, or 255 for a longer one.
constexpr int kBcShort = 31;

// the group's first line, in `first` that line's barcode, and its bytes
__global__ void table_leaders(int64_t n, const unsigned long long* __restrict__ table,
                              unsigned long long* __restrict__ first, const int64_t* __restrict__ num,
                              const uint64_t* __restrict__ loc, const uint8_t* __restrict__ text,
                              int64_t* __restrict__ leader, uint8_t* __restrict__ bc) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x)
    if (table[t]) {
      const unsigned long long line = first[t];
      const int64_t g = num[t] - 1;
      const uint64_t l = loc[line];
      leader[g] = (int64_t)line;
      first[t] = l;
      uint8_t* d = bc + 32 * g;
      const int len = loc_len(l);
      for (int j = 0; j < kBcShort; ++j) d[j] = j < len && len <= kBcShort ? text[loc_off(l) + j] : 0;
      d[kBcShort] = len <= kBcShort ? (uint8_t)len : 255;
    }
}

// Whether the barcode of n <= 31 bytes at p is the one kept in q[0..1]: two
// 16-byte reads of it and the aligned words of the text, all in flight
// together (a word that holds a byte of the text lies inside its allocation).
__device__ __forceinline__ bool same_barcode(const uint8_t* p, int n, const uint4& q0, const uint4& q1) {
  const uint32_t* w = reinterpret_cast<const uint32_t*>((uintptr_t)p & ~(uintptr_t)3);
  const int o = (int)((uintptr_t)p & 3);
  uint32_t x[9];
#pragma unroll
  for (int j = 0; j < 9; ++j) x[j] = 4 * j < o + n ? __ldg(w + j) : 0u;
  const uint32_t k[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w & 0x00ffffffu};
  uint32_t d = (q1.w >> 24) ^ (uint32_t)n;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    uint32_t v = __funnelshift_r(x[j], x[j + 1], 8 * o);
    const int left = n - 4 * j;
    v = left >= 4 ? v : (left > 0 ? v & ((1u << (8 * left)) - 1u) : 0u);
    d |= v ^ k[j];
  }
  return d == 0;
}

// equality of n bytes at any alignment: aligned 4-byte words (a word that
// holds a byte of the text lies inside its allocation), shifted into place
__device__ __forceinline__ bool bytes_equal_wide(const uint8_t* a, const uint8_t* b, int n) {
  const uint32_t* pa = reinterpret_cast<const uint32_t*>((uintptr_t)a & ~(uintptr_t)3);
  const uint32_t* pb = reinterpret_cast<const uint32_t*>((uintptr_t)b & ~(uintptr_t)3);
  const int oa = (int)((uintptr_t)a & 3), ob = (int)((uintptr_t)b & 3);
  if (n <= 0) return true;
  uint32_t xa = __ldg(pa), xb = __ldg(pb);
  for (int k = 0; k < n; k += 4) {
    const int left = n - k;
    uint32_t ya = 0, yb = 0;  // the next words, where bytes of them are wanted
    if (oa + left > 4) ya = __ldg(++pa);
    if (ob + left > 4) yb = __ldg(++pb);
    uint32_t d = __funnelshift_r(xa, ya, 8 * oa) ^ __funnelshift_r(xb, yb, 8 * ob);
    if (left < 4) d &= (1u << (8 * left)) - 1u;
    if (d) return false;
    xa = ya;
    xb = yb;
  }
  return true;
}

struct Groups {
  // pairs of 32-bit counts (a text of 2^32 lines is beyond the memory of the GPU)
  unsigned long long* recs;   // records with this barcode | with end != start << 32
  unsigned long long* gen;    // ... of these in the genome, not mitochondrial | mitochondrial << 32
  unsigned long long* total;  // sum of the count column over in-genome records
  long long* rmin;            // first / last rank among records with end != start
  long long* rmax;
  long long* err;             // lowest line with a position or size error
  int64_t* leader;            // line of the group's first record
  int64_t* cell;              // cell row, or -1
  uint8_t* wl;                // whitelisted
  int64_t* keep;              // kept flag, then its scan
  __device__ unsigned long long n_all(int64_t i) const { return recs[i] & 0xffffffffull; }
  __device__ unsigned long long n_len(int64_t i) const { return recs[i] >> 32; }
  __device__ unsigned long long uniq(int64_t i) const { return gen[i] & 0xffffffffull; }
  __device__ unsigned long long mito(int64_t i) const { return gen[i] >> 32; }
};

__global__ void init_groups(int64_t G, Groups g) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < G; i += (int64_t)gridDim.x * blockDim.x) {
    g.recs[i] = g.gen[i] = g.total[i] = 0;
    g.rmin[i] = LLONG_MAX;
    g.rmax[i] = -1;
    g.err[i] = LLONG_MAX;
    g.cell[i] = -1;
    g.wl[i] = 0;
  }
}

// Per-group counts over the records in line order, and the byte comparison
// with the group's first record.  Up to kSmallGroups groups are counted per CTA
// in shared memory (a record is of one of four classes, so it takes one
// counter and the sum of the count column) and added up at the end.  What
// bounds it are the scattered reads of the byte comparison, one L1 lookup a
// lane: over the text of the first line, word by word, they took 1.19 ms for
// 1.8e7 records in genome order, over the 32-byte copies 0.62.  A warp whose records share a barcode (input
// sorted by barcode) adds them up first; the ranks are wanted for it only.
constexpr int kSmallGroups = 2048;

template <bool SMALL>
__global__ void __launch_bounds__(kThreads) group_stats(int64_t n, const uint16_t* __restrict__ flags,
                                                        const int64_t* __restrict__ num,
                                                        const unsigned long long* __restrict__ first,
                                                        uint32_t* __restrict__ slot, const uint64_t* __restrict__ loc,
                                                        const uint8_t* __restrict__ text,
                                                        const uint4* __restrict__ bc,
                                                        const uint32_t* __restrict__ cnt,
                                                        const int64_t* __restrict__ lrank,
                                                        const int64_t* __restrict__ val, int paired, int64_t G,
                                                        Groups g, unsigned long long* __restrict__ max_abs,
                                                        int* __restrict__ collide) {
  // classes: 0 in the genome, 1 mitochondrial, 2 outside the genome, 3 of no length; 4: sum of small counts
  __shared__ uint32_t few[SMALL ? 5 : 1][SMALL ? kSmallGroups : 1];
  const int lane = threadIdx.x & 31;
  const int64_t stride = (int64_t)gridDim.x * kThreads;
  if (SMALL) {
    for (int t = threadIdx.x; t < 5 * kSmallGroups; t += kThreads) few[t / kSmallGroups][t % kSmallGroups] = 0;
    __syncthreads();
  }
  // a CTA's sums of counts below kFewCount stay below 2^32 for up to 2^22 lines a CTA
  const unsigned long long few_count = SMALL && n / gridDim.x < (1 << 22) ? 1024 : 0;
  auto add = [&](int64_t gid, unsigned long long recs, unsigned long long gen, unsigned long long tot) {
    atomicAdd(g.recs + gid, recs);
    if (gen) atomicAdd(g.gen + gid, gen);
    if (tot) atomicAdd(g.total + gid, tot);
  };
  unsigned long long my_amax = 0;
  bool clash = false;
  for (int64_t i0 = blockIdx.x * (int64_t)kThreads; i0 < n; i0 += stride) {
    const int64_t i = i0 + threadIdx.x;
    const uint16_t f = i < n ? flags[i] : 0;
    const bool rec = is_record(f);
    int gid = -1, cls = 3;
    unsigned long long tot = 0;
    long long rmn = LLONG_MAX, rmx = -1, er = LLONG_MAX;
    if (rec) {
      const uint32_t t = slot[i];
      gid = (int)(num[t] - 1);
      slot[i] = (uint32_t)gid;  // the record's group from here on
      const uint64_t a = loc[i];
      if (loc_len(a) <= kBcShort) {
        clash |= !same_barcode(text + loc_off(a), loc_len(a), __ldg(bc + 2 * gid), __ldg(bc + 2 * gid + 1));
      } else {
        const uint64_t b = first[t];
        if (a != b)
          clash |= loc_len(a) != loc_len(b) || !bytes_equal_wide(text + loc_off(a), text + loc_off(b), loc_len(a));
      }
      if ((f & F_LEN) && (f & F_GEN)) {
        cls = (f & F_MITO) ? 1 : 0;
        tot = cnt[i];
        const bool fits = paired ? (f & F_FITU32) : (f & F_FITI32);
        if ((f & F_POSERR) || !fits) er = i;
        if (fits) {
          const int64_t v = val[i];
          const unsigned long long av = (unsigned long long)(v < 0 ? -v : v);
          my_amax = av > my_amax ? av : my_amax;
        }
      } else if (f & F_LEN) {
        cls = 2;
      }
      if (lrank && (f & F_LEN)) rmn = rmx = lrank[i];
    }
    const int top = __reduce_max_sync(0xffffffffu, gid);
    if (top < 0) continue;
    unsigned long long recs = rec ? 1ull | (cls < 3 ? 1ull << 32 : 0ull) : 0ull;
    unsigned long long gen = rec && cls < 2 ? (cls ? 1ull << 32 : 1ull) : 0ull;
    if (__all_sync(0xffffffffu, gid < 0 || gid == top)) {
#pragma unroll
      for (int o = 16; o; o >>= 1) {
        recs += __shfl_xor_sync(0xffffffffu, recs, o);
        gen += __shfl_xor_sync(0xffffffffu, gen, o);
        tot += __shfl_xor_sync(0xffffffffu, tot, o);
        const long long a = __shfl_xor_sync(0xffffffffu, rmn, o), b = __shfl_xor_sync(0xffffffffu, rmx, o),
                        c = __shfl_xor_sync(0xffffffffu, er, o);
        rmn = a < rmn ? a : rmn;
        rmx = b > rmx ? b : rmx;
        er = c < er ? c : er;
      }
      if (lane) gid = -1;
      else add(gid = top, recs, gen, tot);
    } else if (gid >= 0) {
      if (SMALL) {
        atomicAdd(&few[cls][gid], 1u);
        if (SMALL && tot < few_count) {
          if (tot) atomicAdd(&few[4][gid], (uint32_t)tot);
        } else {
          atomicAdd(g.total + gid, tot);
        }
      } else {
        add(gid, recs, gen, tot);
      }
    }
    if (gid >= 0) {
      if (rmx >= 0) {
        atomicMin(g.rmin + gid, rmn);
        atomicMax(g.rmax + gid, rmx);
      }
      if (er != LLONG_MAX) atomicMin(g.err + gid, er);
    }
  }
  if (SMALL) {
    __syncthreads();
    for (int t = threadIdx.x; t < (int)G; t += kThreads) {
      const unsigned long long c0 = few[0][t], c1 = few[1][t], c2 = few[2][t], c3 = few[3][t];
      if (c0 + c1 + c2 + c3) add(t, (c0 + c1 + c2 + c3) | (c0 + c1 + c2) << 32, c0 | c1 << 32, few[4][t]);
    }
  }
  if (clash) *collide = 1;
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const unsigned long long x = __shfl_xor_sync(0xffffffffu, my_amax, o);
    my_amax = x > my_amax ? x : my_amax;
  }
  if (lane == 0 && my_amax) atomicMax(max_abs, my_amax);
}

// ---- whitelist ---------------------------------------------------------------
__global__ void wl_hash(int64_t W, const uint8_t* __restrict__ blob, const int64_t* __restrict__ off, uint64_t seed,
                        uint64_t* __restrict__ keys, uint64_t* __restrict__ vals) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < W; k += (int64_t)gridDim.x * blockDim.x) {
    keys[k] = hash_bytes(blob + off[k], off[k + 1] - off[k], seed);
    vals[k] = (uint64_t)k;
  }
}

__global__ void wl_lookup(int64_t G, const int64_t* __restrict__ leader, const uint64_t* __restrict__ loc,
                          const uint8_t* __restrict__ text, uint64_t seed, int64_t W,
                          const uint64_t* __restrict__ wkeys, const uint64_t* __restrict__ wvals,
                          const uint8_t* __restrict__ blob, const int64_t* __restrict__ off, uint8_t* __restrict__ wl) {
  for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < G; g += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t l = loc[leader[g]];
    const uint8_t* b = text + loc_off(l);
    const int n = loc_len(l);
    const uint64_t h = hash_bytes(b, n, seed);
    int64_t lo = 0, hi = W;
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if (wkeys[mid] < h) lo = mid + 1;
      else hi = mid;
    }
    uint8_t hit = 0;
    for (int64_t k = lo; k < W && wkeys[k] == h && !hit; ++k) {
      const int64_t e = (int64_t)wvals[k];
      if (off[e + 1] - off[e] == n && bytes_equal(blob + off[e], b, n)) hit = 1;
    }
    wl[g] = hit;
  }
}

// ---- decisions ---------------------------------------------------------------
__global__ void decide_groups(int64_t G, Groups g, const uint16_t* __restrict__ flags, int has_wl, int pre_min,
                              int sorted_input, uint64_t min_frag, unsigned long long* bad, int* status) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < G; i += (int64_t)gridDim.x * blockDim.x) {
    bool pass = (!has_wl || g.wl[i]) && g.n_len(i) > 0;
    if (pre_min) pass = pass && g.n_all(i) >= min_frag;
    if (pass) {
      if (sorted_input && (unsigned long long)(g.rmax[i] - g.rmin[i] + 1) != g.n_len(i))
        set_error(status, bad, SG_ERR_UNSORTED, g.leader[i]);
      if (g.err[i] != LLONG_MAX) {
        const int64_t line = g.err[i];
        set_error(status, bad, (flags[line] & F_POSERR) ? SG_ERR_RANGE : SG_ERR_CONVERT, line);
      }
    }
    g.keep[i] = pass && g.uniq(i) >= min_frag;
  }
}

__global__ void kept_keys(int64_t G, const Groups g, const int64_t* __restrict__ keep_scan, int sorted_input,
                          const uint64_t* __restrict__ loc, uint64_t* __restrict__ keys, uint64_t* __restrict__ vals) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < G; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t prev = i ? keep_scan[i - 1] : 0;
    if (keep_scan[i] != prev) {
      keys[prev] = sorted_input ? (uint64_t)g.rmin[i] : (uint64_t)loc_len(loc[g.leader[i]]);
      vals[prev] = (uint64_t)i;
    }
  }
}

// Order of up to kRankGroups groups by counting: each group's place is the
// number of groups before it.  One launch, where the radix passes over the
// lengths and the barcode's words take five launches for each of 25 digits.
constexpr int64_t kRankGroups = 8192;

__global__ void __launch_bounds__(256) rank_numbers(int64_t K, const uint64_t* __restrict__ keys,
                                                    const uint64_t* __restrict__ vals, uint64_t* __restrict__ order) {
  __shared__ uint64_t k[256];
  const int64_t i = blockIdx.x * (int64_t)256 + threadIdx.x;
  const uint64_t mine = i < K ? keys[i] : 0;
  int64_t before = 0;
  for (int64_t j0 = 0; j0 < K; j0 += 256) {
    __syncthreads();
    k[threadIdx.x] = j0 + threadIdx.x < K ? keys[j0 + threadIdx.x] : ~0ull;
    __syncthreads();
    const int m = (int)(K - j0 < 256 ? K - j0 : 256);
    for (int j = 0; j < m; ++j) before += k[j] < mine || (k[j] == mine && j0 + j < i);
  }
  if (i < K) order[before] = vals[i];
}

// By barcode bytes, a prefix before what it begins (the barcodes differ):
// words[w K + i] = big-endian 8-byte word w of barcode i, zero padded; differ[w]
// says that not all barcodes have the same word w.  Names with a sample in
// front agree in their first words in every pair, so the comparison starts at
// the first word that differs, and goes on word by word where two names agree
// in it (looked for after the count, so that the count has no branch).  1,500
// random barcodes take 30 us (91 with the branch and the bytes of the text); a
// call on 8,000 cells of 200 fragments 1.16 ms (1.49), with 11 bytes in front of
// the barcodes 1.65 ms (7.1), with 40 bytes 1.58 ms (29).
constexpr int kRankWords = 8;  // longer barcodes are ordered by the radix passes

__global__ void __launch_bounds__(256) rank_barcodes(int64_t K, int nwords, const uint64_t* __restrict__ words,
                                                     const int* __restrict__ differ,
                                                     const uint64_t* __restrict__ vals,
                                                     const int64_t* __restrict__ leader,
                                                     const uint64_t* __restrict__ loc, uint64_t* __restrict__ order) {
  __shared__ uint64_t k[256];
  __shared__ int len[256];
  int w0 = 0;
  while (w0 + 1 < nwords && !differ[w0]) ++w0;
  const uint64_t* first = words + w0 * K;
  const int64_t i = blockIdx.x * (int64_t)256 + threadIdx.x;
  const uint64_t mine = i < K ? first[i] : 0;
  const int n = i < K ? loc_len(loc[leader[vals[i]]]) : 0;
  int64_t before = 0;
  for (int64_t j0 = 0; j0 < K; j0 += 256) {
    const int64_t t = j0 + threadIdx.x;
    __syncthreads();
    if (t < K) {
      k[threadIdx.x] = first[t];
      len[threadIdx.x] = loc_len(loc[leader[vals[t]]]);
    }
    __syncthreads();
    const int m = (int)(K - j0 < 256 ? K - j0 : 256);
    const int self = i < K && j0 / 256 == blockIdx.x ? (int)threadIdx.x : -1;
    int less = 0, same = 0, at = 0;  // at: the last other one that agrees
#pragma unroll 8
    for (int j = 0; j < m; ++j) {
      const bool eq = k[j] == mine && j != self;
      less += k[j] < mine;
      same += eq;
      at = eq ? j : at;
    }
    before += less;
    if (i >= K || same == 0) continue;
    for (int j = same == 1 ? at : 0; j <= at; ++j) {
      if (k[j] != mine || j == self) continue;
      uint64_t a = 0, b = 0;
      for (int w = w0 + 1; w < nwords && a == b; ++w) {
        a = words[w * K + j0 + j];
        b = words[w * K + i];
      }
      before += a != b ? a < b : len[j] < n;
    }
  }
  if (i < K) order[before] = vals[i];
}

// big-endian 8-byte word w of a barcode, zero padded
__device__ __forceinline__ uint64_t barcode_word(uint64_t l, const uint8_t* __restrict__ text, int w) {
  const uint8_t* b = text + loc_off(l);
  const int n = loc_len(l);
  uint64_t k = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int p = 8 * w + j;
    k = (k << 8) | (p < n ? b[p] : 0u);
  }
  return k;
}

// keys[r] = word w of each kept group's barcode
__global__ void word_keys(int64_t K, const uint64_t* __restrict__ vals, const int64_t* __restrict__ leader,
                          const uint64_t* __restrict__ loc, const uint8_t* __restrict__ text, int w,
                          uint64_t* __restrict__ keys) {
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < K; r += (int64_t)gridDim.x * blockDim.x)
    keys[r] = barcode_word(loc[leader[vals[r]]], text, w);
}

// rank_barcodes' words and differ, word w = blockIdx.y
__global__ void word_table(int64_t K, const uint64_t* __restrict__ vals, const int64_t* __restrict__ leader,
                           const uint64_t* __restrict__ loc, const uint8_t* __restrict__ text,
                           uint64_t* __restrict__ words, int* __restrict__ differ) {
  const int w = blockIdx.y;
  const uint64_t k0 = barcode_word(loc[leader[vals[0]]], text, w);
  bool other = false;
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < K; r += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t k = barcode_word(loc[leader[vals[r]]], text, w);
    words[w * K + r] = k;
    other |= k != k0;
  }
  if (other) differ[w] = 1;
}

// per cell row r (kept groups in final order): QC columns, barcode, row length
__global__ void cell_rows(int64_t K, const uint64_t* __restrict__ order, Groups g, const uint64_t* __restrict__ loc,
                          int64_t* __restrict__ row_len, uint64_t* __restrict__ bc_loc, uint64_t* __restrict__ nfrag,
                          double* __restrict__ fdup, double* __restrict__ fmito) {
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < K; r += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = (int64_t)order[r];
    g.cell[i] = r;
    const unsigned long long u = g.uniq(i), m = g.mito(i), t = g.total[i];
    row_len[r] = (int64_t)(u + m);
    bc_loc[r] = loc[g.leader[i]];
    nfrag[r] = u;
    // qc.rs:454-465, FP64 and IEEE division (0/0 gives NaN as in the reference)
    fdup[r] = 1.0 - (double)(u + m) / (double)t;
    fmito[r] = (double)m / (double)(u + m);
  }
}

struct KeyLayout {
  int vbits, pbits, rbits;
  int64_t vbias;
  bool combined;  // one 64-bit key (cell | position | size)
};

// Records of the matrix, compacted in line order, kMatTile lines per CTA:
// counted per tile, then (after a scan of the tile counts) written.
constexpr int kMatItems = 8;
constexpr int kMatTile = kThreads * kMatItems;

__device__ __forceinline__ int64_t matrix_cell(int64_t i, int64_t n, const uint16_t* __restrict__ flags,
                                               const uint32_t* __restrict__ group, const int64_t* __restrict__ cell) {
  if (i >= n) return -1;
  const uint16_t f = flags[i];
  return is_record(f) && (f & F_LEN) && (f & F_GEN) ? cell[group[i]] : -1;
}

__global__ void __launch_bounds__(kThreads) matrix_count(int64_t n, const uint16_t* __restrict__ flags,
                                                         const uint32_t* __restrict__ group,
                                                         const int64_t* __restrict__ cell,
                                                         int64_t* __restrict__ counts) {
  const int64_t i0 = blockIdx.x * (int64_t)kMatTile + threadIdx.x;
  int c = 0;
#pragma unroll
  for (int k = 0; k < kMatItems; ++k) c += matrix_cell(i0 + k * kThreads, n, flags, group, cell) >= 0;
  __shared__ int ws[kThreads / 32];
  c = __reduce_add_sync(0xffffffffu, c);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kThreads / 32; ++w) c += ws[w];
    counts[blockIdx.x] = c;
  }
}

// combined: key = cell << (pbits + vbits) | pos << vbits | (val + bias) in
// `slot`, and in `keys` cell << cbits | chromosome; otherwise: keys = val +
// bias, slot = index, k2 = pos, k3 = cell (sorted in that order)
__global__ void __launch_bounds__(kThreads) matrix_keys(int64_t n, const uint16_t* __restrict__ flags,
                                                        const uint32_t* __restrict__ group,
                                                        const int64_t* __restrict__ cell,
                                                        const int64_t* __restrict__ counts,
                                                        const int64_t* __restrict__ pos,
                                                        const int64_t* __restrict__ val,
                                                        const uint64_t* __restrict__ chrom_base, int n_chrom,
                                                        int cbits, KeyLayout kl, uint64_t* __restrict__ keys,
                                                        uint64_t* __restrict__ slot, int64_t* __restrict__ k2,
                                                        int64_t* __restrict__ k3) {
  __shared__ int ws[kMatItems][kThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t i0 = blockIdx.x * (int64_t)kMatTile + threadIdx.x;
  int64_t c[kMatItems];
  int rank[kMatItems];
#pragma unroll
  for (int k = 0; k < kMatItems; ++k) {
    c[k] = matrix_cell(i0 + k * kThreads, n, flags, group, cell);
    const unsigned m = __ballot_sync(0xffffffffu, c[k] >= 0);
    rank[k] = __popc(m & lanemask_lt());
    if (lane == 0) ws[k][w] = __popc(m);
  }
  __syncthreads();
  int64_t at = blockIdx.x ? counts[blockIdx.x - 1] : 0;
#pragma unroll
  for (int k = 0; k < kMatItems; ++k) {
    int before = 0, all = 0;
#pragma unroll
    for (int v = 0; v < kThreads / 32; ++v) {
      before += v < w ? ws[k][v] : 0;
      all += ws[k][v];
    }
    if (c[k] >= 0) {
      const int64_t i = i0 + k * kThreads, j = at + before + rank[k];
      const uint64_t vb = (uint64_t)(val[i] + kl.vbias);
      const uint64_t p = (uint64_t)pos[i];
      if (kl.combined) {
        slot[j] = ((uint64_t)c[k] << (kl.pbits + kl.vbits)) | (p << kl.vbits) | vb;
        int a = 0, b = n_chrom - 1;  // last chromosome that starts at or before p
        while (a < b) {
          const int m = (a + b + 1) >> 1;
          if (__ldg(chrom_base + m) <= p) a = m;
          else b = m - 1;
        }
        keys[j] = ((uint64_t)c[k] << cbits) | (uint64_t)a;
      } else {
        keys[j] = vb;
        slot[j] = (uint64_t)j;
        k2[j] = (int64_t)p;
        k3[j] = c[k];
      }
    }
    at += all;
  }
}

// state[0]: a (cell, position) below the one before it; state[1]: equal ones
// whose sizes are out of order
__global__ void order_check(int64_t n, const uint64_t* __restrict__ keys, int vbits, int* __restrict__ state) {
  bool bad = false, mend = false;
  for (int64_t j = 1 + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < n; j += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t a = keys[j - 1], b = keys[j];
    if (b < a) {
      if ((a >> vbits) == (b >> vbits)) mend = true;
      else bad = true;
    }
  }
  if (bad) state[0] = 1;
  if (mend) state[1] = 1;
}

// Sorts the sizes of every run of one (cell, position) that is out of order;
// a run of more than kMendRun goes to the full sort (state[0]).
constexpr int kMendRun = 64;

__global__ void order_mend(int64_t n, uint64_t* __restrict__ keys, int vbits, int* __restrict__ state) {
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j + 1 < n; j += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t run = keys[j] >> vbits;  // the run's (cell, position) stays while its sizes move
    if ((j > 0 && (keys[j - 1] >> vbits) == run) || (keys[j + 1] >> vbits) != run) continue;
    int len = 2;
    while (len <= kMendRun && j + len < n && (keys[j + len] >> vbits) == run) ++len;
    if (len > kMendRun) {
      for (int64_t q = j + 1; q < n && (keys[q] >> vbits) == run; ++q)
        if (keys[q] < keys[q - 1]) {
          state[0] = 1;
          break;
        }
      continue;
    }
    for (int a = 1; a < len; ++a) {
      const uint64_t x = keys[j + a];
      int b = a;
      for (; b > 0 && keys[j + b - 1] > x; --b) keys[j + b] = keys[j + b - 1];
      keys[j + b] = x;
    }
  }
}

__global__ void gather_keys(int64_t n, const uint64_t* __restrict__ slot, const int64_t* __restrict__ src,
                            uint64_t* __restrict__ keys) {
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < n; j += (int64_t)gridDim.x * blockDim.x)
    keys[j] = (uint64_t)src[slot[j]];
}

__global__ void decode_combined(int64_t n, const uint64_t* __restrict__ keys, KeyLayout kl, int64_t* __restrict__ pos,
                                int32_t* __restrict__ val) {
  const uint64_t vmask = kl.vbits >= 64 ? ~0ull : ((1ull << kl.vbits) - 1);
  const uint64_t pmask = kl.pbits >= 64 ? ~0ull : ((1ull << kl.pbits) - 1);
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < n; j += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t k = keys[j];
    pos[j] = (int64_t)((k >> kl.vbits) & pmask);
    val[j] = (int32_t)(int64_t)((k & vmask) - (uint64_t)kl.vbias);
  }
}

__global__ void decode_slots(int64_t n, const uint64_t* __restrict__ slot, const int64_t* __restrict__ k2,
                             const uint64_t* __restrict__ vb_sorted_by_slot, int64_t vbias, int64_t* __restrict__ pos,
                             int32_t* __restrict__ val) {
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < n; j += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t s = slot[j];
    pos[j] = k2[s];
    val[j] = (int32_t)((int64_t)vb_sorted_by_slot[s] - vbias);
  }
}

__global__ void scatter_by_slot(int64_t n, const uint64_t* __restrict__ keys, const uint64_t* __restrict__ slot,
                                uint64_t* __restrict__ out) {
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < n; j += (int64_t)gridDim.x * blockDim.x)
    out[slot[j]] = keys[j];
}

// ---- workspace ---------------------------------------------------------------
inline int64_t al(int64_t b) { return (b + 255) / 256 * 256; }

struct Layout {
  int64_t hash, loc, pos, val, cnt, flags, slot, b;
  int64_t table, first, num;         // barcode table of up to table_slots(L) entries
  int64_t x0, y0, x1, y1;            // group order, then matrix sort
  int64_t wk0, wv0, wk1, wv1;        // whitelist sort
  int64_t g_recs, g_gen, g_total, g_rmin, g_rmax, g_err, g_leader, g_cell, g_wl, g_keep;
  int64_t order, row_ptr, bc, nfrag, fdup, fmito, mcount, k2, k3, mpos, mval, words;
  int64_t radix, scan, scal, pk;
  int64_t total;
};

// the largest power of two up to 2 L (more than L): room for every line's own barcode
inline int64_t table_slots(int64_t L) {
  int64_t t = 2;
  while (2 * t <= 2 * L) t *= 2;
  return t;
}

Layout frag_layout(int64_t L, int64_t W) {
  Layout y{};
  int64_t o = 0;
  auto take = [&](int64_t bytes) { const int64_t r = o; o += al(bytes < 256 ? 256 : bytes); return r; };
  const int64_t L8 = 8 * (L < 1 ? 1 : L), W8 = 8 * (W < 1 ? 1 : W), S8 = 8 * table_slots(L);
  y.hash = take(L8); y.loc = take(L8); y.pos = take(L8); y.val = take(L8);
  y.cnt = take(4 * L); y.flags = take(2 * L); y.slot = take(4 * L); y.b = take(L8);
  y.table = take(S8); y.first = take(S8); y.num = take(S8);
  y.x0 = take(L8); y.y0 = take(L8); y.x1 = take(L8); y.y1 = take(L8);
  y.wk0 = take(W8); y.wv0 = take(W8); y.wk1 = take(W8); y.wv1 = take(W8);
  y.g_recs = take(L8); y.g_gen = take(L8); y.g_total = take(L8);
  y.g_rmin = take(L8); y.g_rmax = take(L8); y.g_err = take(L8); y.g_leader = take(L8); y.g_cell = take(L8);
  y.g_wl = take(L); y.g_keep = take(L8);
  y.order = take(L8); y.row_ptr = take(L8 + 8); y.bc = take(L8); y.nfrag = take(L8); y.fdup = take(L8);
  y.fmito = take(L8); y.mcount = take(L8); y.k2 = take(L8); y.k3 = take(L8); y.mpos = take(L8); y.mval = take(4 * L);
  y.words = take(8 * kRankWords * std::min(L, kRankGroups));
  const int64_t big = L > W ? L : W;
  y.radix = take(radix_scratch_bytes(big < 1 ? 1 : big));
  y.scan = take(scan_scratch_bytes(table_slots(L) + 1));
  y.scal = take(256);
  y.pk = take(8 * kMaxChroms);
  y.total = o;
  return y;
}

inline int bits_for(uint64_t maxv) {  // bits to hold values 0..maxv
  int b = 0;
  while (b < 64 && (maxv >> b)) ++b;
  return b < 1 ? 1 : b;
}

int grid_of(int64_t n) { return grid_for(n, kThreads, 8 * 152 * 8); }

// device-resident scalars in the workspace
struct Scalars {
  unsigned long long first_rec;  // 2 x line of the first record + whether it is stranded
  unsigned long long max_bc, bad, max_abs, n_rec;
  int status, collide, full;
  int order[2];  // order_check
  int differ[kRankWords];  // word_table
};

}  // namespace
}  // namespace sg

using namespace sg;

extern "C" int64_t sg_frag_line_scratch_bytes(int64_t nbytes) {
  if (nbytes < 0) return -1;
  const int64_t nc = (nbytes + kChunk - 1) / kChunk;
  return al((nc + 1) * 8) + scan_scratch_bytes(nc + 1);
}

extern "C" int sg_frag_count_lines(const uint8_t* text, int64_t nbytes, void* scratch, int64_t* n_lines,
                                   void* stream) {
  if (nbytes < 0 || !n_lines || (nbytes > 0 && (!text || !scratch))) return SG_ERR_ARG;
  if (((uintptr_t)text & 15) != 0) return SG_ERR_ARG;
  *n_lines = 0;
  if (nbytes == 0) return SG_OK;
  cudaStream_t s = as_stream(stream);
  const int64_t nc = (nbytes + kChunk - 1) / kChunk;
  int64_t* counts = static_cast<int64_t*>(scratch);
  line_count_kernel<<<(unsigned)nc, kThreads, 0, s>>>(text, nbytes, counts);
  SG_CHECK_LAUNCH();
  if (inclusive_scan_i64(counts, nc + 1, static_cast<char*>(scratch) + al((nc + 1) * 8), s) != cudaSuccess)
    return SG_ERR_CUDA;
  int64_t nl = 0;
  uint8_t last = 0;
  if (cudaMemcpyAsync(&nl, counts + nc, 8, cudaMemcpyDeviceToHost, s) != cudaSuccess) return SG_ERR_CUDA;
  if (cudaMemcpyAsync(&last, text + nbytes - 1, 1, cudaMemcpyDeviceToHost, s) != cudaSuccess) return SG_ERR_CUDA;
  if (cudaStreamSynchronize(s) != cudaSuccess) return SG_ERR_CUDA;
  *n_lines = nl + (last != '\n' ? 1 : 0);
  return SG_OK;
}

extern "C" int sg_frag_index_lines(const uint8_t* text, int64_t nbytes, const void* scratch, int64_t n_lines,
                                   int64_t* line_start, void* stream) {
  if (nbytes < 0 || n_lines < 0 || !line_start || (nbytes > 0 && (!text || !scratch))) return SG_ERR_ARG;
  cudaStream_t s = as_stream(stream);
  if (nbytes == 0) {
    return cudaMemsetAsync(line_start, 0, 8, s) == cudaSuccess ? SG_OK : SG_ERR_CUDA;
  }
  const int64_t nc = (nbytes + kChunk - 1) / kChunk;
  line_fill_kernel<<<(unsigned)nc, kThreads, 0, s>>>(text, nbytes, static_cast<const int64_t*>(scratch), n_lines,
                                                     line_start);
  SG_CHECK_LAUNCH();
  return SG_OK;
}

extern "C" int64_t sg_frag_workspace_bytes(int64_t n_lines, int64_t n_whitelist) {
  if (n_lines < 0 || n_whitelist < 0) return -1;
  return frag_layout(n_lines, n_whitelist).total;
}

#define SG_CUDA(x)                                  \
  do {                                              \
    if ((x) != cudaSuccess) return SG_ERR_CUDA;     \
  } while (0)

extern "C" int sg_frag_import(const uint8_t* text, int64_t nbytes, const int64_t* line_start, int64_t n_lines,
                              const uint8_t* chrom_blob, const int64_t* chrom_off, const uint64_t* chrom_size,
                              const uint64_t* chrom_base, const uint8_t* chrom_mito, int n_chrom,
                              uint64_t genome_size, const uint8_t* wl_blob, const int64_t* wl_off, int64_t n_whitelist,
                              int has_whitelist, uint64_t min_num_fragments, int sorted_by_barcode,
                              int64_t shift_left, int64_t shift_right, uint64_t seed, void* workspace,
                              int64_t workspace_bytes, int64_t* info, void* stream) {
  if (!info || n_lines < 0 || n_chrom <= 0 || n_chrom > kMaxChroms || n_whitelist < 0 || nbytes < 0)
    return SG_ERR_ARG;
  if (n_lines > 0 && (!text || !line_start || !workspace)) return SG_ERR_ARG;
  if (!chrom_blob || !chrom_off || !chrom_size || !chrom_base || !chrom_mito) return SG_ERR_ARG;
  if (has_whitelist && n_whitelist > 0 && (!wl_blob || !wl_off)) return SG_ERR_ARG;
  if (shift_left < -(int64_t(1) << 62) || shift_left > (int64_t(1) << 62) || shift_right < -(int64_t(1) << 62) ||
      shift_right > (int64_t(1) << 62) || nbytes >= (int64_t(1) << 47))
    return SG_ERR_ARG;
  for (int i = 0; i < 10; ++i) info[i] = 0;
  info[2] = -1;
  info[3] = -1;
  if (n_lines == 0) return SG_OK;
  const Layout y = frag_layout(n_lines, n_whitelist);
  if (workspace_bytes < y.total) return SG_ERR_CAP;
  cudaStream_t s = as_stream(stream);
  char* ws = static_cast<char*>(workspace);
  int64_t nk = 0;  // kernels launched (info[8])
  auto scan_counted = [&](int64_t* d, int64_t n, void* scr, cudaStream_t st) {
    if (n > 0) nk += 3;
    return inclusive_scan_i64(d, n, scr, st);
  };
  auto sort_counted = [&](int64_t n, uint64_t* k, uint64_t* v, uint64_t* ka, uint64_t* va, int b0, int b1,
                          void* scr, cudaStream_t st, bool* alt) {
    if (n > 1 && b1 > b0) nk += 5 * ((b1 - b0 + 7) / 8);
    return radix_sort_u64(n, k, v, ka, va, b0, b1, scr, st, alt);
  };
#define LAUNCHED()   \
  do {               \
    SG_CHECK_LAUNCH(); \
    info[8] = ++nk;  \
  } while (0)
  auto P = [&](int64_t off) { return ws + off; };
  uint64_t* hash = (uint64_t*)P(y.hash);
  uint64_t* loc = (uint64_t*)P(y.loc);
  int64_t* pos = (int64_t*)P(y.pos);
  int64_t* val = (int64_t*)P(y.val);
  uint32_t* cnt = (uint32_t*)P(y.cnt);
  uint16_t* flags = (uint16_t*)P(y.flags);
  uint32_t* slot = (uint32_t*)P(y.slot);
  void* rscr = P(y.radix);
  void* sscr = P(y.scan);
  Scalars* sc = (Scalars*)P(y.scal);
  Scalars h{};
  h.first_rec = ~0ull;
  h.bad = ~0ull;
  SG_CUDA(cudaMemcpyAsync(sc, &h, sizeof(Scalars), cudaMemcpyHostToDevice, s));

  const int grid = grid_of(n_lines);
  uint64_t* pk = (uint64_t*)P(y.pk);
  ChromTable ct{chrom_blob, chrom_off, chrom_size, chrom_base, chrom_mito, pk, n_chrom};
  chrom_pack<<<(n_chrom + 255) / 256, 256, 0, s>>>(ct, pk);
  LAUNCHED();
  const int pre_min = !sorted_by_barcode && min_num_fragments > 0;
  parse_kernel<<<std::min(grid, 8 * 152), kThreads, 0, s>>>(text, nbytes, line_start, n_lines, ct, shift_left, shift_right, seed, pre_min,
                                         ParseOut{hash, loc, pos, val, cnt, flags}, &sc->first_rec, &sc->max_bc,
                                         &sc->n_rec, &sc->bad, &sc->status);
  LAUNCHED();
  SG_CUDA(cudaMemcpyAsync(&h, sc, sizeof(Scalars), cudaMemcpyDeviceToHost, s));
  SG_CUDA(cudaStreamSynchronize(s));
  const int64_t nrec = (int64_t)h.n_rec;
  info[4] = nrec;
  if (h.status) {
    info[3] = (int64_t)h.bad;
    { info[8] = nk; return h.status; }
  }
  if (h.first_rec == ~0ull) { info[8] = nk; return SG_OK; }  // comments only: nothing imported
  const int paired = (h.first_rec & 1) ? 0 : 1;
  info[2] = paired;
  if (nrec == 0) { info[8] = nk; return SG_OK; }

  int64_t* lrank = nullptr;  // b[i] - 1 = rank among records with end != start
  if (sorted_by_barcode) {
    lrank = (int64_t*)P(y.b);
    mark_len<<<grid, kThreads, 0, s>>>(n_lines, flags, lrank);
    LAUNCHED();
    SG_CUDA(scan_counted(lrank, n_lines, sscr, s));
  }
  // Group records by barcode.  A table of 2^20 slots (16 MB, in L2) serves
  // most files; one that runs full is given up for one 16 times as large.
  unsigned long long* table = (unsigned long long*)P(y.table);
  unsigned long long* first = (unsigned long long*)P(y.first);
  int64_t* num = (int64_t*)P(y.num);
  uint8_t* bc = (uint8_t*)P(y.x0);  // 32 bytes a group; the sort buffers (x0 to y1, 32 bytes a line) are free until then
  Groups g{(unsigned long long*)P(y.g_recs), (unsigned long long*)P(y.g_gen), (unsigned long long*)P(y.g_total),
           (long long*)P(y.g_rmin), (long long*)P(y.g_rmax), (long long*)P(y.g_err), (int64_t*)P(y.g_leader),
           (int64_t*)P(y.g_cell), (uint8_t*)P(y.g_wl), (int64_t*)P(y.g_keep)};
  const int64_t most_slots = table_slots(n_lines);
  int64_t slots = std::min<int64_t>(most_slots, 1 << 20);
  uint64_t cur_seed = seed;
  int tries = 0;
  int64_t G = 0;
  for (;; ++tries) {
    if (tries > 0) {  // a collision: the same records keyed with another seed
      cur_seed = seed + 0x9e3779b97f4a7c15ull * (uint64_t)tries;
      rehash_records<<<grid, kThreads, 0, s>>>(n_lines, flags, loc, text, cur_seed, hash);
      LAUNCHED();
    }
    while (true) {
      SG_CUDA(cudaMemsetAsync(table, 0, slots * 8, s));
      SG_CUDA(cudaMemsetAsync(first, 0xff, slots * 8, s));
      SG_CUDA(cudaMemsetAsync(&sc->collide, 0, 8, s));  // collide and full
      table_insert<<<grid, kThreads, 0, s>>>(n_lines, flags, hash, (uint64_t)slots - 1,
                                             slots == most_slots ? slots : kProbe, table, first, slot, &sc->full);
      LAUNCHED();
      table_used<<<grid_of(slots), kThreads, 0, s>>>(slots, table, num);
      LAUNCHED();
      SG_CUDA(scan_counted(num, slots, sscr, s));
      SG_CUDA(cudaMemcpyAsync(&G, num + slots - 1, 8, cudaMemcpyDeviceToHost, s));
      SG_CUDA(cudaMemcpyAsync(&h, sc, sizeof(Scalars), cudaMemcpyDeviceToHost, s));
      SG_CUDA(cudaStreamSynchronize(s));
      if (!h.full) break;
      slots = std::min<int64_t>(most_slots, slots * 16);
    }
    init_groups<<<grid_of(G), kThreads, 0, s>>>(G, g);
    LAUNCHED();
    table_leaders<<<grid_of(slots), kThreads, 0, s>>>(slots, table, first, num, loc, text, g.leader,
                                                         bc);
    LAUNCHED();
    if (G <= kSmallGroups)
      group_stats<true><<<std::min(grid, 5 * 152), kThreads, 0, s>>>(n_lines, flags, num, first, slot, loc, text,
                                                                      reinterpret_cast<const uint4*>(bc), cnt,
                                                                      lrank, val, paired, G, g, &sc->max_abs,
                                                                      &sc->collide);
    else
      group_stats<false><<<grid, kThreads, 0, s>>>(n_lines, flags, num, first, slot, loc, text,
                                                   reinterpret_cast<const uint4*>(bc), cnt, lrank, val, paired, G, g, &sc->max_abs, &sc->collide);
    LAUNCHED();
    SG_CUDA(cudaMemcpyAsync(&h, sc, sizeof(Scalars), cudaMemcpyDeviceToHost, s));
    SG_CUDA(cudaStreamSynchronize(s));
    if (!h.collide) break;
    if (tries >= 3) return SG_ERR_COLLISION;
  }
  info[5] = G;
  info[6] = tries;
  if (has_whitelist && n_whitelist > 0) {
    uint64_t* wk0 = (uint64_t*)P(y.wk0);
    uint64_t* wv0 = (uint64_t*)P(y.wv0);
    uint64_t* wk1 = (uint64_t*)P(y.wk1);
    uint64_t* wv1 = (uint64_t*)P(y.wv1);
    wl_hash<<<grid_of(n_whitelist), kThreads, 0, s>>>(n_whitelist, wl_blob, wl_off, cur_seed, wk0, wv0);
    LAUNCHED();
    bool alt = false;
    SG_CUDA(sort_counted(n_whitelist, wk0, wv0, wk1, wv1, 0, 64, rscr, s, &alt));
    wl_lookup<<<grid_of(G), kThreads, 0, s>>>(G, g.leader, loc, text, cur_seed, n_whitelist, alt ? wk1 : wk0,
                                              alt ? wv1 : wv0, wl_blob, wl_off, g.wl);
    LAUNCHED();
  }
  decide_groups<<<grid_of(G), kThreads, 0, s>>>(G, g, flags, has_whitelist, pre_min, sorted_by_barcode,
                                                min_num_fragments, &sc->bad, &sc->status);
  LAUNCHED();
  SG_CUDA(scan_counted(g.keep, G, sscr, s));
  int64_t K = 0;
  SG_CUDA(cudaMemcpyAsync(&K, g.keep + G - 1, 8, cudaMemcpyDeviceToHost, s));
  SG_CUDA(cudaMemcpyAsync(&h, sc, sizeof(Scalars), cudaMemcpyDeviceToHost, s));
  SG_CUDA(cudaStreamSynchronize(s));
  if (h.status) {
    info[3] = (int64_t)h.bad;
    { info[8] = nk; return h.status; }
  }
  info[0] = K;
  if (K == 0) { info[8] = nk; return SG_OK; }

  // order the kept groups: first appearance, or barcode bytes
  uint64_t* x0 = (uint64_t*)P(y.x0);
  uint64_t* y0 = (uint64_t*)P(y.y0);
  uint64_t* x1 = (uint64_t*)P(y.x1);
  uint64_t* y1 = (uint64_t*)P(y.y1);
  kept_keys<<<grid_of(G), kThreads, 0, s>>>(G, g, g.keep, sorted_by_barcode, loc, x0, y0);
  LAUNCHED();
  uint64_t *ok = x0, *ov = y0, *ak = x1, *av = y1;
  auto sort_kv = [&](int bits) -> int {
    bool alt = false;
    if (sort_counted(K, ok, ov, ak, av, 0, bits, rscr, s, &alt) != cudaSuccess) return SG_ERR_CUDA;
    if (alt) {
      std::swap(ok, ak);
      std::swap(ov, av);
    }
    return SG_OK;
  };
  uint64_t* order = (uint64_t*)P(y.order);
  const unsigned kgrid = (unsigned)((K + 255) / 256);
  if (K <= kRankGroups && sorted_by_barcode) {
    rank_numbers<<<kgrid, 256, 0, s>>>(K, ok, ov, order);
    LAUNCHED();
  } else if (K <= kRankGroups && h.max_bc <= 8 * kRankWords) {
    const int nwords = (int)std::max<uint64_t>(1, (h.max_bc + 7) / 8);
    uint64_t* words = (uint64_t*)P(y.words);
    word_table<<<dim3(grid_of(K), nwords), kThreads, 0, s>>>(K, ov, g.leader, loc, text, words, sc->differ);
    LAUNCHED();
    rank_barcodes<<<kgrid, 256, 0, s>>>(K, nwords, words, sc->differ, ov, g.leader, loc, order);
    LAUNCHED();
  } else {
    if (sorted_by_barcode) {
      if (int e = sort_kv(bits_for((uint64_t)n_lines))) return e;
    } else {
      if (int e = sort_kv(bits_for(h.max_bc))) return e;
      for (int w = (int)((h.max_bc + 7) / 8) - 1; w >= 0; --w) {
        word_keys<<<grid_of(K), kThreads, 0, s>>>(K, ov, g.leader, loc, text, w, ok);
        LAUNCHED();
        if (int e = sort_kv(64)) return e;
      }
    }
    SG_CUDA(cudaMemcpyAsync(order, ov, K * 8, cudaMemcpyDeviceToDevice, s));
  }
  int64_t* row_ptr = (int64_t*)P(y.row_ptr);
  SG_CUDA(cudaMemsetAsync(row_ptr, 0, 8, s));
  cell_rows<<<grid_of(K), kThreads, 0, s>>>(K, order, g, loc, row_ptr + 1, (uint64_t*)P(y.bc), (uint64_t*)P(y.nfrag),
                                            (double*)P(y.fdup), (double*)P(y.fmito));
  LAUNCHED();
  SG_CUDA(scan_counted(row_ptr + 1, K, sscr, s));

  // the matrix: kept in-genome records sorted by (cell, position, size)
  int64_t* mcount = (int64_t*)P(y.mcount);
  const int64_t mtiles = (n_lines + kMatTile - 1) / kMatTile;
  matrix_count<<<(unsigned)mtiles, kThreads, 0, s>>>(n_lines, flags, slot, g.cell, mcount);
  LAUNCHED();
  SG_CUDA(scan_counted(mcount, mtiles, sscr, s));
  int64_t nnz = 0;
  SG_CUDA(cudaMemcpyAsync(&nnz, mcount + mtiles - 1, 8, cudaMemcpyDeviceToHost, s));
  SG_CUDA(cudaStreamSynchronize(s));
  info[1] = nnz;
  if (nnz == 0) { info[8] = nk; return SG_OK; }
  KeyLayout kl{};
  const uint64_t amax = h.max_abs;
  kl.vbias = paired ? 0 : (int64_t)amax;
  kl.vbits = bits_for(paired ? amax : 2 * amax);
  kl.pbits = bits_for(genome_size > 0 ? genome_size - 1 : 0);
  kl.rbits = bits_for((uint64_t)(K - 1));
  kl.combined = kl.vbits + kl.pbits + kl.rbits <= 64;
  info[7] = kl.combined ? 0 : 1;
  int64_t* k2 = (int64_t*)P(y.k2);
  int64_t* k3 = (int64_t*)P(y.k3);
  int64_t* mpos = (int64_t*)P(y.mpos);
  int32_t* mval = (int32_t*)P(y.mval);
  const int cbits = bits_for((uint64_t)(n_chrom - 1));
  matrix_keys<<<(unsigned)mtiles, kThreads, 0, s>>>(n_lines, flags, slot, g.cell, mcount, pos, val, chrom_base,
                                                    n_chrom, cbits, kl, x0, y0, k2, k3);
  LAUNCHED();
  if (kl.combined) {
    // Order of the matrix.  A file is nearly always in position order within
    // every chromosome, so a stable sort by (cell, chromosome), 16 bits at
    // 1,500 cells, leaves (cell, position) ascending, and only sizes at equal
    // positions may be out of order; a file in cell and genome order needs no
    // sort at all.  What each attempt left is checked, and the sort over all
    // bits (cell, position, size) is done where the checks fail, or at once
    // where its passes over 8 bytes are no more work than those over 16.
    const int full = kl.vbits + kl.pbits + kl.rbits, part = cbits + kl.rbits;
    uint64_t *src = y0, *alt = y1;
    auto settled = [&](bool* ok) -> int {
      int st[2] = {0, 0};
      SG_CUDA(cudaMemsetAsync(sc->order, 0, sizeof(st), s));
      order_check<<<grid_of(nnz), kThreads, 0, s>>>(nnz, src, kl.vbits, sc->order);
      LAUNCHED();
      SG_CUDA(cudaMemcpyAsync(st, sc->order, sizeof(st), cudaMemcpyDeviceToHost, s));
      SG_CUDA(cudaStreamSynchronize(s));
      if (!st[0] && st[1]) {
        order_mend<<<grid_of(nnz), kThreads, 0, s>>>(nnz, src, kl.vbits, sc->order);
        LAUNCHED();
        SG_CUDA(cudaMemcpyAsync(st, sc->order, sizeof(st), cudaMemcpyDeviceToHost, s));
        SG_CUDA(cudaStreamSynchronize(s));
      }
      *ok = !st[0];
      return SG_OK;
    };
    bool in_order = false;
    if (sorted_by_barcode || K == 1)
      if (int e = settled(&in_order)) return e;
    if (!in_order && 2 * ((part + 7) / 8) < (full + 7) / 8) {
      bool flip = false;
      SG_CUDA(sort_counted(nnz, x0, src, x1, alt, 0, part, rscr, s, &flip));
      if (flip) std::swap(src, alt);
      if (int e = settled(&in_order)) return e;
    }
    if (!in_order) {
      bool flip = false;
      SG_CUDA(sort_counted(nnz, src, nullptr, alt, nullptr, 0, full, rscr, s, &flip));
      if (flip) std::swap(src, alt);
    }
    decode_combined<<<grid_of(nnz), kThreads, 0, s>>>(nnz, src, kl, mpos, mval);
    LAUNCHED();
  } else {
    // LSD over three keys with the slot as payload: size, then position, then cell
    uint64_t *ck = x0, *cv = y0, *dk = x1, *dv = y1;
    bool alt = false;
    SG_CUDA(sort_counted(nnz, ck, cv, dk, dv, 0, kl.vbits, rscr, s, &alt));
    if (alt) { std::swap(ck, dk); std::swap(cv, dv); }
    // remember each slot's biased size before the keys are overwritten
    uint64_t* vb_by_slot = (uint64_t*)P(y.order);  // order is no longer needed (cells are assigned)
    scatter_by_slot<<<grid_of(nnz), kThreads, 0, s>>>(nnz, ck, cv, vb_by_slot);
    LAUNCHED();
    gather_keys<<<grid_of(nnz), kThreads, 0, s>>>(nnz, cv, k2, ck);
    LAUNCHED();
    SG_CUDA(sort_counted(nnz, ck, cv, dk, dv, 0, kl.pbits, rscr, s, &alt));
    if (alt) { std::swap(ck, dk); std::swap(cv, dv); }
    gather_keys<<<grid_of(nnz), kThreads, 0, s>>>(nnz, cv, k3, ck);
    LAUNCHED();
    SG_CUDA(sort_counted(nnz, ck, cv, dk, dv, 0, kl.rbits, rscr, s, &alt));
    if (alt) { std::swap(ck, dk); std::swap(cv, dv); }
    decode_slots<<<grid_of(nnz), kThreads, 0, s>>>(nnz, cv, k2, vb_by_slot, kl.vbias, mpos, mval);
    LAUNCHED();
  }
  SG_CUDA(cudaStreamSynchronize(s));
  info[8] = nk;
  return SG_OK;
}
#undef LAUNCHED

extern "C" int sg_frag_emit(const void* workspace, int64_t n_lines, int64_t n_whitelist, const int64_t* info,
                            int64_t* out_indptr, int64_t* out_indices, int32_t* out_data, uint64_t* out_bc_loc,
                            uint64_t* out_n_fragment, double* out_frac_dup, double* out_frac_mito, void* stream) {
  if (!workspace || !info || n_lines < 0 || n_whitelist < 0) return SG_ERR_ARG;
  const int64_t K = info[0], nnz = info[1];
  if (K <= 0) return SG_OK;
  if (!out_indptr || !out_bc_loc || !out_n_fragment || !out_frac_dup || !out_frac_mito) return SG_ERR_ARG;
  if (nnz > 0 && (!out_indices || !out_data)) return SG_ERR_ARG;
  const Layout y = frag_layout(n_lines, n_whitelist);
  const char* ws = static_cast<const char*>(workspace);
  cudaStream_t s = as_stream(stream);
  SG_CUDA(cudaMemcpyAsync(out_indptr, ws + y.row_ptr, (K + 1) * 8, cudaMemcpyDeviceToDevice, s));
  SG_CUDA(cudaMemcpyAsync(out_bc_loc, ws + y.bc, K * 8, cudaMemcpyDeviceToDevice, s));
  SG_CUDA(cudaMemcpyAsync(out_n_fragment, ws + y.nfrag, K * 8, cudaMemcpyDeviceToDevice, s));
  SG_CUDA(cudaMemcpyAsync(out_frac_dup, ws + y.fdup, K * 8, cudaMemcpyDeviceToDevice, s));
  SG_CUDA(cudaMemcpyAsync(out_frac_mito, ws + y.fmito, K * 8, cudaMemcpyDeviceToDevice, s));
  if (nnz > 0) {
    SG_CUDA(cudaMemcpyAsync(out_indices, ws + y.mpos, nnz * 8, cudaMemcpyDeviceToDevice, s));
    SG_CUDA(cudaMemcpyAsync(out_data, ws + y.mval, nnz * 4, cudaMemcpyDeviceToDevice, s));
  }
  return SG_OK;
}
