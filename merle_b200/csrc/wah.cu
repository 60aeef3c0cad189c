// wah.cu - WAH (word-aligned hybrid) compressed bitmaps: conversion between
// this library's bitmaps and the WAH streams of the reference's
// compressed-bitmap baseline, AND / OR / XOR between streams, and the
// reference's WAH file layout.
//
// Stream layout (merle/host/wahCpu.c:20-24, merle/host/wahConv.c:36-57): the
// rows are cut into 31-bit groups; a literal word (bit 31 clear) holds one
// group in its low 31 bits; a fill word (bit 31 set) stands for a run of
// groups that are all 0 (bit 30 clear) or all 0x7fffffff (bit 30 set), the
// run length in bits 0..29.  Streams written here are canonical: every run
// of equal all-0 / all-1 groups is one fill (wahCmprsCPU's output).
//
// The reference builds its GPU side from moderngpu passes (transform_scan,
// transform_lbs, transform_compact; merle/wahGpuCmprs.cu).  Here every pass works
// on blocks of 4,096 groups = 3,968 bitmap words, so that groups and words meet at
// block boundaries, and a thread on 32 groups = 31 words, so that every shift
// between the two is a constant:
//   encode  (1) per block the stream words its groups start (a group starts a
//           word when it is a literal or differs in kind from the group before
//           it): three 32-bit masks a thread; (2) each block writes its words,
//           fills with the run they have inside the block, through a
//           shared-memory buffer; (3) a block whose first groups continue the
//           run before it adds them to that fill.
//   decode  (1) group counts per block of stream words; (2) each word's first
//           group (what wahCntExcScan computes, merle/wahGpuCmprs.cu:6-14): the
//           word under every 4,096th group is noted; (3) each block of groups
//           expands the words between two notes in shared memory and composes
//           its bitmap words.
//   AND / OR / XOR: (1)-(2) of both streams, then the encoder on the groups
//           expanded from them; no bitmap is written.
// What bounds the passes is instruction issue and, at 6 to 40 microseconds each,
// the latency of a block's steps and the launches.
// 120M rows, three predicate bitmaps compressed, ANDed and the result expanded:
// 690 us with a thread per group and a binary search per output block, 373 us;
// two 600M-row bitmaps of 1 % non-zero words: 702 -> 324 us.
#include <string.h>
#include <stdio.h>
#include <algorithm>
#include <vector>
#include "common.cuh"

namespace mb {
namespace {

constexpr uint32_t WT = 256;          // threads of the stream-counting and direct passes
constexpr uint32_t WI = 16;           // stream words of a thread of the counting passes
constexpr uint32_t WB = WT * WI;      // per block
// Pieces of a thread of the direct passes, whose binary searches wait for one another (with
// 16: 1.3 to 1.55 times as long; 600M rows, one word in a thousand: 165 -> 257 us).
constexpr uint32_t DI = 8;
constexpr uint32_t DB = WT * DI;      // per block
constexpr uint32_t GT = 128;          // threads of a group block
constexpr uint32_t GB = 32 * GT;      // its groups
constexpr uint32_t GW = 31 * GT;      // its bitmap words
constexpr uint32_t GLONG = 64;        // runs longer than 32 groups a group block fills together
constexpr uint32_t FILL = 0x80000000u, ONES = 0x40000000u, CNT = 0x3fffffffu, LIT = 0x7fffffffu;
constexpr uint64_t MAX_GROUPS = CNT;  // a run must fit the 30-bit count
constexpr uint32_t WAH_MAGIC = 0x44f8a1efu;
// Blocks up to which a pass sums the block counts before its own itself instead
// of after a scan launch (at most 64 KB of counts read by each).
constexpr uint64_t DIRECT_SUM = 8192;
// mb_wah_op's automatic choice: the direct form where it is expected to be the faster,
// from what the forms take in ns.  The explicit one's time grows with the groups, the
// direct one's with the words of both streams: steeply while its few blocks wait for their
// binary searches, slowly from 2,500 words on.  Explicit / direct in us, by
// groups (across) and words (down):
//              0.6M      6.5M       19.4M       30M        58M      300M
//     200    58 / 78   85 / 76    125 / 80   165 / 82   250 / 79   986 / 80
//   2,000    55 / 133  88 / 133   146 / 134  190 / 136  288 / 135  1,124 / 133
//   6,000    57 / 145  71 / 145   146 / 148  192 / 147  289 / 147  1,129 / 148
//    200K    59 / 176  71 / 173   112 / 174  154 / 171  238 / 175  974 / 173
//      6M                                   178 / 1,227            977 / 1,282
// (The explicit form is slower by 30 % while most of its blocks hold a word or two.)  The
// form taken is within 14 % of the faster one at each of 204 points measured from 20K to
// 300M groups and 10 to 6M words; a word for every 2,048 groups, the line before, was off by
// up to 4.7 times (300M groups and 600K words: 960 us instead of 209).
inline bool direct_pays(uint64_t words, uint64_t groups) {
  const uint64_t expl = 56000 + groups * (2048 * words < groups ? 45 : 32) / 10000;
  const uint64_t direct = 76000 + std::min<uint64_t>(31 * words, 66000) + words * 2 / 11;
  return direct < expl;
}

__device__ __forceinline__ uint32_t kind_of(uint32_t v) { return v == 0 ? 0u : v == LIT ? 1u : 2u; }
__device__ __forceinline__ uint64_t word_groups(uint32_t w) { return (w & FILL) ? (w & CNT) : 1u; }
__device__ __forceinline__ uint32_t group_value(uint32_t word, uint32_t order) {
  uint32_t x = (word & FILL) ? ((word & ONES) ? LIT : 0u) : (word & LIT);
  return order ? __brev(x) >> 1 : x;
}

// Block-wide exclusive scan of one value per thread of N threads; returns the
// thread's prefix and sets *total.
template <uint32_t N, typename T>
__device__ __forceinline__ T block_excl_scan(T x, T *total) {
  __shared__ T warp_sum[N / 32];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T inc = x;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const T y = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= (uint32_t)d) inc += y;
  }
  if (lane == 31) warp_sum[warp] = inc;
  __syncthreads();
  T before = 0, all = 0;
#pragma unroll
  for (uint32_t i = 0; i < N / 32; ++i) {
    if (i < warp) before += warp_sum[i];
    all += warp_sum[i];
  }
  __syncthreads();  // warp_sum is reused by the next call
  *total = all;
  return before + inc - x;
}

// Exclusive prefix of one flag per thread over the block (lane order within
// warps, warps in order); *total = the block's flags.  All WT threads call it.
__device__ __forceinline__ uint32_t block_flag_scan(uint32_t f, uint32_t *total) {
  __shared__ uint32_t wsum[WT / 32];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t bal = __ballot_sync(0xffffffffu, f);
  if (lane == 0) wsum[warp] = __popc(bal);
  __syncthreads();
  uint32_t before = 0, all = 0;
#pragma unroll
  for (uint32_t i = 0; i < WT / 32; ++i) {
    if (i < warp) before += wsum[i];
    all += wsum[i];
  }
  __syncthreads();
  *total = all;
  return before + __popc(bal & ((1u << lane) - 1u));
}

// Exclusive scan of n block values in place (one CTA, four values a thread per
// round); v[n] = total.
__global__ void __launch_bounds__(1024) wah_scan_blocks(uint64_t *v, uint64_t n) {
  __shared__ uint64_t part[32];
  __shared__ uint64_t carry;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (uint64_t base = 0; base < n; base += 4096) {
    const uint64_t i0 = base + 4ull * threadIdx.x;
    uint64_t x[4], sum = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) x[j] = i0 + j < n ? v[i0 + j] : 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) sum += x[j];
    uint64_t inc = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint64_t y = __shfl_up_sync(0xffffffffu, inc, d);
      if (lane >= (uint32_t)d) inc += y;
    }
    if (lane == 31) part[warp] = inc;
    __syncthreads();
    uint64_t at = carry, all = 0;
    for (uint32_t k = 0; k < 32; ++k) {
      if (k < warp) at += part[k];
      all += part[k];
    }
    at += inc - sum;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (i0 + j < n) v[i0 + j] = at, at += x[j];
    __syncthreads();
    if (threadIdx.x == 0) carry += all;
    __syncthreads();
  }
  if (threadIdx.x == 0) v[n] = carry;
}

// The sum of the block values before block b: v[b] of a scanned array, else
// added up here (block-collective, N threads).
template <uint32_t N>
__device__ __forceinline__ uint64_t sum_before(const uint64_t *v, uint64_t b, bool scanned) {
  if (scanned) return v[b];
  uint64_t s = 0, total;
  for (uint64_t i0 = 0; i0 < b; i0 += 8 * N) {
    uint64_t x[8];
#pragma unroll
    for (uint32_t r = 0; r < 8; ++r) {
      const uint64_t i = i0 + r * N + threadIdx.x;
      x[r] = i < b ? v[i] : 0;
    }
#pragma unroll
    for (uint32_t r = 0; r < 8; ++r) s += x[r];
  }
  block_excl_scan<N, uint64_t>(s, &total);
  return total;
}

// ----------------------------------------------------------------- streams
// A stream prepared for reading by group blocks: note[b] and start[b] = the
// stream word under group max(GB b - 1, 0) and that word's first group, for the
// blocks that begin inside the stream; *total = the groups it stands for.
struct StreamSrc {
  const uint32_t *w;
  uint64_t n;
  const uint64_t *note;
  const uint32_t *start;
  const uint64_t *total;
};

// (1) group counts per block of WB stream words (word i * WT + t of the block in
// round i: coalesced).
__global__ void __launch_bounds__(WT) wah_dec_count(const uint32_t *wah, uint64_t n, uint64_t *bsum) {
  const uint64_t kbase = (uint64_t)blockIdx.x * WB;
  uint64_t c = 0;
#pragma unroll
  for (uint32_t i = 0; i < WI; ++i) {
    const uint64_t k = kbase + i * WT + threadIdx.x;
    if (k < n) c += word_groups(__ldg(wah + k));
  }
  uint64_t total;
  block_excl_scan<WT, uint64_t>(c, &total);
  if (threadIdx.x == 0) bsum[blockIdx.x] = total;
}

// Group blocks b in [b0, b1] have their note under word k, which starts at group
// s.
__device__ __forceinline__ void note_blocks(uint64_t *note, uint32_t *start, uint64_t b0, uint64_t b1, uint64_t k,
                                            uint32_t s, uint32_t first, uint32_t step) {
  for (uint64_t b = b0 + first; b <= b1; b += step) note[b] = k, start[b] = s;
}

// (2) every word's first group, and the notes of nblk group blocks.
__global__ void __launch_bounds__(WT) wah_dec_note(const uint32_t *wah, uint64_t n, const uint64_t *bsum, bool scanned,
                                                   uint64_t nblk, uint64_t *note, uint32_t *start, uint64_t *total) {
  // counts in round order (coalesced loads), regrouped through shared memory so
  // that each thread owns WI consecutive words: one block scan
  __shared__ uint32_t xs[WB + WB / 32];  // padded: index i at i + i / 32
  __shared__ uint64_t long_b0[GLONG], long_b1[GLONG], long_k[GLONG];
  __shared__ uint32_t long_s[GLONG], nlong;
  const uint64_t kbase = (uint64_t)blockIdx.x * WB;
  if (threadIdx.x == 0) nlong = 0;
#pragma unroll
  for (uint32_t i = 0; i < WI; ++i) {
    const uint32_t l = i * WT + threadIdx.x;
    xs[l + l / 32] = kbase + l < n ? (uint32_t)word_groups(__ldg(wah + kbase + l)) : 0u;
  }
  const uint64_t before = sum_before<WT>(bsum, blockIdx.x, scanned);  // (synchronises)
  __syncthreads();
  uint64_t sum = 0, all;
#pragma unroll
  for (uint32_t i = 0; i < WI; ++i) {
    const uint32_t l = threadIdx.x * WI + i;
    sum += xs[l + l / 32];
  }
  uint64_t at = before + block_excl_scan<WT, uint64_t>(sum, &all);
  if (threadIdx.x == 0 && kbase + WB >= n) *total = before + all;
  // (most threads' words reach no new group block)
  const bool none = at != 0 && (at / GB == (at + sum) / GB || at / GB >= nblk);
#pragma unroll 1
  for (uint32_t i = 0; i < WI && !none; ++i) {
    const uint32_t l = threadIdx.x * WI + i, ci = xs[l + l / 32];
    const uint64_t s = at, e = at + ci, k = kbase + l;
    at = e;
    if (ci == 0 || s / GB >= nblk) continue;
    // blocks b >= 1 with s <= GB b - 1 < e, and block 0 under the first group
    const uint64_t b0 = s == 0 ? 0 : s / GB + 1, b1 = e / GB < nblk ? e / GB : nblk - 1;
    if (b0 > b1) continue;
    if (b1 - b0 < 8) {
      note_blocks(note, start, b0, b1, k, (uint32_t)s, 0, 1);
    } else {
      const uint32_t r = atomicAdd(&nlong, 1u);
      if (r < GLONG) long_b0[r] = b0, long_b1[r] = b1, long_k[r] = k, long_s[r] = (uint32_t)s;
      else note_blocks(note, start, b0, b1, k, (uint32_t)s, 0, 1);
    }
  }
  __syncthreads();
  const uint32_t nl = nlong < GLONG ? nlong : GLONG;
  for (uint32_t r = 0; r < nl; ++r) note_blocks(note, start, long_b0[r], long_b1[r], long_k[r], long_s[r], threadIdx.x, WT);
}

// Index of group-block entry x (0: the group before the block, 1 + j: its group
// j) and of stream word x in shared memory, padded so that threads 32 apart hit
// different banks.
__device__ __forceinline__ uint32_t gpad(uint32_t x) { return x + (x >> 5); }
constexpr uint32_t GPAD = GB + 1 + (GB + 1) / 32 + 1;

// Entries [at, e) of a group block get value x: a short run by its lane, a long
// one through the block's list (LongRuns), filled by all threads together.
struct LongRuns {
  uint32_t lo[GLONG], hi[GLONG], v[GLONG], n;
};
__device__ __forceinline__ void place_run(uint32_t *grp, LongRuns &R, uint32_t at, uint32_t e, uint32_t x) {
  if (!x || at >= e) return;
  if (e - at <= 32) {
    for (uint32_t j = at; j < e; ++j) grp[gpad(j)] = x;
    return;
  }
  const uint32_t r = atomicAdd(&R.n, 1u);
  if (r < GLONG) R.lo[r] = at, R.hi[r] = e, R.v[r] = x;
  else
    for (uint32_t j = at; j < e; ++j) grp[gpad(j)] = x;
}

// The groups of block b (entry 1 + j: group GB b + j; entry 0: the group before)
// expanded from stream T into grp; groups past the stream are 0.  Each warp takes
// a quarter of the block's words, 32 a round: one pass for the quarters' first
// entries, one that places the words, in which a round of one-group words only
// needs no scan.  (Rounds unrolled with their words kept in registers ran 1.6x
// longer: the code outgrew the instruction cache.)  Block-collective (GT threads),
// ends synchronised.
__device__ __forceinline__ void expand_groups(const StreamSrc &T, uint64_t b, uint64_t nblk, uint32_t order,
                                              uint32_t *grp) {
  constexpr uint32_t NW = GT / 32, U = 4;
  __shared__ LongRuns R;
  __shared__ uint32_t wsum[NW];
  const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
  for (uint32_t i = t; i < GPAD; i += GT) grp[i] = 0;
  const uint64_t total = T.n ? *T.total : 0, g0 = b ? b * GB - 1 : 0, gend = (b + 1) * GB;
  if (g0 >= total) {
    __syncthreads();
    return;
  }
  const uint64_t k0 = T.note[b], k1 = gend <= total && b + 1 < nblk ? T.note[b + 1] : T.n - 1;
  const uint32_t skip = (uint32_t)(g0 - T.start[b]);  // groups of the first word before g0
  uint32_t at0 = b ? 0u : 1u;                         // entry of the next word (group g0's at first)
  for (uint64_t kc = k0; kc <= k1 && at0 <= GB; kc += GB) {
    const uint32_t m = k1 - kc + 1 < GB ? (uint32_t)(k1 - kc + 1) : GB;
    const uint32_t rounds = (m + GT - 1) / GT, i0 = warp * rounds * 32 + lane;  // the lane's words: i0 + 32 r
    const uint32_t *w = T.w + kc;
    if (t == 0) R.n = 0;
    auto load = [&](uint32_t r) -> uint32_t {  // past the words: a fill of no group
      return r < rounds && i0 + 32 * r < m ? __ldg(w + i0 + 32 * r) : FILL;
    };
    // entries a word fills; the first word's part before g0 is left out, and no
    // word counts for more than the block has
    auto fills = [&](uint32_t x, uint32_t r) -> uint32_t {
      uint32_t c = (x & FILL) ? x & CNT : 1u;
      if (kc == k0 && i0 + 32 * r == 0) c -= skip;
      return c < GB + 1 ? c : GB + 1;
    };
    uint32_t sum = 0;
    for (uint32_t r = 0; r < rounds; r += 2 * U) {
      uint32_t x[2 * U];
#pragma unroll
      for (uint32_t u = 0; u < 2 * U; ++u) x[u] = load(r + u);
#pragma unroll
      for (uint32_t u = 0; u < 2 * U; ++u) sum += fills(x[u], r + u);
    }
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (lane == 0) wsum[warp] = sum;
    __syncthreads();
    uint32_t at = at0, all = 0;
#pragma unroll
    for (uint32_t k = 0; k < NW; ++k) {
      if (k < warp) at += wsum[k];
      all += wsum[k];
    }
    uint32_t x[U];
#pragma unroll
    for (uint32_t u = 0; u < U; ++u) x[u] = load(u);
#pragma unroll 1
    for (uint32_t r = 0; r < rounds && at <= GB; r += U) {
      uint32_t y[U];  // the next words meanwhile
#pragma unroll
      for (uint32_t u = 0; u < U; ++u) y[u] = load(r + U + u);
#pragma unroll
      for (uint32_t u = 0; u < U; ++u) {
        const uint32_t c = fills(x[u], r + u), v = group_value(x[u], order);
        if (__all_sync(0xffffffffu, c == 1)) {
          if (at + lane <= GB) grp[gpad(at + lane)] = v;
          at += 32;
          continue;
        }
        uint32_t inc = c;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const uint32_t z = __shfl_up_sync(0xffffffffu, inc, d);
          if (lane >= (uint32_t)d) inc += z;
        }
        const uint32_t from = at + inc - c;
        if (c == 1) {
          if (from <= GB) grp[gpad(from)] = v;
        } else {
          place_run(grp, R, from, at + inc < GB + 1 ? at + inc : GB + 1, v);
        }
        at += __shfl_sync(0xffffffffu, inc, 31);
      }
#pragma unroll
      for (uint32_t u = 0; u < U; ++u) x[u] = y[u];
    }
    at0 = at0 + all < GB + 1 ? at0 + all : GB + 1;
    __syncthreads();
    const uint32_t nl = R.n < GLONG ? R.n : GLONG;
    for (uint32_t r = 0; r < nl; ++r)
      for (uint32_t j = R.lo[r] + t; j < R.hi[r]; j += GT) grp[gpad(j)] = R.v[r];
    __syncthreads();
  }
}

// (3) the bitmap words of group block blockIdx.x: thread t composes words 31 t ..
// 31 t + 30 of the block from its 32 groups.
__global__ void __launch_bounds__(GT) wah_dec_emit(const StreamSrc T, uint64_t nblk, uint32_t order, uint64_t nrows,
                                                   uint64_t nw, uint64_t stride, uint32_t *bm) {
  __shared__ uint32_t grp[GPAD];
  const uint32_t t = threadIdx.x;
  const uint64_t b = blockIdx.x, wbase = b * GW;
  expand_groups(T, b, nblk, order, grp);
  uint32_t v[32];
#pragma unroll
  for (uint32_t j = 0; j < 32; ++j) v[j] = grp[gpad(1 + 32 * t + j)];
  __syncthreads();
#pragma unroll
  for (uint32_t i = 0; i < 31; ++i) grp[31 * t + i] = (v[i] >> i) | (v[i + 1] << (31 - i));
  __syncthreads();
  for (uint32_t l = t; l < GW; l += GT) {
    const uint64_t w = wbase + l;
    if (w >= stride) break;
    uint32_t o = w < nw ? grp[l] : 0u;
    if (w < nw && 32 * w + 32 > nrows) o &= (1u << (nrows - 32 * w)) - 1u;
    bm[w] = o;
  }
}

// ------------------------------------------------------------------ encode
// The groups to compress: a bitmap's, or op(a, b) over two streams' (0 AND, 1 OR,
// 2 XOR).
struct EncSrc {
  const uint32_t *bm;  // the bitmap (NULL: the streams)
  uint64_t nrows, nw;  // its rows and words
  StreamSrc a, b;
  uint32_t *groups;    // the streams' combined groups: written by the counting pass, read by the writing one
  uint32_t op, order;
  uint64_t G, nblk;    // groups, group blocks
};
enum { SRC_BITMAP = 0, SRC_STREAMS = 1, SRC_GROUPS = 2 };

// The 32 groups of thread t of block b into v, and the group before them.
// Block-collective; s0: GPAD words of shared memory.
template <int SRC>
__device__ __forceinline__ uint32_t enc_groups(const EncSrc &S, uint64_t b, uint32_t (&v)[32], uint32_t *s0) {
  const uint32_t t = threadIdx.x;
  if constexpr (SRC == SRC_GROUPS) {
    const uint32_t *g = S.groups + b * GB + t;  // group j of thread t at j GT + t
#pragma unroll
    for (uint32_t j = 0; j < 32; ++j) v[j] = __ldg(g + j * GT);
    return t ? __ldg(g + 31 * GT - 1) : b ? __ldg(g - 1) : 0u;
  } else if constexpr (SRC == SRC_BITMAP) {
    // s0[4 + i] = word i of the block, s0[3] the word before; every load issued
    // before the first store
    const uint64_t base = b * GW;
    if (base + GW < S.nw && (reinterpret_cast<uintptr_t>(S.bm) & 15) == 0) {
      constexpr uint32_t Q = GW / 4, R = (Q + GT - 1) / GT;  // 16-byte pieces
      uint4 x[R];
#pragma unroll
      for (uint32_t r = 0; r < R; ++r)
        if (r * GT + t < Q) x[r] = __ldg(reinterpret_cast<const uint4 *>(S.bm + base) + r * GT + t);
      if (t == 0) s0[3] = b ? __ldg(S.bm + base - 1) : 0u;
#pragma unroll
      for (uint32_t r = 0; r < R; ++r)
        if (r * GT + t < Q) reinterpret_cast<uint4 *>(s0 + 4)[r * GT + t] = x[r];
    } else {
      uint32_t x[31];
#pragma unroll
      for (uint32_t r = 0; r < 31; ++r) {
        const uint64_t w = base + r * GT + t;
        x[r] = w < S.nw ? __ldg(S.bm + w) : 0u;
        if (w < S.nw && w * 32 + 32 > S.nrows) x[r] &= (1u << (S.nrows - w * 32)) - 1u;
      }
      if (t == 0) s0[3] = b ? __ldg(S.bm + base - 1) : 0u;
#pragma unroll
      for (uint32_t r = 0; r < 31; ++r) s0[4 + r * GT + t] = x[r];
    }
    __syncthreads();
    // groups 32 t + j: bits 31 j .. 31 j + 30 of the thread's 31 words
    const uint32_t *w = s0 + 4 + 31 * t;
    uint32_t prev = w[-1] >> 1, lo = w[0];
    v[0] = lo & LIT;
#pragma unroll
    for (uint32_t j = 1; j < 31; ++j) {
      const uint32_t hi = w[j];
      v[j] = __funnelshift_r(lo, hi, 32 - j) & LIT;
      lo = hi;
    }
    v[31] = lo >> 1;
    if (S.order) {
#pragma unroll
      for (uint32_t j = 0; j < 32; ++j) v[j] = __brev(v[j]) >> 1;
      prev = __brev(prev) >> 1;
    }
    return prev;
  } else {
    expand_groups(S.a, b, S.nblk, 0, s0);
    uint32_t prev = s0[gpad(32 * t)];
#pragma unroll
    for (uint32_t j = 0; j < 32; ++j) v[j] = s0[gpad(1 + 32 * t + j)];
    __syncthreads();
    expand_groups(S.b, b, S.nblk, 0, s0);
    const uint32_t q = s0[gpad(32 * t)];
    prev = S.op == 0 ? prev & q : S.op == 1 ? prev | q : prev ^ q;
#pragma unroll
    for (uint32_t j = 0; j < 32; ++j) {
      const uint32_t x = s0[gpad(1 + 32 * t + j)];
      v[j] = S.op == 0 ? v[j] & x : S.op == 1 ? v[j] | x : v[j] ^ x;
      S.groups[b * GB + j * GT + t] = v[j];
    }
    return prev;
  }
}

// Which of a thread's valid groups (bits of `valid`) are literals, and which start
// a stream word: a literal, the table's first group, or a kind unlike the group
// before.
struct GroupMasks {
  uint32_t lit, ones, start;
};
__device__ __forceinline__ GroupMasks group_masks(const uint32_t (&v)[32], uint32_t prev, uint32_t valid, bool first) {
  uint32_t z = 0, o = 0;
#pragma unroll
  for (uint32_t j = 0; j < 32; ++j) {
    z |= (v[j] == 0 ? 1u : 0u) << j;
    o |= (v[j] == LIT ? 1u : 0u) << j;
  }
  GroupMasks M;
  M.lit = ~(z | o) & valid;
  M.ones = o;
  M.start = (M.lit | (z & ~(z << 1 | (prev == 0 ? 1u : 0u))) | (o & ~(o << 1 | (prev == LIT ? 1u : 0u))) |
             (first ? 1u : 0u)) & valid;
  return M;
}

__device__ __forceinline__ uint32_t valid_groups(const EncSrc &S, uint64_t b, uint32_t t) {  // of thread t: 0 .. 32
  const uint64_t g = b * GB + 32ull * t;
  return g >= S.G ? 0u : S.G - g < 32 ? (uint32_t)(S.G - g) : 32u;
}

// (1) stream words each block starts.
template <int SRC>
__global__ void __launch_bounds__(GT) wah_enc_count(const __grid_constant__ EncSrc S, uint64_t *bcnt) {
  __shared__ __align__(16) uint32_t s0[GPAD];
  const uint64_t b = blockIdx.x;
  uint32_t v[32];
  const uint32_t prev = enc_groups<SRC>(S, b, v, s0);
  const uint32_t nv = valid_groups(S, b, threadIdx.x);
  const GroupMasks M = group_masks(v, prev, nv == 32 ? 0xffffffffu : (1u << nv) - 1u, b == 0 && threadIdx.x == 0);
  uint32_t total;
  block_excl_scan<GT, uint32_t>(__popc(M.start), &total);
  if (threadIdx.x == 0) bcnt[b] = total;
}

// (2) the stream words, in order: literals, and fills with the part of their run
// that lies in the block.  off[b] = the block's first word, cont[b] = its groups
// that continue the run before it; *nwords = the stream's words.
template <int SRC>
__global__ void __launch_bounds__(GT, 7) wah_enc_write(const __grid_constant__ EncSrc S, const uint64_t *bcnt,
                                                    bool scanned, uint32_t *out, uint64_t *off, uint32_t *cont,
                                                    uint64_t *nwords) {
  __shared__ __align__(16) uint32_t s0[GPAD];
  __shared__ uint32_t wfirst[GT / 32];  // per warp: groups before its first start (all its groups if none)
  __shared__ uint32_t whas[GT / 32];
  const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const uint64_t b = blockIdx.x;
  uint32_t v[32];
  const uint32_t prev = enc_groups<SRC>(S, b, v, s0);
  const uint32_t nv = valid_groups(S, b, t);
  const GroupMasks M = group_masks(v, prev, nv == 32 ? 0xffffffffu : (1u << nv) - 1u, b == 0 && t == 0);
  const uint64_t at = sum_before<GT>(bcnt, b, scanned);
  uint32_t total;
  uint32_t pos = block_excl_scan<GT, uint32_t>(__popc(M.start), &total);
  // groups from the end of the thread's to the next start, or to the block's end
  const uint32_t first = M.start ? (uint32_t)__ffs(M.start) - 1 : nv;
  const uint32_t has = __ballot_sync(0xffffffffu, M.start != 0);
  const uint32_t wgroups = __reduce_add_sync(0xffffffffu, nv);
  const uint32_t fl = has ? (uint32_t)__ffs(has) - 1 : 0u, ff = __shfl_sync(0xffffffffu, first, fl);
  if (lane == 0) wfirst[warp] = has ? 32 * fl + ff : wgroups, whas[warp] = has ? 1u : 0u;
  __syncthreads();
  const uint32_t later = lane == 31 ? 0u : has & (0xffffffffu << (lane + 1));
  const uint32_t nl = later ? (uint32_t)__ffs(later) - 1 : lane, nf = __shfl_sync(0xffffffffu, first, nl);
  uint32_t dist;
  if (later) {
    dist = 32 * (nl - lane - 1) + nf;
  } else {
    dist = wgroups > 32 * (lane + 1) ? wgroups - 32 * (lane + 1) : 0u;
    for (uint32_t w = warp + 1; w < GT / 32; ++w) {
      dist += wfirst[w];
      if (whas[w]) break;
    }
  }
  if (t == 0) {
    uint32_t c = 0;
    for (uint32_t w = 0; w < GT / 32; ++w) {
      c += wfirst[w];
      if (whas[w]) break;
    }
    off[b] = at;
    cont[b] = c;
    if (b + 1 == S.nblk) *nwords = at + total;
  }
  // the words into s0 (at most GB), then out
#pragma unroll
  for (uint32_t j = 0; j < 32; ++j)
    if ((M.start >> j) & 1u) {
      uint32_t w = v[j];
      if (!((M.lit >> j) & 1u)) {
        const uint32_t rest = M.start >> j >> 1;
        const uint32_t run = rest ? (uint32_t)__ffs(rest) : nv - j + dist;
        w = FILL | ((M.ones >> j) & 1u ? ONES : 0u) | run;
      }
      s0[pos++] = w;
    }
  __syncthreads();
  for (uint32_t i = t; i < total; i += GT) out[at + i] = s0[i];
}

// (3) a block's groups before its first start belong to the last fill before it.
__global__ void wah_enc_join(uint32_t *out, const uint64_t *off, const uint32_t *cont, uint64_t nblk) {
  const uint64_t b = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (b == 0 || b >= nblk) return;
  if (cont[b]) atomicAdd(&out[off[b] - 1], cont[b]);
}

// (direct) fill runs.
__global__ void wah_enc_fills(uint32_t *out, const uint32_t *pos, uint64_t K, uint64_t G) {
  for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < K; k += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t w = out[k];
    if (w & FILL) {
      const uint64_t next = k + 1 < K ? pos[k + 1] : G;
      out[k] = w + (uint32_t)(next - pos[k]);
    }
  }
}

// Largest k in [lo, hi] with S[k] <= g (S ascending, S[lo] <= g).
__device__ __forceinline__ uint64_t last_le(const uint32_t *S, uint64_t lo, uint64_t hi, uint64_t g) {
  while (lo < hi) {
    const uint64_t mid = lo + (hi - lo + 1) / 2;
    if (S[mid] <= g) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// (direct) the exclusive scan of every word's group count; S[n] = total.
// S is stored saturated at 2^32 - 1: lookups are of groups below 2^30 only, and
// min(x, cap) keeps the order of every prefix below the cap.
__device__ __forceinline__ uint32_t sat32(uint64_t x) { return x > 0xffffffffull ? 0xffffffffu : (uint32_t)x; }

__global__ void __launch_bounds__(WT) wah_dec_scan(const uint32_t *wah, uint64_t n, const uint64_t *boff,
                                                   uint64_t nblk, uint32_t *S) {
  // counts in round order (coalesced loads), regrouped through shared
  // memory so that each thread owns WI consecutive words: one block scan
  __shared__ uint32_t xs[WB + WB / 32];  // padded: index i at i + i / 32
  const uint64_t kbase = (uint64_t)blockIdx.x * WB;
  uint32_t c[WI];
#pragma unroll
  for (uint32_t i = 0; i < WI; ++i) {
    const uint64_t k = kbase + i * WT + threadIdx.x;
    c[i] = k < n ? (uint32_t)word_groups(__ldg(wah + k)) : 0u;
  }
#pragma unroll
  for (uint32_t i = 0; i < WI; ++i) {
    const uint32_t l = i * WT + threadIdx.x;
    xs[l + l / 32] = c[i];
  }
  __syncthreads();
  uint64_t sum = 0;
#pragma unroll
  for (uint32_t i = 0; i < WI; ++i) {
    const uint32_t l = threadIdx.x * WI + i;
    c[i] = xs[l + l / 32];
    sum += c[i];
  }
  uint64_t total;
  uint64_t at = boff[blockIdx.x] + block_excl_scan<WT, uint64_t>(sum, &total);
#pragma unroll
  for (uint32_t i = 0; i < WI; ++i) {
    const uint32_t l = threadIdx.x * WI + i;
    xs[l + l / 32] = sat32(at);
    at += c[i];
  }
  __syncthreads();
#pragma unroll
  for (uint32_t i = 0; i < WI; ++i) {
    const uint32_t l = i * WT + threadIdx.x;
    const uint64_t k = kbase + l;
    if (k < n) S[k] = xs[l + l / 32];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) S[n] = sat32(boff[nblk]);
}

// A pinned host word per thread that kernels write a result to.
struct HostWord {
  uint64_t *p = nullptr;
  ~HostWord() {
    if (p) cudaFreeHost(p);
  }
};
mb_status host_word(uint64_t **out) {
  static thread_local HostWord w;
  if (!w.p) MB_CUDA(cudaHostAlloc(reinterpret_cast<void **>(&w.p), sizeof(uint64_t), cudaHostAllocPortable | cudaHostAllocMapped));
  *out = w.p;
  return MB_OK;
}

// A call's scratch: one allocation, carved into 16-byte aligned pieces (an
// allocation and its release cost the host 3-4 us a pair).
struct Carve {
  uint8_t *base = nullptr;
  size_t used = 0;  // counted without a base, handed out with one
  template <typename T>
  T *take(uint64_t n) {
    T *p = reinterpret_cast<T *>(base ? base + used : nullptr);
    used += round_up(std::max<uint64_t>(n, 1) * sizeof(T), 16);
    return p;
  }
};
// Runs `plan` twice: to count the bytes, then with them allocated.
template <typename F>
mb_status carve(Scratch &sc, F plan) {
  Carve c;
  plan(c);
  MB_CHECK(sc.get(&c.base, c.used));
  c.used = 0;
  plan(c);
  return MB_OK;
}

// Block values v[0 .. n) ready for sum_before: scanned when there are many, or
// when the caller needs the total in v[n].
mb_status block_sums(uint64_t *v, uint64_t n, bool total, bool *scanned, cudaStream_t st) {
  *scanned = total || n > DIRECT_SUM;
  if (!*scanned) return MB_OK;
  wah_scan_blocks<<<1, 1024, 0, st>>>(v, n);
  MB_LAUNCH_CHECK("wah_scan_blocks");
  return MB_OK;
}

// Scratch of an encoding of nblk group blocks, and of a stream's notes for them.
struct EncBufs {
  uint64_t *bcnt, *off, *total;
  uint32_t *cont, *groups;
  void plan(Carve &c, uint64_t nblk, bool streams) {
    groups = streams ? c.take<uint32_t>(nblk * GB) : nullptr;
    bcnt = c.take<uint64_t>(nblk + 1), off = c.take<uint64_t>(nblk), cont = c.take<uint32_t>(nblk);
    total = c.take<uint64_t>(1);
  }
};
struct NoteBufs {
  uint64_t *bsum, *note;
  uint32_t *start;
  void plan(Carve &c, uint64_t n, uint64_t nblk) {
    bsum = c.take<uint64_t>(ceil_div(n, WB) + 2), note = c.take<uint64_t>(nblk), start = c.take<uint32_t>(nblk);
  }
};

// Encodes the groups of S into out (capacity words); *nwords = words of the
// stream, also when it does not fit (nothing is written then).
template <int SRC>
mb_status encode(const EncSrc &S, const EncBufs &B, uint32_t *out, uint64_t capacity, uint64_t *nwords,
                 cudaStream_t st, const char *who) {
  const unsigned grid = (unsigned)S.nblk;
  uint64_t *hw;
  MB_CHECK(host_word(&hw));
  wah_enc_count<SRC><<<grid, GT, 0, st>>>(S, B.bcnt);
  MB_LAUNCH_CHECK("wah_enc_count");
  // a stream has at most a word a group: only a smaller output needs the size first
  const bool sized = !out || capacity < S.G;
  bool scanned = false;
  MB_CHECK(block_sums(B.bcnt, S.nblk, sized, &scanned, st));
  if (sized) {
    MB_CUDA(cudaMemcpyAsync(hw, B.bcnt + S.nblk, 8, cudaMemcpyDeviceToHost, st));
    MB_CUDA(cudaStreamSynchronize(st));
    *nwords = *hw;
    if (!out) return MB_OK;  // a size query
    if (*nwords > capacity) return fail(MB_ERR_INVALID, "%s: the stream has %llu words, the output holds %llu", who,
                                        (unsigned long long)*nwords, (unsigned long long)capacity);
  }
  // the words to the host, unless it has them: the call need not wait again then
  wah_enc_write<SRC == SRC_STREAMS ? SRC_GROUPS : SRC><<<grid, GT, 0, st>>>(S, B.bcnt, scanned, out, B.off, B.cont,
                                                                           sized ? B.total : hw);
  MB_LAUNCH_CHECK("wah_enc_write");
  if (S.nblk > 1) {
    wah_enc_join<<<(unsigned)ceil_div(S.nblk, 256), 256, 0, st>>>(out, B.off, B.cont, S.nblk);
    MB_LAUNCH_CHECK("wah_enc_join");
  }
  if (sized) return MB_OK;
  MB_CUDA(cudaStreamSynchronize(st));  // *hw
  *nwords = *hw;
  return MB_OK;
}

// The notes of stream (wah, n) for nblk group blocks.
mb_status prepare_stream(const uint32_t *wah, uint64_t n, uint64_t nblk, const NoteBufs &B, StreamSrc *T,
                         cudaStream_t st) {
  *T = StreamSrc{wah, n, nullptr, nullptr, nullptr};
  if (n == 0) return MB_OK;
  const uint64_t sblk = ceil_div(n, WB);
  wah_dec_count<<<(unsigned)sblk, WT, 0, st>>>(wah, n, B.bsum);
  MB_LAUNCH_CHECK("wah_dec_count");
  bool scanned = false;
  MB_CHECK(block_sums(B.bsum, sblk, false, &scanned, st));
  wah_dec_note<<<(unsigned)sblk, WT, 0, st>>>(wah, n, B.bsum, scanned, nblk, B.note, B.start, B.bsum + sblk + 1);
  MB_LAUNCH_CHECK("wah_dec_note");
  T->note = B.note, T->start = B.start, T->total = B.bsum + sblk + 1;
  return MB_OK;
}

// The exclusive scan of the stream's group counts into a new scratch array
// S[0..n] (S[n] = the groups the stream stands for).
mb_status group_scan(const uint32_t *wah, uint64_t n, Scratch &sc, uint32_t **S_out, cudaStream_t st) {
  const uint64_t nblk = ceil_div(n, WB);
  uint64_t *boff;
  uint32_t *S;
  MB_CHECK(sc.get(&boff, nblk + 1));
  MB_CHECK(sc.get(&S, n + 1));
  wah_dec_count<<<(unsigned)nblk, WT, 0, st>>>(wah, n, boff);
  MB_LAUNCH_CHECK("wah_dec_count");
  wah_scan_blocks<<<1, 1024, 0, st>>>(boff, nblk);
  MB_LAUNCH_CHECK("wah_scan_blocks");
  wah_dec_scan<<<(unsigned)nblk, WT, 0, st>>>(wah, n, boff, nblk, S);
  MB_LAUNCH_CHECK("wah_dec_scan");
  *S_out = S;
  return MB_OK;
}

mb_status decode(const uint32_t *wah, uint64_t n, uint32_t order, uint64_t nrows, uint32_t *bm, cudaStream_t st) {
  const uint64_t stride = mb_bitmap_stride(nrows), nw = mb_bitmap_words(nrows);
  if (stride == 0) return MB_OK;
  if (n == 0) {
    MB_CUDA(cudaMemsetAsync(bm, 0, stride * 4, st));
    return MB_OK;
  }
  Scratch sc(st);
  const uint64_t nblk = ceil_div(stride, GW);
  NoteBufs B;
  MB_CHECK(carve(sc, [&](Carve &c) { B.plan(c, n, nblk); }));
  StreamSrc T;
  MB_CHECK(prepare_stream(wah, n, nblk, B, &T, st));
  wah_dec_emit<<<(unsigned)nblk, GT, 0, st>>>(T, nblk, order, nrows, nw, stride, bm);
  MB_LAUNCH_CHECK("wah_dec_emit");
  return MB_OK;
}

bool aligned4(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 3) == 0; }

// ----------------------------------------------- direct (compressed) ops
// The reference's direct operations (wahAnd / wahOr / wahXor,
// merle/wahGpuDirect.cu) never expand the streams: the runs of both are cut
// at the union of their word boundaries and each piece is combined whole.
// Here: (1) the group scans SA, SB of both streams (saturated, clamped to G);
// (2) a merge of the two boundary lists by rank (an A boundary's rank is its
// index plus the B boundaries below it, a B boundary's its index plus the A
// boundaries at or below it); (3) piece r is [m[r], m[r+1]) (the last one
// ends at G), its value op(A's word, B's word) at its first group; a piece
// starts an output word when its value is a literal or its kind differs from
// the kind at the group before it; (4) fill runs as in the encoder.
struct DirectSrc {
  const uint32_t *a, *b, *SA, *SB;  // streams and their exclusive group scans
  uint64_t na, nb, G;
  uint32_t op;
};

// Value (31 bits) of op(A, B) at group g (< G), with its kind.
__device__ __forceinline__ uint32_t direct_value(const DirectSrc &D, uint64_t g) {
  uint32_t va = 0, vb = 0;
  if (D.na && g < D.SA[D.na]) va = group_value(__ldg(D.a + last_le(D.SA, 0, D.na - 1, g)), 0);
  if (D.nb && g < D.SB[D.nb]) vb = group_value(__ldg(D.b + last_le(D.SB, 0, D.nb - 1, g)), 0);
  return D.op == 0 ? va & vb : D.op == 1 ? va | vb : va ^ vb;
}

__device__ __forceinline__ uint32_t clamp_g(uint32_t x, uint64_t G) { return x < G ? x : (uint32_t)G; }

// (2) the merged boundary list m[0 .. na + nb + 1].
__global__ void wah_direct_merge(const DirectSrc D, uint32_t *m) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i <= D.na) {
    const uint32_t v = clamp_g(D.SA[i], D.G);
    uint64_t lo = 0, hi = D.nb + 1;  // B boundaries < v
    while (lo < hi) {
      const uint64_t mid = (lo + hi) / 2;
      if (clamp_g(D.SB[mid], D.G) < v) lo = mid + 1;
      else hi = mid;
    }
    m[i + lo] = v;
  } else if (i <= D.na + 1 + D.nb) {
    const uint64_t j = i - D.na - 1;
    const uint32_t v = clamp_g(D.SB[j], D.G);
    uint64_t lo = 0, hi = D.na + 1;  // A boundaries <= v
    while (lo < hi) {
      const uint64_t mid = (lo + hi) / 2;
      if (clamp_g(D.SA[mid], D.G) <= v) lo = mid + 1;
      else hi = mid;
    }
    m[j + lo] = v;
  }
}

// Piece r starts an output word: *v = its value, *x = its first group.
__device__ __forceinline__ bool direct_flag(const DirectSrc &D, const uint32_t *m, uint64_t M, uint64_t r,
                                            uint32_t *v, uint64_t *x) {
  if (r >= M) return false;
  const uint64_t x0 = m[r], y0 = r + 1 < M ? m[r + 1] : D.G;
  *x = x0;
  if (x0 >= y0 || x0 >= D.G) return false;
  *v = direct_value(D, x0);
  const uint32_t k = kind_of(*v);
  if (k == 2u || x0 == 0) return true;
  return k != kind_of(direct_value(D, x0 - 1));
}

// (3a) output words per block of DB pieces.
__global__ void __launch_bounds__(WT) wah_direct_count(const DirectSrc D, const uint32_t *m, uint64_t M,
                                                       uint64_t *bcnt) {
  uint32_t c = 0, v;
  uint64_t x;
#pragma unroll
  for (uint32_t i = 0; i < DI; ++i)
    c += direct_flag(D, m, M, (uint64_t)blockIdx.x * DB + i * WT + threadIdx.x, &v, &x) ? 1u : 0u;
  uint64_t total;
  block_excl_scan<WT, uint64_t>(c, &total);
  if (threadIdx.x == 0) bcnt[blockIdx.x] = total;
}

// (3b) the words, in piece order; each word's first group into pos.
__global__ void __launch_bounds__(WT) wah_direct_write(const DirectSrc D, const uint32_t *m, uint64_t M,
                                                       const uint64_t *boff, uint32_t *out, uint32_t *pos) {
  uint64_t at = boff[blockIdx.x];
#pragma unroll 1
  for (uint32_t i = 0; i < DI; ++i) {
    uint32_t v = 0, total;
    uint64_t x = 0;
    const bool f = direct_flag(D, m, M, (uint64_t)blockIdx.x * DB + i * WT + threadIdx.x, &v, &x);
    const uint32_t ex = block_flag_scan(f ? 1u : 0u, &total);
    if (f) {
      const uint32_t k = kind_of(v);
      out[at + ex] = k == 2u ? v : (k == 1u ? FILL | ONES : FILL);
      pos[at + ex] = (uint32_t)x;
    }
    at += total;
  }
}

mb_status direct_op(uint32_t op, const uint32_t *a, uint64_t na, const uint32_t *b, uint64_t nb, uint64_t G,
                    uint32_t *out, uint64_t capacity, uint64_t *nwords, cudaStream_t st) {
  Scratch sc(st);
  DirectSrc D{a, b, nullptr, nullptr, na, nb, G, op};
  uint32_t *SA, *SB, *m;
  const uint32_t zero = 0;
  if (na) {
    MB_CHECK(group_scan(a, na, sc, &SA, st));
  } else {
    MB_CHECK(sc.get(&SA, 1));
    MB_CUDA(cudaMemcpyAsync(SA, &zero, 4, cudaMemcpyHostToDevice, st));
  }
  if (nb) {
    MB_CHECK(group_scan(b, nb, sc, &SB, st));
  } else {
    MB_CHECK(sc.get(&SB, 1));
    MB_CUDA(cudaMemcpyAsync(SB, &zero, 4, cudaMemcpyHostToDevice, st));
  }
  D.SA = SA, D.SB = SB;
  const uint64_t M = na + nb + 2;
  MB_CHECK(sc.get(&m, M));
  wah_direct_merge<<<(unsigned)ceil_div(M, 256), 256, 0, st>>>(D, m);
  MB_LAUNCH_CHECK("wah_direct_merge");
  const uint64_t nblk = ceil_div(M, DB);
  uint64_t *boff;
  MB_CHECK(sc.get(&boff, nblk + 1));
  wah_direct_count<<<(unsigned)nblk, WT, 0, st>>>(D, m, M, boff);
  MB_LAUNCH_CHECK("wah_direct_count");
  wah_scan_blocks<<<1, 1024, 0, st>>>(boff, nblk);
  MB_LAUNCH_CHECK("wah_scan_blocks");
  uint64_t K = 0;
  MB_CUDA(cudaMemcpyAsync(&K, boff + nblk, 8, cudaMemcpyDeviceToHost, st));
  MB_CUDA(cudaStreamSynchronize(st));
  *nwords = K;
  if (!out) return MB_OK;
  if (K > capacity) return fail(MB_ERR_INVALID, "mb_wah_op: the stream has %llu words, the output holds %llu",
                                (unsigned long long)K, (unsigned long long)capacity);
  uint32_t *pos;
  MB_CHECK(sc.get(&pos, K));
  wah_direct_write<<<(unsigned)nblk, WT, 0, st>>>(D, m, M, boff, out, pos);
  MB_LAUNCH_CHECK("wah_direct_write");
  const unsigned grid = (unsigned)std::min<uint64_t>(ceil_div(K, 256), (uint64_t)dev_info().sms * 8);
  wah_enc_fills<<<grid, 256, 0, st>>>(out, pos, K, G);
  MB_LAUNCH_CHECK("wah_enc_fills");
  return MB_OK;
}

}  // namespace
}  // namespace mb

using namespace mb;

extern "C" uint64_t mb_wah_groups(uint64_t nrows) { return ceil_div(nrows, 31); }

extern "C" mb_status mb_wah_encode(const uint32_t *bitmap, uint64_t nrows, uint32_t order, uint32_t *wah,
                                   uint64_t capacity, uint64_t *nwords, void *stream) {
  NvtxRange nvtx_("mb_wah_encode");
  if (!nwords) return fail(MB_ERR_INVALID, "mb_wah_encode: NULL word count");
  *nwords = 0;
  if (nrows && !bitmap) return fail(MB_ERR_INVALID, "mb_wah_encode: NULL bitmap");
  if (order > 1) return fail(MB_ERR_INVALID, "mb_wah_encode: order %u (0 or 1)", order);
  if (ceil_div(nrows, 31) > MAX_GROUPS)
    return fail(MB_ERR_INVALID, "mb_wah_encode: %llu rows exceed the 30-bit run count", (unsigned long long)nrows);
  if (!aligned4(bitmap) || !aligned4(wah)) return fail(MB_ERR_INVALID, "mb_wah_encode: misaligned pointer");
  EncSrc S{};
  S.bm = bitmap, S.nrows = nrows, S.nw = mb_bitmap_words(nrows), S.order = order, S.G = ceil_div(nrows, 31);
  if (S.G == 0) return MB_OK;
  S.nblk = ceil_div(S.G, GB);
  cudaStream_t st = as_stream(stream);
  Scratch sc(st);
  EncBufs B;
  MB_CHECK(carve(sc, [&](Carve &c) { B.plan(c, S.nblk, false); }));
  return encode<SRC_BITMAP>(S, B, wah, capacity, nwords, st, "mb_wah_encode");
}

extern "C" mb_status mb_wah_decode(const uint32_t *wah, uint64_t nwords, uint32_t order, uint64_t nrows,
                                   uint32_t *bitmap, void *stream) {
  NvtxRange nvtx_("mb_wah_decode");
  if (nwords && !wah) return fail(MB_ERR_INVALID, "mb_wah_decode: NULL stream");
  if (nrows && !bitmap) return fail(MB_ERR_INVALID, "mb_wah_decode: NULL bitmap");
  if (order > 1) return fail(MB_ERR_INVALID, "mb_wah_decode: order %u (0 or 1)", order);
  if (!aligned4(bitmap) || !aligned4(wah)) return fail(MB_ERR_INVALID, "mb_wah_decode: misaligned pointer");
  return decode(wah, nwords, order, nrows, bitmap, as_stream(stream));
}

extern "C" mb_status mb_wah_ngroups(const uint32_t *wah, uint64_t nwords, uint64_t *ngroups, void *stream) {
  if (!ngroups || (nwords && !wah)) return fail(MB_ERR_INVALID, "mb_wah_ngroups: NULL argument");
  *ngroups = 0;
  if (nwords == 0) return MB_OK;
  cudaStream_t st = as_stream(stream);
  Scratch sc(st);
  const uint64_t nblk = ceil_div(nwords, WB);
  uint64_t *boff;
  MB_CHECK(sc.get(&boff, nblk + 1));
  wah_dec_count<<<(unsigned)nblk, WT, 0, st>>>(wah, nwords, boff);
  MB_LAUNCH_CHECK("wah_dec_count");
  wah_scan_blocks<<<1, 1024, 0, st>>>(boff, nblk);
  MB_LAUNCH_CHECK("wah_scan_blocks");
  MB_CUDA(cudaMemcpyAsync(ngroups, boff + nblk, 8, cudaMemcpyDeviceToHost, st));
  MB_CUDA(cudaStreamSynchronize(st));
  return MB_OK;
}

extern "C" mb_status mb_wah_op(uint32_t op, const uint32_t *a, uint64_t na, const uint32_t *b, uint64_t nb,
                               uint64_t ngroups, uint32_t *out, uint64_t capacity, uint64_t *nwords, void *stream) {
  return mb_wah_op_ex(op, a, na, b, nb, ngroups, MB_WAH_AUTO, out, capacity, nwords, stream);
}

extern "C" mb_status mb_wah_op_ex(uint32_t op, const uint32_t *a, uint64_t na, const uint32_t *b, uint64_t nb,
                                  uint64_t ngroups, uint32_t method, uint32_t *out, uint64_t capacity,
                                  uint64_t *nwords, void *stream) {
  NvtxRange nvtx_("mb_wah_op");
  if (!nwords) return fail(MB_ERR_INVALID, "mb_wah_op: NULL word count");
  *nwords = 0;
  if (op > MB_WAH_XOR) return fail(MB_ERR_INVALID, "mb_wah_op: op %u", op);
  if (method > MB_WAH_DIRECT) return fail(MB_ERR_INVALID, "mb_wah_op: method %u", method);
  if ((na && !a) || (nb && !b)) return fail(MB_ERR_INVALID, "mb_wah_op: NULL stream");
  if (ngroups > MAX_GROUPS) return fail(MB_ERR_INVALID, "mb_wah_op: %llu groups exceed the 30-bit run count",
                                        (unsigned long long)ngroups);
  if (ngroups == 0) return MB_OK;
  cudaStream_t st = as_stream(stream);
  // the direct form's work follows the words (with binary searches per piece), the
  // other form's the groups
  if (method == MB_WAH_DIRECT || (method == MB_WAH_AUTO && direct_pays(na + nb, ngroups)))
    return direct_op(op, a, na, b, nb, ngroups, out, capacity, nwords, st);
  // the encoder on the groups of both streams, expanded block by block (their
  // bit order is immaterial: both sides and the result keep their own)
  Scratch sc(st);
  EncSrc S{};
  S.op = op, S.G = ngroups, S.nblk = ceil_div(ngroups, GB);
  EncBufs B;
  NoteBufs A1, A2;
  MB_CHECK(carve(sc, [&](Carve &c) { B.plan(c, S.nblk, true), A1.plan(c, na, S.nblk), A2.plan(c, nb, S.nblk); }));
  MB_CHECK(prepare_stream(a, na, S.nblk, A1, &S.a, st));
  MB_CHECK(prepare_stream(b, nb, S.nblk, A2, &S.b, st));
  S.groups = B.groups;
  return encode<SRC_STREAMS>(S, B, out, capacity, nwords, st, "mb_wah_op");
}

// The reference's WAH file (struct wahHost_s, merle/host/wahCpu.h:10-15, read
// whole by loadWahFile, merle/host/wahConv.c:93-109): has1Fill (bool, then 3
// pad bytes), magic 0x44f8a1ef, cmprsNrWord, decmprsNrWord (uint64 each),
// then the stream words.
namespace {
struct WahFileHdr {
  uint8_t has1fill, pad[3];
  uint32_t magic;
  uint64_t cmprs, decmprs;
};
static_assert(sizeof(WahFileHdr) == 24, "the reference's header is 24 bytes");
}  // namespace

extern "C" mb_status mb_wah_save(const char *path, const uint32_t *words, uint64_t nwords, uint64_t ngroups) {
  if (!path || (nwords && !words)) return fail(MB_ERR_INVALID, "mb_wah_save: NULL argument");
  WahFileHdr h{};
  h.magic = WAH_MAGIC;
  h.cmprs = nwords;
  h.decmprs = ngroups;
  for (uint64_t i = 0; i < nwords; ++i)
    if ((words[i] >> 30) == 3u) {
      h.has1fill = 1;
      break;
    }
  FILE *f = fopen(path, "wb");
  if (!f) return fail(MB_ERR_IO, "mb_wah_save: cannot open %s", path);
  bool ok = fwrite(&h, sizeof(h), 1, f) == 1 && (nwords == 0 || fwrite(words, 4, nwords, f) == nwords);
  ok = fclose(f) == 0 && ok;
  return ok ? MB_OK : fail(MB_ERR_IO, "mb_wah_save: write to %s failed", path);
}

extern "C" mb_status mb_wah_load(const char *path, uint32_t *words, uint64_t capacity, uint64_t *nwords,
                                 uint64_t *ngroups) {
  if (!path || !nwords) return fail(MB_ERR_INVALID, "mb_wah_load: NULL argument");
  FILE *f = fopen(path, "rb");
  if (!f) return fail(MB_ERR_IO, "mb_wah_load: cannot open %s", path);
  WahFileHdr h{};
  mb_status st = MB_OK;
  long size = -1;
  if (fread(&h, sizeof(h), 1, f) != 1) st = fail(MB_ERR_IO, "mb_wah_load: %s: short header", path);
  else if (h.magic != WAH_MAGIC) st = fail(MB_ERR_IO, "mb_wah_load: %s: bad magic 0x%08x", path, h.magic);
  else if (fseek(f, 0, SEEK_END) != 0 || (size = ftell(f)) < 0 || h.cmprs > ((uint64_t)size) / 4 ||
           (uint64_t)size != sizeof(h) + 4 * h.cmprs)
    st = fail(MB_ERR_IO, "mb_wah_load: %s: %ld bytes for %llu words", path, size, (unsigned long long)h.cmprs);
  if (st == MB_OK) {
    *nwords = h.cmprs;
    if (ngroups) *ngroups = h.decmprs;
    if (words) {
      if (capacity < h.cmprs)
        st = fail(MB_ERR_INVALID, "mb_wah_load: %llu words, the buffer holds %llu", (unsigned long long)h.cmprs,
                  (unsigned long long)capacity);
      else if (fseek(f, sizeof(h), SEEK_SET) != 0 ||
               (h.cmprs && fread(words, 4, h.cmprs, f) != h.cmprs))
        st = fail(MB_ERR_IO, "mb_wah_load: %s: short read", path);
    }
  }
  fclose(f);
  return st;
}
