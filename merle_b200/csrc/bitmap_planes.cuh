// bitmap_planes.cuh - bitmaps of sorted, disjoint bins by bit planes: the kernel
// and its launch (bitmap.cu cuts the bins into classes and picks the form).
#pragma once
#include <algorithm>
#include <type_traits>
#include "common.cuh"

namespace mb {

// Bitmaps of sorted, disjoint bins (one level, or the levels of a hierarchy
// together) from one pass over the column, without a shared-memory atomic or a
// ballot per row.
//
// The levels' boundaries cut the value domain into classes (at most 254), each
// inside one bin of every level or outside it, so that a bin is a run of
// consecutive classes.  A warp takes 4,096 rows at a time:
//   1. coalesced 16-byte loads; each value (or the dimension value behind it)
//      becomes a code, one byte that grows with its class, by a lookup table in
//      shared memory, or a division or binary search where the domain is wider
//      than the table; a 1-byte column of equality bins is its own code.  The
//      bytes go to the warp's tile in shared memory;
//   2. lane L reads the 128 codes of its four words 4L .. 4L+3 back (small tables: one word) and
//      transposes each 32 of them into 8 bit planes (an 8 x 8 bit transpose
//      over eight registers, four matrices at a time);
//   3. code by code, the word of a class is the AND of its planes or their
//      complements, built once per eight codes but for one AND a word, and
//      stored: 16 bytes a lane, 512 contiguous bytes a warp.  Where a level's bins
//      are the classes themselves (FINE) the word is that bin's; coarser levels
//      OR the words of a bin's classes together.  Row counts are taken per
//      class (three POPCs for four words with a carry-save add: the population
//      count runs at a quarter of the rate of the logic).
// Nothing is shared between warps but the row counts, so there is no block
// barrier in the loop.
//
// What bounds it: the bitmaps' stores and instruction issue for the columns read
// directly (120M rows, 2,525 -> 1,799 us for the ten levels of the star index
// against one shared atomic per row and level: date 463 -> 316 us for 1.6 GB,
// 79 % of the measured copy rate; discount and quantity 407 -> 228; supplier city
// 317 -> 125), and the random dimension reads for the columns behind a foreign
// key (650 -> 527 and 707 -> 594 us: about 0.9 sectors a clock and SM, of which
// the same reads alone take 454 and 520 us).  24M rows, 214 equality and range
// bins of three int32 columns: 623 -> 200 us against match_any per word.  85
// registers and 3 CTAs an SM: 2 CTAs 3 % slower, 4 (spills) 45 %.
constexpr int BP_THREADS = 256;
constexpr int BP_WARPS = BP_THREADS / 32;
// Rows of a warp tile at V words a lane: 4,096 (V = 4), or 1,024 (V = 1) for
// tables too small to give every warp a tile.
__host__ __device__ constexpr uint32_t bp_rows(int V) { return 1024u * V; }
// Rows below which a lane takes one word: a warp's latency for a tile (its class
// loop above all) counts while there are fewer 4,096-row tiles than warps.  V = 1 /
// V = 4, us: three bin sets of int32 columns, 1M rows 59 / 82, 6M 107 / 106, 24M
// 291 / 244; the star index, 1M 90 / 146, 10M 223 / 232, 24M 437 / 408.  The line lies
// between the two crossings, 6M for the one, past 10M for the other.
constexpr uint64_t BP_SMALL = 8000000;
constexpr uint32_t BP_LUT = 16384;        // values of the lookup table
constexpr uint32_t BP_MAXCLASS = 254;
constexpr int BP_MAXLEVELS = MB_MAXLEVELS;
constexpr uint32_t BP_NOCODE = 255;       // code of a value in no class
enum { BP_TABLE = 0, BP_SEARCH = 1, BP_DIRECT = 2 };

struct PlaneSpec {
  uint32_t ncls;                 // classes; class c has code code0 + c
  uint32_t code0;
  uint32_t dom_n;                // BP_TABLE: values [dom_lo, dom_lo + dom_n)
  uint32_t div_m, div_s1, div_s2;  // BP_SEARCH over equal bins of a column of at most 4 bytes: division magic
  uint32_t count;                // 1: some level wants its row counts
  uint32_t nlevels;
  uint64_t dom_lo;
  uint64_t width;                // BP_SEARCH: equal bins of this width from dom_lo (0: search the bounds)
  // Level 0 is the one whose bins are the classes, if there is one (FINE).
  uint32_t *out[BP_MAXLEVELS];
  unsigned long long *pop[BP_MAXLEVELS];
  // Per level, by code: bit c & 7 of byte c >> 3: the class lies in a bin of the
  // level; it is the last class of that bin.
  alignas(4) uint8_t in[BP_MAXLEVELS][32], end[BP_MAXLEVELS][32];
  uint64_t bound[2 * BP_MAXCLASS];  // class c = [bound[2c], bound[2c+1])
};

// Join output of the pass: the dimension value of every row (0 where the key
// leaves the dimension) written to dout, and the rows whose key leaves it
// counted in *bad; both optional.
struct LevelsJoinOut {
  void *dout;
  unsigned long long *bad;
};

// 8 x 8 bit transpose (by swaps of 4, 2 and 1: Warren, Hacker's Delight, 2nd edition,
// section 7-3) of the four byte columns of r: afterwards bit 8 i + j of
// r[b] is bit b of byte i of the former r[j].
template <int S>
__device__ __forceinline__ void bit_swap8(uint32_t (&r)[8]) {
  constexpr uint32_t m = S == 4 ? 0x0f0f0f0fu : S == 2 ? 0x33333333u : 0x55555555u;
#pragma unroll
  for (int j = 0; j < 8; ++j)
    if ((j & S) == 0) {
      const uint32_t a = r[j], b = r[j | S];
      r[j] = (a & m) | ((b & m) << S);
      r[j | S] = ((a >> S) & m) | (b & ~m);
    }
}
__device__ __forceinline__ void bit_transpose8(uint32_t (&r)[8]) {
  bit_swap8<4>(r);
  bit_swap8<2>(r);
  bit_swap8<1>(r);
}

// The classes of 32 consecutive rows (q: bytes in row order) as bit planes:
// bit i of p[b] is bit b of row i's class.
__device__ __forceinline__ void class_planes(const uint32_t (&q)[8], uint32_t (&p)[8]) {
  // byte i of p[j] = row 8 i + j: two 4 x 4 byte transposes
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t a = q[h], b = q[2 + h], c = q[4 + h], d = q[6 + h];
    const uint32_t ab0 = __byte_perm(a, b, 0x5140), ab1 = __byte_perm(a, b, 0x7362);
    const uint32_t cd0 = __byte_perm(c, d, 0x5140), cd1 = __byte_perm(c, d, 0x7362);
    p[4 * h + 0] = __byte_perm(ab0, cd0, 0x5410);
    p[4 * h + 1] = __byte_perm(ab0, cd0, 0x7632);
    p[4 * h + 2] = __byte_perm(ab1, cd1, 0x5410);
    p[4 * h + 3] = __byte_perm(ab1, cd1, 0x7632);
  }
  bit_transpose8(p);
}

template <int W>
struct ColVec;  // the values of one 16-byte load
template <>
struct ColVec<1> { static constexpr int N = 16; };
template <>
struct ColVec<2> { static constexpr int N = 8; };
template <>
struct ColVec<4> { static constexpr int N = 4; };
template <>
struct ColVec<8> { static constexpr int N = 2; };

template <int W>
__device__ __forceinline__ typename std::conditional<(W <= 4), uint32_t, uint64_t>::type vec_elem(const uint4 &x, int i) {
  if constexpr (W == 8) return i == 0 ? (uint64_t)x.x | (uint64_t)x.y << 32 : (uint64_t)x.z | (uint64_t)x.w << 32;
  else {
    const uint32_t w[4] = {x.x, x.y, x.z, x.w};
    if (W == 4) return w[i & 3];
    if (W == 2) return (w[(i >> 1) & 3] >> (16 * (i & 1))) & 0xffffu;
    return (w[(i >> 2) & 3] >> (8 * (i & 3))) & 0xffu;
  }
}

// The code of value v (BP_NOCODE: in no class).
template <int MODE, int VW, typename T>
__device__ __forceinline__ uint32_t code_of(const PlaneSpec &S, const uint8_t *lut, const uint64_t *bound, T v) {
  if (MODE == BP_DIRECT) return (uint32_t)v;
  if (MODE == BP_TABLE) {
    if (VW == 1) return lut[(uint32_t)v];  // the table covers every byte
    if (VW <= 4) {                         // a value below dom_lo wraps far above the table
      const uint32_t d = (uint32_t)v - (uint32_t)S.dom_lo;
      return lut[d < S.dom_n ? d : S.dom_n];
    }
    const uint64_t d = (uint64_t)v - S.dom_lo;
    return lut[d < S.dom_n ? (uint32_t)d : S.dom_n];
  }
  if (S.width) {
    if ((uint64_t)v < S.dom_lo) return BP_NOCODE;
    const uint64_t d = (uint64_t)v - S.dom_lo;
    const uint64_t b = VW <= 4 ? div_by_magic((uint32_t)d, S.div_m, S.div_s1, S.div_s2) : d / S.width;
    return b < S.ncls ? (uint32_t)b : BP_NOCODE;
  }
  uint32_t lo = 0, hi = S.ncls;  // first class whose end is above v
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (bound[2 * mid + 1] <= (uint64_t)v) lo = mid + 1;
    else hi = mid;
  }
  return lo < S.ncls && bound[2 * lo] <= (uint64_t)v ? lo : BP_NOCODE;
}

// Shared memory before the warps' code tiles: the classes' bounds and the
// lookup table after them, as the mode needs them.
__host__ __device__ inline uint32_t planes_bound(const PlaneSpec &S, int mode) {
  return mode == BP_DIRECT ? 0u : S.ncls * 16;
}
__host__ __device__ inline uint32_t planes_table(const PlaneSpec &S, int mode) {
  return planes_bound(S, mode) + (mode == BP_TABLE ? (S.dom_n + 1 + 15) & ~15u : 0u);
}

// The lookup table or the bounds into shared memory (block-collective; callers
// __syncthreads() afterwards).
template <int MODE>
__device__ __forceinline__ void planes_fill(const PlaneSpec &S, uint8_t *lut, uint64_t *bound) {
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (MODE == BP_DIRECT) return;
  for (uint32_t i = tid; i < 2 * S.ncls; i += BP_THREADS) bound[i] = S.bound[i];
  if (MODE == BP_TABLE) {
    for (uint32_t i = tid; i < (S.dom_n + 1 + 15) / 16 * 4; i += BP_THREADS)
      reinterpret_cast<uint32_t *>(lut)[i] = 0xffffffffu;  // BP_NOCODE
    __syncthreads();
    for (uint32_t c = warp; c < S.ncls; c += BP_WARPS) {
      const uint64_t lo = bound[2 * c] - S.dom_lo, hi = bound[2 * c + 1] - S.dom_lo;
      for (uint64_t i = lo + lane; i < hi && i < S.dom_n; i += 32) lut[i] = (uint8_t)c;
    }
  }
}

// The rows of every class (cnt by code) to its bin of each level, a class per
// thread.
__device__ __forceinline__ void planes_flush(const PlaneSpec &S, const uint32_t *cnt) {
  const uint32_t c = S.code0 + threadIdx.x;
  if (!S.count || threadIdx.x >= S.ncls || cnt[c] == 0) return;
  for (uint32_t l = 0; l < S.nlevels; ++l) {
    const uint32_t *in = reinterpret_cast<const uint32_t *>(S.in[l]), *end = reinterpret_cast<const uint32_t *>(S.end[l]);
    if (!S.pop[l] || !((in[c >> 5] >> (c & 31u)) & 1u)) continue;
    uint32_t b = __popc(end[c >> 5] & ((1u << (c & 31u)) - 1u));  // bins that end before the class
    for (uint32_t i = 0; i < c >> 5; ++i) b += __popc(end[i]);
    atomicAdd(&S.pop[l][b], (unsigned long long)cnt[c]);
  }
}

// Byte of row r's code in a warp's tile: lane L reads its 32 V rows back 16 at
// a time; the 16-byte chunks of a lane are XOR-swizzled by the lane so that those
// reads have no bank conflicts.
template <int V>
__device__ __forceinline__ uint32_t code_at(uint32_t r) {
  const uint32_t L = r / (32 * V), c = (r >> 4) & (2 * V - 1);
  return L * 32 * V + ((c ^ (V == 4 ? L & 7u : (L >> 2) & 1u)) << 4) + (r & 15u);
}

// Step 1 for one tile of a warp: the codes of rows [row0, row0 + 1024 V) (those
// past n: none) into the warp's tile.  Load j of lane l holds rows (32 j + l) N
// on.
template <int W, bool JOIN, int DW, int MODE, int V, bool FULL>
__device__ __forceinline__ void planes_codes(const PlaneSpec &S, const void *col, const void *dim, uint64_t dimsz,
                                             uint64_t n, uint64_t row0, const uint8_t *lut, const uint64_t *bound,
                                             uint8_t *tile, const LevelsJoinOut &jo, uint32_t &nbad) {
  using VT = typename std::conditional<((JOIN ? DW : W) <= 4), uint32_t, uint64_t>::type;
  constexpr int VW = JOIN ? DW : W;
  constexpr int N = ColVec<W>::N;                 // rows of a 16-byte load
  constexpr int LOADS = (int)bp_rows(V) / (32 * N);  // loads of a tile
  constexpr int MOST = W == 1 || JOIN ? 4 : 8, BATCH = LOADS < MOST ? LOADS : MOST;
  const uint32_t lane = threadIdx.x & 31;
#pragma unroll 1
  for (int j0 = 0; j0 < LOADS; j0 += BATCH) {
    uint4 x[BATCH];
#pragma unroll
    for (int j = 0; j < BATCH; ++j) {
      const uint64_t r = row0 + (uint64_t)(32 * (j0 + j) + lane) * N;
      if (FULL) {
        x[j] = __ldcs(reinterpret_cast<const uint4 *>(reinterpret_cast<const uint8_t *>(col) + r * W));
      } else {
        uint32_t w[4] = {0, 0, 0, 0};
#pragma unroll
        for (int i = 0; i < N; ++i)
          if (r + i < n) {
            const uint64_t e = load_width(col, r + i, W);
            if (W == 8) w[(2 * i) & 3] = (uint32_t)e, w[(2 * i + 1) & 3] = (uint32_t)(e >> 32);
            else w[(i * W / 4) & 3] |= (uint32_t)e << (8 * ((i * W) & 3));
          }
        x[j] = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
    VT v[JOIN ? BATCH : 1][N];
    uint32_t bad[JOIN ? BATCH : 1];
    if constexpr (JOIN) {  // the dimension reads of the whole batch in flight together
#pragma unroll
      for (int j = 0; j < BATCH; ++j) {
        bad[j] = 0;
#pragma unroll
        for (int i = 0; i < N; ++i) {
          const uint32_t key = (uint32_t)vec_elem<W>(x[j], i);
          const bool here = FULL || row0 + (uint64_t)(32 * (j0 + j) + lane) * N + i < n;
          const bool ok = here && (dimsz == 0 || key < dimsz);
          if (!ok) bad[j] |= 1u << i;
          nbad += here && !ok ? 1u : 0u;
          v[j][i] = ok ? (VT)load_width(dim, key, DW) : (VT)0;
        }
      }
    }
#pragma unroll
    for (int j = 0; j < BATCH; ++j) {
      const uint32_t r = (32u * (j0 + j) + lane) * N;  // row in the tile
      if constexpr (JOIN) {
        if (jo.dout) {
          if (FULL && DW == 1) {
            reinterpret_cast<uint32_t *>(jo.dout)[(row0 + r) / 4] =
                (uint32_t)v[j][0] | (uint32_t)v[j][1] << 8 | (uint32_t)v[j][2] << 16 | (uint32_t)v[j][3] << 24;
          } else if (FULL && DW == 2) {
            reinterpret_cast<uint2 *>(jo.dout)[(row0 + r) / 4] =
                make_uint2((uint32_t)v[j][0] | (uint32_t)v[j][1] << 16, (uint32_t)v[j][2] | (uint32_t)v[j][3] << 16);
          } else {
#pragma unroll
            for (int i = 0; i < N; ++i)
              if (FULL || row0 + r + i < n) {
                if (DW == 1) reinterpret_cast<uint8_t *>(jo.dout)[row0 + r + i] = (uint8_t)v[j][i];
                else if (DW == 2) reinterpret_cast<uint16_t *>(jo.dout)[row0 + r + i] = (uint16_t)v[j][i];
                else if (DW == 4) reinterpret_cast<uint32_t *>(jo.dout)[row0 + r + i] = (uint32_t)v[j][i];
                else reinterpret_cast<unsigned long long *>(jo.dout)[row0 + r + i] = (unsigned long long)v[j][i];
              }
          }
        }
      }
      uint8_t *dst = tile + code_at<V>(r);
      uint32_t c[N];
#pragma unroll
      for (int i = 0; i < N; ++i) {
        if constexpr (JOIN) {
          c[i] = code_of<MODE, VW>(S, lut, bound, v[j][i]);
          if ((bad[j] >> i) & 1u) c[i] = BP_NOCODE;
        } else {
          c[i] = code_of<MODE, VW>(S, lut, bound, (VT)vec_elem<W>(x[j], i));
          if (!FULL && row0 + r + i >= n) c[i] = BP_NOCODE;
        }
      }
      if constexpr (MODE == BP_DIRECT && FULL) {
        *reinterpret_cast<uint4 *>(dst) = x[j];
      } else if constexpr (N == 2) {
        *reinterpret_cast<uint16_t *>(dst) = (uint16_t)(c[0] | c[1] << 8);
      } else {
        uint32_t w[N / 4];
#pragma unroll
        for (int i = 0; i < N / 4; ++i)
          w[i] = __byte_perm(__byte_perm(c[4 * i], c[4 * i + 1], 0x0040),
                             __byte_perm(c[4 * i + 2], c[4 * i + 3], 0x0040), 0x5410);
        if constexpr (N == 4) *reinterpret_cast<uint32_t *>(dst) = w[0];
        else if constexpr (N == 8) *reinterpret_cast<uint2 *>(dst) = make_uint2(w[0], w[1]);
        else *reinterpret_cast<uint4 *>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
  }
}

// W: bytes of the column read by row (4 for a join: the foreign key); DW: bytes
// of the dimension element (join only).  FINE: level 0's bins are the classes;
// NC: the other levels (all of them without FINE).
template <int W, bool JOIN, int DW, int MODE, int V, bool FINE, int NC>
__global__ void __launch_bounds__(BP_THREADS, 3)
bitmap_planes_kernel(const __grid_constant__ PlaneSpec S, const void *__restrict__ col, const void *__restrict__ dim,
                     uint64_t dimsz, uint64_t n, uint64_t stride, LevelsJoinOut jo) {
  extern __shared__ __align__(128) uint8_t smem[];
  constexpr int L0 = FINE ? 1 : 0;  // first of the levels with accumulated bins
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint64_t *bound = reinterpret_cast<uint64_t *>(smem);
  uint8_t *lut = smem + planes_bound(S, MODE);
  // Rows by code, of this CTA: a column of more than 2^32 rows a CTA (148 of them at
  // least) would not fit the memory.
  uint32_t *cnt = reinterpret_cast<uint32_t *>(smem + planes_table(S, MODE));
  constexpr uint32_t ROWS = bp_rows(V);
  uint8_t *tile = smem + planes_table(S, MODE) + 1024 + warp * ROWS;
  for (uint32_t i = tid; i < 256; i += BP_THREADS) cnt[i] = 0;
  planes_fill<MODE>(S, lut, bound);
  __syncthreads();

  const uint64_t nwords = (n + 31) / 32, ntiles = (n + ROWS - 1) / ROWS;
  // the codes of this CTA: all, or its share where a small table's are split (planes_split)
  uint32_t cbeg = S.code0 & ~7u, cend = S.code0 + S.ncls;
  if constexpr (V == 1 && NC == 0) {
    const uint32_t per = ((cend - cbeg + 7) / 8 + gridDim.y - 1) / gridDim.y * 8;
    cbeg += blockIdx.y * per;
    cend = cbeg + per < cend ? cbeg + per : cend;
  }
  uint32_t nbad = 0;
  for (uint64_t t = (uint64_t)blockIdx.x * BP_WARPS + warp; t < ntiles; t += (uint64_t)gridDim.x * BP_WARPS) {
    const uint64_t row0 = t * ROWS;
    const bool full = row0 + ROWS <= n;
    if (full) planes_codes<W, JOIN, DW, MODE, V, true>(S, col, dim, dimsz, n, row0, lut, bound, tile, jo, nbad);
    else planes_codes<W, JOIN, DW, MODE, V, false>(S, col, dim, dimsz, n, row0, lut, bound, tile, jo, nbad);
    __syncwarp();
    // 2. bit planes of the lane's words; the low two planes as their four products
    uint32_t P[6][V], ab[4][V];
#pragma unroll
    for (int k = 0; k < V; ++k) {
      uint32_t q[8], p[8];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint4 y = *reinterpret_cast<const uint4 *>(tile + code_at<V>(lane * 32 * V + 32 * k + 16 * h));
        q[4 * h] = y.x, q[4 * h + 1] = y.y, q[4 * h + 2] = y.z, q[4 * h + 3] = y.w;
      }
      class_planes(q, p);
#pragma unroll
      for (int b = 0; b < 6; ++b) P[b][k] = p[b + 2];
      ab[0][k] = ~p[0] & ~p[1], ab[1][k] = p[0] & ~p[1], ab[2][k] = ~p[0] & p[1], ab[3][k] = p[0] & p[1];
    }
    __syncwarp();  // the tile is rewritten by the next round
    // 3. code by code
    const uint64_t w = t * (ROWS / 32) + lane * V;
    const bool whole = full || w + V <= nwords;
    auto store = [&](uint32_t *d, const uint32_t (&m)[V]) {
      if (V == 4 && whole) {
        *reinterpret_cast<uint4 *>(d) = make_uint4(m[0], m[1 % V], m[2 % V], m[3 % V]);
      } else {
#pragma unroll
        for (int k = 0; k < V; ++k)
          if (whole || w + k < nwords) d[k] = m[k];
      }
    };
    uint32_t *fine = FINE ? S.out[0] + w + (cbeg > S.code0 ? cbeg - S.code0 : 0) * stride : nullptr;
    uint32_t acc[NC ? NC : 1][V];
    uint32_t *dst[NC ? NC : 1];
#pragma unroll
    for (int l = 0; l < NC; ++l) {
      dst[l] = S.out[L0 + l] + w;
#pragma unroll
      for (int k = 0; k < V; ++k) acc[l][k] = 0;
    }
#pragma unroll 1
    for (uint32_t c0 = cbeg; c0 < cend; c0 += 8) {
      uint32_t high[2][V];  // the products of planes 3 .. 7, with plane 2 clear and set
#pragma unroll
      for (int k = 0; k < V; ++k) high[1][k] = 0xffffffffu;
#pragma unroll
      for (int b = 3; b < 8; ++b) {
        const uint32_t m = (c0 >> b) & 1u ? 0u : 0xffffffffu;
#pragma unroll
        for (int k = 0; k < V; ++k) high[1][k] &= P[b - 2][k] ^ m;
      }
#pragma unroll
      for (int k = 0; k < V; ++k) high[0][k] = high[1][k] & ~P[0][k], high[1][k] &= P[0][k];
      uint32_t in[NC ? NC : 1], end[NC ? NC : 1];
#pragma unroll
      for (int l = 0; l < NC; ++l) in[l] = S.in[L0 + l][c0 >> 3], end[l] = S.end[L0 + l][c0 >> 3];
      uint32_t rows = 0;  // lane i (< 8): the rows of code c0 + i
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (c0 + i - S.code0 >= S.ncls) continue;
        uint32_t m[V];
#pragma unroll
        for (int k = 0; k < V; ++k) m[k] = high[i >> 2][k] & ab[i & 3][k];
        if (FINE) {
          store(fine, m);
          fine += stride;
        }
        if (S.count) {
          uint32_t r = __popc(m[V - 1]);
          if constexpr (V == 4) {
            const uint32_t s1 = m[0] ^ m[1] ^ m[2], c1 = (m[0] & m[1]) | (m[2] & (m[0] | m[1]));
            r += __popc(s1) + 2 * __popc(c1);
          }
          r = __reduce_add_sync(0xffffffffu, r);
          if (lane == (uint32_t)i) rows = r;
        }
#pragma unroll
        for (int l = 0; l < NC; ++l) {
          if (!((in[l] >> i) & 1u)) continue;
#pragma unroll
          for (int k = 0; k < V; ++k) acc[l][k] |= m[k];
          if (!((end[l] >> i) & 1u)) continue;
          store(dst[l], acc[l]);
          dst[l] += stride;
#pragma unroll
          for (int k = 0; k < V; ++k) acc[l][k] = 0;
        }
      }
      if (rows) atomicAdd(&cnt[c0 + lane], rows);
    }
  }
  if (JOIN && jo.bad) {
    nbad = __reduce_add_sync(0xffffffffu, nbad);
    if (lane == 0 && nbad) atomicAdd(jo.bad, (unsigned long long)nbad);
  }
  __syncthreads();
  planes_flush(S, cnt);
}

// A pass: the classes, the column (or key and dimension), and where the stream
// and the join's outputs are.
struct PlanePass {
  const PlaneSpec &S;
  const mb_src *src;
  uint64_t n, stride;
  cudaStream_t st;
  LevelsJoinOut jo;
};

// Shares of a level's codes on a small table, a row of CTAs each, while there are warps without a
// tile: a warp takes about 0.7 us for 8 codes, and 32 of those one after the other are most
// of the time of the table (250 bins with their row counts, 300K rows: 31 -> 19 us, as with one
// shared atomic a row and level).  Join outputs are written by one pass alone.
inline uint32_t planes_split(const PlanePass &P, uint64_t warps) {
  if (P.jo.dout || P.jo.bad) return 1;
  const uint64_t tiles = ceil_div(P.n, bp_rows(1)), groups = ((P.S.code0 & 7u) + P.S.ncls + 7) / 8;
  return (uint32_t)std::max<uint64_t>(1, std::min(warps / tiles, groups));
}

template <int W, bool JOIN, int DW, int MODE, int V, bool FINE, int NC>
mb_status launch_planes_v(const PlanePass &P) {
  auto kern = bitmap_planes_kernel<W, JOIN, DW, MODE, V, FINE, NC>;
  const size_t smem = planes_table(P.S, MODE) + 1024 + (size_t)BP_WARPS * bp_rows(V);
  MB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int occ = 0;
  MB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, BP_THREADS, smem));
  if (occ < 1) return fail(MB_ERR_INVALID, "bitmap planes: %zu bytes of shared memory", smem);
  const DevInfo &di = dev_info();
  uint64_t grid = (uint64_t)di.sms * occ;
  const uint64_t need = ceil_div(ceil_div(P.n, bp_rows(V)), BP_WARPS);
  if (grid > need) grid = need;
  const uint64_t split = V == 1 && NC == 0 ? planes_split(P, (uint64_t)di.sms * occ * BP_WARPS) : 1;
  kern<<<dim3((unsigned)grid, (unsigned)split), BP_THREADS, smem, P.st>>>(P.S, JOIN ? (const void *)P.src->fk : P.src->col,
                                                   JOIN ? P.src->col : nullptr, P.src->dimsz, P.n, P.stride, P.jo);
  MB_LAUNCH_CHECK("bitmap_planes_kernel");
  return MB_OK;
}

template <int W, bool JOIN, int DW, int MODE, bool FINE, int NC>
mb_status launch_planes_k(const PlanePass &P) {
  return P.n < BP_SMALL ? launch_planes_v<W, JOIN, DW, MODE, 1, FINE, NC>(P)
                        : launch_planes_v<W, JOIN, DW, MODE, 4, FINE, NC>(P);
}

// One level over its own classes, or two of a hierarchy, by table.
template <int W, bool JOIN, int DW>
mb_status launch_planes_fine(const PlanePass &P) {
  return P.S.nlevels == 1 ? launch_planes_k<W, JOIN, DW, BP_TABLE, true, 0>(P)
                          : launch_planes_k<W, JOIN, DW, BP_TABLE, true, 1>(P);
}

// Any levels, by table or search.
template <int W, bool JOIN, int DW>
mb_status launch_planes_any(int mode, const PlanePass &P) {
  return mode == BP_SEARCH ? launch_planes_k<W, JOIN, DW, BP_SEARCH, false, BP_MAXLEVELS>(P)
                           : launch_planes_k<W, JOIN, DW, BP_TABLE, false, BP_MAXLEVELS>(P);
}

// The forms, a file each (bitmap_planes_*.cu).  A file's kernels load together when
// the first of them runs, about 1 ms a MB of device code and line tables.  With all
// of them in one file of 24 MB the first pass of a process took 22.6 ms (300K rows;
// 3.6 with the 6 MB of the shared-atomic kernels before), with planes_row and
// planes_join alone, 4 MB, which are all that the star index needs, 1.3.
mb_status planes_row(int mode, const PlanePass &P);       // direct and fine, columns of 1, 2 and 4 bytes
mb_status planes_join(const PlanePass &P);                // fine, dimensions of 1 and 2 bytes
mb_status planes_wide(const PlanePass &P);                // fine, 8-byte columns, dimensions of 4 and 8 bytes
mb_status planes_search(const PlanePass &P);              // one level over its own classes, by search
mb_status planes_any_row(int mode, const PlanePass &P);   // any levels, columns
mb_status planes_any_join(int mode, const PlanePass &P);  // any levels, dimensions

}  // namespace mb
