// bitmap.cu - one-pass multi-bin bitmap-index creation (mb_bitmap_create).
//
// Reference: create_bin (bmpidx_create.cu:14-56) launching the multi-bin
// bmpcreate kernel (primitive.cuh:102-118): one thread per row, one
// __ballot_sync per (row-word, bin), lane 0 storing each word to HBM.
//
// Sorted, disjoint bins (an index level, a hierarchy of levels, one range) run
// in bitmap_planes_kernel: classes by table lookup, bit planes by transposition
// in registers, bitmaps as products of planes (see there).  Overlapping,
// unsorted or empty bins run in bitmap_create_kernel, one ballot per bin and word
// as in the reference:
//  - Persistent CTAs (SMs x occupancy) walk 4096-row tiles.  A 3-stage ring of
//    column tiles is filled by 1-D TMA bulk copies (cp.async.bulk) with mbarrier
//    completion, so HBM reads stream ahead of the compute.  For join bitmaps the
//    staged column is the foreign key and the dimension value is gathered from
//    the (L2-resident) dimension array.
//  - Words are assembled in a shared-memory tile [bin][128 words] and written
//    out with coalesced 128-bit stores, instead of one 4-byte store per word.
// In both the tail is exact: bits of rows >= n are zero (the reference's
// single-predicate kernel writes past the bitmap end, primitive.cuh:94-99,
// and its multi-bin kernel breaks out of a full-mask ballot,
// primitive.cuh:110-113; neither happens here).
#include <stddef.h>
#include <string.h>
#include <algorithm>
#include <type_traits>
#include "common.cuh"
#include "tma.cuh"

namespace mb {

constexpr int BC_THREADS = 256;
constexpr int BC_TILE_ROWS = 4096;
constexpr int BC_TILE_WORDS = BC_TILE_ROWS / 32;  // 128
constexpr int BC_STAGES = 3;
constexpr int BC_MAXBINS = 256;

struct BinSpec {
  uint32_t nbins;
  uint32_t pad_;
  uint64_t lo[BC_MAXBINS], hi[BC_MAXBINS];
};

template <int W>
__device__ __forceinline__ uint64_t ld_smem_w(const uint8_t *p, uint32_t i) {
  if (W == 1) return p[i];
  if (W == 2) return reinterpret_cast<const uint16_t *>(p)[i];
  if (W == 4) return reinterpret_cast<const uint32_t *>(p)[i];
  return reinterpret_cast<const unsigned long long *>(p)[i];
}

// Word wi of bin b in the shared tile: groups of 4 words are XOR-swizzled by
// the bin so that leaders of different bins storing the same word index hit
// different banks, while each bin's 4-word groups stay contiguous.
__device__ __forceinline__ uint32_t tile_word(uint32_t b, uint32_t wi) {
  return b * BC_TILE_WORDS + ((((wi >> 2) ^ b) & 31u) << 2) + (wi & 3u);
}

// W: bytes of the staged column element (4 for join: the foreign key);
// DW: bytes of the dimension element (join only).
template <int W, bool JOIN, int DW>
__global__ void __launch_bounds__(BC_THREADS)
bitmap_create_kernel(const __grid_constant__ BinSpec S, const void *__restrict__ col,
                     const void *__restrict__ dim, uint64_t dimsz, uint64_t n,
                     uint32_t *__restrict__ out, uint64_t stride,
                     unsigned long long *__restrict__ pop, uint32_t *errw) {
  extern __shared__ __align__(128) uint8_t smem[];
  constexpr uint32_t STAGE_BYTES = BC_TILE_ROWS * W;
  uint8_t *stage = smem;
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + BC_STAGES * STAGE_BYTES);
  uint32_t *obuf = reinterpret_cast<uint32_t *>(smem + BC_STAGES * STAGE_BYTES + 128);
  unsigned long long *cnt = reinterpret_cast<unsigned long long *>(obuf + S.nbins * BC_TILE_WORDS);
  uint64_t *slo = reinterpret_cast<uint64_t *>(cnt + S.nbins);
  uint64_t *shi = slo + S.nbins;

  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint64_t nwords = (n + 31) / 32;
  const uint64_t ntiles = (n + BC_TILE_ROWS - 1) / BC_TILE_ROWS;
  const uint8_t *colb = reinterpret_cast<const uint8_t *>(col);

  for (uint32_t b = tid; b < S.nbins; b += BC_THREADS) {
    cnt[b] = 0;
    slo[b] = S.lo[b];
    shi[b] = S.hi[b];
  }
  if (tid == 0) {
    for (int s = 0; s < BC_STAGES; ++s) mbar_init(&bars[s], 1);
    fence_mbar_init();
  }
  __syncthreads();

  // Bytes of tile t that the bulk copy moves: whole 16-byte chunks only.
  auto tile_bulk_bytes = [&](uint64_t t) -> uint32_t {
    uint64_t rows = n - t * BC_TILE_ROWS;
    if (rows > BC_TILE_ROWS) rows = BC_TILE_ROWS;
    return (uint32_t)((rows * W) & ~(uint64_t)15);
  };
  auto issue = [&](uint64_t t, int s) {
    uint32_t bytes = tile_bulk_bytes(t);
    fence_proxy_async_smem();
    mbar_arrive_expect_tx(&bars[s], bytes);
    if (bytes) bulk_g2s(stage + s * STAGE_BYTES, colb + t * (uint64_t)STAGE_BYTES, bytes, &bars[s]);
  };

  if (tid == 0) {
    uint64_t t = blockIdx.x;
    for (int s = 0; s < BC_STAGES && t < ntiles; ++s, t += gridDim.x) issue(t, s);
  }

  uint32_t it = 0;
  for (uint64_t t = blockIdx.x; t < ntiles; t += gridDim.x, ++it) {
    const int s = it % BC_STAGES;
    const uint32_t parity = (it / BC_STAGES) & 1u;
    // Every thread waits (bounded) for the stage; the block leaves together if
    // any wait ran out, after one more bounded wait for the copy in flight.
    const bool arrived = mbar_wait_bounded(&bars[s], parity, errw, MB_DEVERR_TMA_WAIT);
    if (!__syncthreads_and(arrived)) {
      if (tid == 0) mbar_wait_bounded(&bars[s], parity, nullptr, 0, 1u << 16);
      return;
    }
    const uint8_t *sp = stage + s * STAGE_BYTES;
    const uint32_t bulk_rows = tile_bulk_bytes(t) / W;
    const uint64_t row0 = t * BC_TILE_ROWS;

    for (uint32_t wi = warp; wi < BC_TILE_WORDS; wi += BC_THREADS / 32) {
      const uint32_t r = wi * 32 + lane;
      const uint64_t row = row0 + r;
      bool valid = row < n;
      uint64_t v = 0;
      if (valid) {
        uint64_t x = r < bulk_rows ? ld_smem_w<W>(sp, r) : load_width(col, row, W);
        if (JOIN) {
          if (dimsz != 0 && x >= dimsz) valid = false;
          else v = load_width(dim, x, DW);
        } else {
          v = x;
        }
      }
      for (uint32_t b = 0; b < S.nbins; ++b) {
        uint32_t m = __ballot_sync(0xffffffffu, valid && v >= slo[b] && v < shi[b]);
        if (lane == (b & 31)) obuf[tile_word(b, wi)] = m;
      }
    }
    __syncthreads();  // stage s fully read, obuf complete

    if (tid == 0 && t + (uint64_t)BC_STAGES * gridDim.x < ntiles)
      issue(t + (uint64_t)BC_STAGES * gridDim.x, s);

    // Coalesced write-out: per bin 128 consecutive words = 32 x uint4.  A
    // warp covers exactly one bin per iteration (i / 32 is warp-uniform).
    const uint64_t w0 = t * BC_TILE_WORDS;
    for (uint32_t i = tid; i < S.nbins * (BC_TILE_WORDS / 4); i += BC_THREADS) {
      const uint32_t b = i / (BC_TILE_WORDS / 4), q = i % (BC_TILE_WORDS / 4);
      const uint64_t w = w0 + q * 4;
      uint32_t c = 0;
      if (w < nwords) {  // obuf beyond the last word is never written
        const uint4 v4 = *reinterpret_cast<const uint4 *>(&obuf[tile_word(b, q * 4)]);
        uint32_t *dst = out + b * stride + w;
        if (w + 4 <= nwords) {
          *reinterpret_cast<uint4 *>(dst) = v4;
        } else {
          dst[0] = v4.x;
          if (w + 1 < nwords) dst[1] = v4.y;
          if (w + 2 < nwords) dst[2] = v4.z;
        }
        c = __popc(v4.x) + __popc(v4.y) + __popc(v4.z) + __popc(v4.w);
      }
      if (pop) {
        c = __reduce_add_sync(0xffffffffu, c);
        if (lane == 0 && c) atomicAdd(&cnt[b], (unsigned long long)c);
      }
    }
    __syncthreads();  // obuf reused by the next tile
  }
  if (pop) {
    __syncthreads();
    for (uint32_t b = tid; b < S.nbins; b += BC_THREADS)
      if (cnt[b]) atomicAdd(&pop[b], cnt[b]);
  }
}

// ---------------------------------------------------------------- planes
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
// 291 / 244; the star index, 1M 90 / 146, 10M 223 / 232, 24M 437 / 408.
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

// 8 x 8 bit transpose of the four byte columns of r: afterwards bit 8 i + j of
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
  uint32_t *cnt = reinterpret_cast<uint32_t *>(smem + planes_table(S, MODE));  // by code
  constexpr uint32_t ROWS = bp_rows(V);
  uint8_t *tile = smem + planes_table(S, MODE) + 1024 + warp * ROWS;
  for (uint32_t i = tid; i < 256; i += BP_THREADS) cnt[i] = 0;
  planes_fill<MODE>(S, lut, bound);
  __syncthreads();

  const uint64_t nwords = (n + 31) / 32, ntiles = (n + ROWS - 1) / ROWS;
  const uint32_t cend = S.code0 + S.ncls;
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
    uint32_t *fine = FINE ? S.out[0] + w : nullptr;
    uint32_t acc[NC ? NC : 1][V];
    uint32_t *dst[NC ? NC : 1];
#pragma unroll
    for (int l = 0; l < NC; ++l) {
      dst[l] = S.out[L0 + l] + w;
#pragma unroll
      for (int k = 0; k < V; ++k) acc[l][k] = 0;
    }
#pragma unroll 1
    for (uint32_t c0 = S.code0 & ~7u; c0 < cend; c0 += 8) {
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

// ---------------------------------------------------------------- host
template <int W, bool JOIN, int DW>
static mb_status launch_bc(const BinSpec &S, const mb_src *src, uint64_t n, uint32_t *out,
                           uint64_t stride, uint64_t *pop, cudaStream_t st) {
  auto kern = bitmap_create_kernel<W, JOIN, DW>;
  size_t smem = (size_t)BC_STAGES * BC_TILE_ROWS * W + 128 +
                (size_t)S.nbins * BC_TILE_WORDS * 4 + (size_t)S.nbins * 24;
  MB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int occ = 0;
  MB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, BC_THREADS, smem));
  if (occ < 1) return fail(MB_ERR_INVALID, "bitmap_create: %u bins do not fit in shared memory", S.nbins);
  uint64_t ntiles = ceil_div(n, BC_TILE_ROWS);
  uint64_t grid = (uint64_t)dev_info().sms * occ;
  if (grid > ntiles) grid = ntiles;
  uint32_t *errw = device_error_word();
  if (!errw) return fail(MB_ERR_OOM, "bitmap_create: device error word");
  const void *colp = JOIN ? (const void *)src->fk : src->col;
  const void *dimp = JOIN ? src->col : nullptr;
  kern<<<(unsigned)grid, BC_THREADS, smem, st>>>(S, colp, dimp, src->dimsz, n, out, stride,
                                                 reinterpret_cast<unsigned long long *>(pop), errw);
  MB_LAUNCH_CHECK("bitmap_create_kernel");
  return MB_OK;
}

// ---------------------------------------------------------------- planes host
template <int W, bool JOIN, int DW, int MODE, int V, bool FINE, int NC>
static mb_status launch_planes_v(const PlaneSpec &S, const mb_src *src, uint64_t n, uint64_t stride, cudaStream_t st,
                                 LevelsJoinOut jo) {
  auto kern = bitmap_planes_kernel<W, JOIN, DW, MODE, V, FINE, NC>;
  const size_t smem = planes_table(S, MODE) + 1024 + (size_t)BP_WARPS * bp_rows(V);
  MB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int occ = 0;
  MB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, BP_THREADS, smem));
  if (occ < 1) return fail(MB_ERR_INVALID, "bitmap planes: %zu bytes of shared memory", smem);
  uint64_t grid = (uint64_t)dev_info().sms * occ;
  const uint64_t need = ceil_div(ceil_div(n, bp_rows(V)), BP_WARPS);
  if (grid > need) grid = need;
  kern<<<(unsigned)grid, BP_THREADS, smem, st>>>(S, JOIN ? (const void *)src->fk : src->col,
                                                 JOIN ? src->col : nullptr, src->dimsz, n, stride, jo);
  MB_LAUNCH_CHECK("bitmap_planes_kernel");
  return MB_OK;
}

template <int W, bool JOIN, int DW, int MODE, bool FINE, int NC>
static mb_status launch_planes_k(const PlaneSpec &S, const mb_src *src, uint64_t n, uint64_t stride, cudaStream_t st,
                                 LevelsJoinOut jo) {
  return n < BP_SMALL ? launch_planes_v<W, JOIN, DW, MODE, 1, FINE, NC>(S, src, n, stride, st, jo)
                      : launch_planes_v<W, JOIN, DW, MODE, 4, FINE, NC>(S, src, n, stride, st, jo);
}

// One level, or a hierarchy of two, over its own classes has its form; any
// other set of levels, and the wide domains, the general one.
template <int W, bool JOIN, int DW>
static mb_status launch_planes_w(int mode, bool fine, const PlaneSpec &S, const mb_src *src, uint64_t n,
                                 uint64_t stride, cudaStream_t st, LevelsJoinOut jo) {
  if constexpr (W == 1 && !JOIN) {
    if (mode == BP_DIRECT) return launch_planes_k<W, JOIN, DW, BP_DIRECT, true, 0>(S, src, n, stride, st, jo);
  }
  if (mode == BP_SEARCH)
    return fine && S.nlevels == 1
               ? launch_planes_k<W, JOIN, DW, BP_SEARCH, true, 0>(S, src, n, stride, st, jo)
               : launch_planes_k<W, JOIN, DW, BP_SEARCH, false, BP_MAXLEVELS>(S, src, n, stride, st, jo);
  if (fine && S.nlevels == 1) return launch_planes_k<W, JOIN, DW, BP_TABLE, true, 0>(S, src, n, stride, st, jo);
  if (fine && S.nlevels == 2) return launch_planes_k<W, JOIN, DW, BP_TABLE, true, 1>(S, src, n, stride, st, jo);
  return launch_planes_k<W, JOIN, DW, BP_TABLE, false, BP_MAXLEVELS>(S, src, n, stride, st, jo);
}

static mb_status launch_planes(int mode, bool fine, const PlaneSpec &S, const mb_src *src, uint64_t n,
                               uint64_t stride, cudaStream_t st, LevelsJoinOut jo) {
  if (src->fk == nullptr) {
    switch (src->width) {
    case 1: return launch_planes_w<1, false, 1>(mode, fine, S, src, n, stride, st, jo);
    case 2: return launch_planes_w<2, false, 1>(mode, fine, S, src, n, stride, st, jo);
    case 4: return launch_planes_w<4, false, 1>(mode, fine, S, src, n, stride, st, jo);
    default: return launch_planes_w<8, false, 1>(mode, fine, S, src, n, stride, st, jo);
    }
  }
  switch (src->width) {  // the column read by row is the 4-byte key; width is the dimension's
  case 1: return launch_planes_w<4, true, 1>(mode, fine, S, src, n, stride, st, jo);
  case 2: return launch_planes_w<4, true, 2>(mode, fine, S, src, n, stride, st, jo);
  case 4: return launch_planes_w<4, true, 4>(mode, fine, S, src, n, stride, st, jo);
  default: return launch_planes_w<4, true, 8>(mode, fine, S, src, n, stride, st, jo);
  }
}

// The levels as classes, if the planes kernel takes them: every level sorted
// and disjoint without an empty bin, at most BP_MAXCLASS classes together.
// *fine: a level's bins are the classes (made level 0).
static bool planes_spec(const mb_src *src, const mb_level *lv, uint32_t nl, PlaneSpec &S, int *mode, bool *fine) {
  if (nl == 0 || nl > (uint32_t)BP_MAXLEVELS) return false;
  const uint32_t vbytes = src->width;
  memset(&S, 0, offsetof(PlaneSpec, bound));
  S.nlevels = nl;
  for (uint32_t l = 0; l < nl; ++l) {
    const mb_level &L = lv[l];
    if (L.nbins == 0 || L.nbins > BP_MAXCLASS || !L.lo || !L.hi || !L.out) return false;
    for (uint32_t j = 0; j < L.nbins; ++j) {
      if (L.hi[j] <= L.lo[j]) return false;
      if (j + 1 < L.nbins && L.lo[j + 1] < L.hi[j]) return false;
    }
  }
  // classes: the intervals between neighbouring boundaries that lie in some
  // bin, by a sweep over the levels' ascending boundaries; at[l]: the bin of
  // level l still open or to come
  uint8_t in[BP_MAXCLASS], end[BP_MAXCLASS];  // bit l
  uint32_t at[BP_MAXLEVELS] = {0, 0, 0, 0};
  uint64_t x = ~0ull;
  for (uint32_t l = 0; l < nl; ++l) x = std::min<uint64_t>(x, lv[l].lo[0]);
  const uint64_t front = x;
  while (true) {
    // the next boundary above x, and the levels with a bin open at x
    uint64_t y = ~0ull;
    uint8_t ci = 0, ce = 0;
    bool more = false;
    for (uint32_t l = 0; l < nl; ++l) {
      if (at[l] >= lv[l].nbins) continue;
      more = true;
      const uint64_t lo = lv[l].lo[at[l]], hi = lv[l].hi[at[l]];
      if (lo <= x) ci |= (uint8_t)(1u << l);
      y = std::min<uint64_t>(y, lo <= x ? hi : lo);
    }
    if (!more) break;
    for (uint32_t l = 0; l < nl; ++l)
      if (((ci >> l) & 1u) && lv[l].hi[at[l]] == y) ce |= (uint8_t)(1u << l), ++at[l];
    if (ci) {
      if (S.ncls == BP_MAXCLASS) return false;
      in[S.ncls] = ci, end[S.ncls] = ce;
      S.bound[2 * S.ncls] = x, S.bound[2 * S.ncls + 1] = y;
      ++S.ncls;
    }
    x = y;
  }
  const uint64_t back = x;  // the last boundary
  // the level whose bins are the classes comes first
  uint32_t order[BP_MAXLEVELS] = {0, 1, 2, 3};
  *fine = false;
  for (uint32_t l = 0; l < nl && !*fine; ++l) {
    bool all = lv[l].nbins == S.ncls;
    for (uint32_t c = 0; c < S.ncls && all; ++c) all = ((in[c] & end[c]) >> l) & 1u;
    if (all) std::swap(order[0], order[l]), *fine = true;
  }
  const uint64_t dom = back - front;
  const bool unit = *fine && dom == S.ncls;  // equality bins without gaps
  if (unit && nl == 1 && vbytes == 1 && !src->fk && back <= BP_NOCODE) {
    *mode = BP_DIRECT;
    S.code0 = (uint32_t)front;
  } else if (dom <= BP_LUT - 1 && (vbytes == 8 || back <= (1ull << 32))) {
    // the table holds the domain (in 32-bit arithmetic for values of 4
    // bytes); for 1-byte values, every value
    *mode = BP_TABLE;
    S.dom_lo = vbytes == 1 ? 0 : front;
    S.dom_n = vbytes == 1 ? 256u : (uint32_t)dom;
  } else {
    *mode = BP_SEARCH;
    S.dom_lo = front;
    const uint64_t w = S.bound[1] - S.bound[0];
    bool equal = vbytes == 8 || (w <= 0xffffffffull && S.dom_lo <= 0xffffffffull);
    for (uint32_t c = 0; c < S.ncls && equal; ++c)
      equal = S.bound[2 * c] == S.dom_lo + c * w && S.bound[2 * c + 1] - S.bound[2 * c] == w;
    if (equal) {
      S.width = w;
      if (vbytes <= 4) {
        const DivMagic m = div_magic((uint32_t)w);
        S.div_m = m.m, S.div_s1 = m.sh1, S.div_s2 = m.sh2;
      }
    }
  }
  for (uint32_t i = 0; i < nl; ++i) {
    const uint32_t l = order[i];
    S.out[i] = lv[l].out;
    S.pop[i] = reinterpret_cast<unsigned long long *>(lv[l].popcounts);
    if (S.pop[i]) S.count = 1;
    for (uint32_t c = 0; c < S.ncls; ++c) {
      const uint32_t code = S.code0 + c;
      S.in[i][code >> 3] |= (uint8_t)(((in[c] >> l) & 1u) << (code & 7u));
      S.end[i][code >> 3] |= (uint8_t)(((end[c] >> l) & 1u) << (code & 7u));
    }
  }
  return true;
}

}  // namespace mb

using namespace mb;

extern "C" mb_status mb_bitmap_create(const mb_src *src, uint64_t nrows, const uint64_t *lo,
                                      const uint64_t *hi, uint32_t nbins, uint32_t *out,
                                      uint64_t stride_words, uint64_t *popcounts, void *stream) {
  if (!src || !lo || !hi || !out) return fail(MB_ERR_INVALID, "mb_bitmap_create: NULL argument");
  if (nbins == 0) return MB_OK;
  uint32_t w = src->width;
  if (w != 1 && w != 2 && w != 4 && w != 8)
    return fail(MB_ERR_INVALID, "mb_bitmap_create: width %u not in {1,2,4,8}", w);
  if (!src->col) return fail(MB_ERR_INVALID, "mb_bitmap_create: column is NULL");
  if (stride_words < mb_bitmap_words(nrows) || (stride_words & 3) != 0)
    return fail(MB_ERR_INVALID, "mb_bitmap_create: stride %llu < words or not a multiple of 4",
                (unsigned long long)stride_words);
  if (((uintptr_t)out & 15) != 0)
    return fail(MB_ERR_INVALID, "mb_bitmap_create: output not 16-byte aligned");
  const void *staged = src->fk ? (const void *)src->fk : src->col;
  if (((uintptr_t)staged & 15) != 0)
    return fail(MB_ERR_INVALID, "mb_bitmap_create: staged column not 16-byte aligned");
  if (nrows == 0) return MB_OK;
  cudaStream_t st = as_stream(stream);
  // More bins than one pass takes (8-byte staged columns leave room for 224
  // bins next to the ballot kernel's 3 stages): split into passes.
  const uint32_t maxb = (w == 8 && src->fk == nullptr) ? 224u : BP_MAXCLASS;
  PlaneSpec PS;
  for (uint32_t b0 = 0; b0 < nbins; b0 += maxb) {
    uint32_t nb = nbins - b0 < maxb ? nbins - b0 : maxb;
    mb_level one;
    memset(&one, 0, sizeof(one));
    one.lo = lo + b0, one.hi = hi + b0, one.nbins = nb;
    one.out = out + (uint64_t)b0 * stride_words;
    one.popcounts = popcounts ? popcounts + b0 : nullptr;
    int pmode = BP_TABLE;
    bool fine = false;
    if (planes_spec(src, &one, 1, PS, &pmode, &fine)) {
      MB_CHECK(launch_planes(pmode, fine, PS, src, nrows, stride_words, st, LevelsJoinOut{nullptr, nullptr}));
      continue;
    }
    BinSpec S;
    memset(&S, 0, sizeof(S));
    S.nbins = nb;
    for (uint32_t j = 0; j < nb; ++j) {
      S.lo[j] = lo[b0 + j];
      S.hi[j] = hi[b0 + j];
    }
    uint32_t *o = out + (uint64_t)b0 * stride_words;
    uint64_t *p = popcounts ? popcounts + b0 : nullptr;
    mb_status r;
    if (src->fk == nullptr) {
      switch (w) {
      case 1: r = launch_bc<1, false, 1>(S, src, nrows, o, stride_words, p, st); break;
      case 2: r = launch_bc<2, false, 1>(S, src, nrows, o, stride_words, p, st); break;
      case 4: r = launch_bc<4, false, 1>(S, src, nrows, o, stride_words, p, st); break;
      default: r = launch_bc<8, false, 1>(S, src, nrows, o, stride_words, p, st); break;
      }
    } else {
      switch (w) {  // staged column is the 4-byte key; w is the dimension width
      case 1: r = launch_bc<4, true, 1>(S, src, nrows, o, stride_words, p, st); break;
      case 2: r = launch_bc<4, true, 2>(S, src, nrows, o, stride_words, p, st); break;
      case 4: r = launch_bc<4, true, 4>(S, src, nrows, o, stride_words, p, st); break;
      default: r = launch_bc<4, true, 8>(S, src, nrows, o, stride_words, p, st); break;
      }
    }
    if (r != MB_OK) return r;
  }
  return MB_OK;
}

mb_status mb::bitmap_create_levels_join(const mb_src *src, uint64_t nrows, const mb_level *levels,
                                        uint32_t nlevels, uint64_t stride_words, void *stream, void *dout,
                                        unsigned long long *bad) {
  if (!src || (!levels && nlevels)) return fail(MB_ERR_INVALID, "mb_bitmap_create_levels: NULL argument");
  if (nlevels == 0) return MB_OK;
  const uint32_t w = src->width;
  if (w != 1 && w != 2 && w != 4 && w != 8)
    return fail(MB_ERR_INVALID, "mb_bitmap_create_levels: width %u not in {1,2,4,8}", w);
  if (!src->col) return fail(MB_ERR_INVALID, "mb_bitmap_create_levels: column is NULL");
  if (stride_words < mb_bitmap_words(nrows) || (stride_words & 3) != 0)
    return fail(MB_ERR_INVALID, "mb_bitmap_create_levels: stride %llu < words or not a multiple of 4",
                (unsigned long long)stride_words);
  for (uint32_t l = 0; l < nlevels; ++l)
    if (levels[l].nbins && (!levels[l].out || ((uintptr_t)levels[l].out & 15) != 0))
      return fail(MB_ERR_INVALID, "mb_bitmap_create_levels: level %u output NULL or not 16-byte aligned", l);
  const void *staged = src->fk ? (const void *)src->fk : src->col;
  if (((uintptr_t)staged & 15) != 0)
    return fail(MB_ERR_INVALID, "mb_bitmap_create_levels: staged column not 16-byte aligned");
  const bool join_out = dout || bad;
  if (join_out && !src->fk) return fail(MB_ERR_INVALID, "bitmap levels: join outputs without a foreign key");
  if (nrows == 0) return MB_OK;
  cudaStream_t st = as_stream(stream);
  PlaneSpec S;
  int mode = BP_TABLE;
  bool fine = false;
  if (!planes_spec(src, levels, nlevels, S, &mode, &fine)) {  // one pass per level
    if (join_out) return fail(MB_ERR_INVALID, "bitmap levels: join outputs need the one-pass form");
    for (uint32_t l = 0; l < nlevels; ++l)
      MB_CHECK(mb_bitmap_create(src, nrows, levels[l].lo, levels[l].hi, levels[l].nbins, levels[l].out, stride_words,
                                levels[l].popcounts, stream));
    return MB_OK;
  }
  return launch_planes(mode, fine, S, src, nrows, stride_words, st, LevelsJoinOut{dout, bad});
}

extern "C" mb_status mb_bitmap_create_levels(const mb_src *src, uint64_t nrows, const mb_level *levels,
                                             uint32_t nlevels, uint64_t stride_words, void *stream) {
  return mb::bitmap_create_levels_join(src, nrows, levels, nlevels, stride_words, stream, nullptr, nullptr);
}
