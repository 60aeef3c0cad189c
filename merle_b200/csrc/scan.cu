// scan.cu - the plans without an index: every row through the op (mb_join_grpby) and
// the same with dimension filters tested on the foreign keys (mb_hash_join_grpby).
//
// Reference kernels: grpby (primitive.cuh:16-48) and the comparison system's joins
// (crystal/src/ssb/q21.cu and its siblings).
//
// Compiled ops (shape.cuh), and any op that the clauses on fact columns filter alone or with
// key bits: the clauses that are one range on a fact column, and the
// dimensions with a filter of their own, become screens.  A warp takes 1,024 rows, each
// lane four consecutive rows in each of eight 128-row chunks, and tests the screens one
// after the other on vector loads; a lane whose four rows all failed loads no more, so
// a later column's 32-byte sectors without a live row are not fetched.  The surviving
// rows queue per warp, and full batches of 64 run the rest of the op.  Any other op, and
// small tables, go row by row (join_grpby_kernel): one clause screens, the rows that pass
// queue, and full warps of them run the op.
//
// A dimension's screen is one bit a dimension row (dimension keys are row numbers 0 ..
// dimsz - 1, so the key itself is a perfect hash): built by one pass over the dimension,
// staged in every block's shared memory while SC_STAGE_MAX bytes hold it.  The attributes
// of a surviving row are read from the dimension's columns.
//
// What bounds it: instruction issue and the bytes of the columns about equally (60 % of the
// issue slots, 60-70 % of the measured copy rate).  120M rows, 1- to 4-byte columns, one
// query of each template: 336 / 378 / 540 / 591 us with one clause screened and the op
// interpreted, 137 / 112 / 148 / 210 us here; with joins (600K customers, 1.06M parts) 532 / 1335
// / 1631 us through open-addressing tables of {key, attributes}, 168 / 220 / 327 us.
// 32 warps an SM (64 registers a thread) against 24: 187 and 220 us on template 1; tiles of 1,024
// rows against 512 and 256: 160 / 187 / 284 us; failures shifted into words instead
// of set bit by bit and one compaction a tile: 160 -> 137 us.  Key bits staged up to
// 32 / 100 / 140 KB: template 2's joined query 188 / 186 / 169 us.
#include <string.h>
#include <algorithm>
#include "common.cuh"
#include "opeval.cuh"
#include "shape.cuh"
#include "vbp.cuh"

namespace mb {

constexpr uint32_t SC_WARPS = 32;                  // one block an SM: 64 registers a thread
constexpr uint32_t SC_CHUNKS = 8;                  // 128-row chunks of a tile
constexpr uint32_t SC_TILE = 128 * SC_CHUNKS;
constexpr uint32_t SC_QCAP = 256 + 64;             // two chunks' rows + fewer than 64 pending
constexpr uint32_t SC_STAGE_MAX = 140 * 1024;      // bytes of staged key bits
constexpr uint32_t HJ_MAXT = 4;                    // dimensions (distinct foreign keys) with a filter per op
constexpr uint32_t HJ_PAY = 3;                     // op attributes on one such key

// A screen: lo <= value <= lo + span over a fact column of `width` bytes, or (width 0)
// bit key of `bits` set, the key read from `col`.
struct Screen {
  const void *col;
  const uint32_t *bits;
  uint64_t lo, span;
  uint64_t nkeys;       // width 0: keys >= nkeys fail
  uint32_t width;
  uint32_t vec;         // the column is aligned for loads of four elements
  uint32_t staged;      // width 0: word offset of the staged copy, or ~0u
  uint32_t pad_;
};

struct ScanArgs {
  uint32_t ns;
  uint32_t ntab;             // dimensions whose key bits were built
  const uint32_t *any;       // [ntab]: 1 if a row of the dimension passes
  Screen s[MB_MAXCLAUSE];
};

// Clauses `mask` of O, evaluated on dimension rows, and where their bits go.
struct DimFilter {
  uint64_t n;            // dimension rows
  uint32_t *bits;        // ceil(n / 32) words
  uint32_t clauses;
};
struct DimFilters {
  DimFilter d[HJ_MAXT];
  uint32_t *any;
};

// Key bits of dimension blockIdx.y: one row a lane, one word a warp step.
__global__ void __launch_bounds__(256)
dim_bits_kernel(const __grid_constant__ mb_op O, const __grid_constant__ DimFilters F) {
  const DimFilter &D = F.d[blockIdx.y];
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t nw = (uint64_t)gridDim.x * (blockDim.x / 32), words = (D.n + 31) / 32;
  uint32_t some = 0;
  for (uint64_t w = (uint64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; w < words; w += nw) {
    const uint64_t d = w * 32 + lane;
    bool pass = d < D.n;
    uint32_t t = 0;
    for (uint32_t c = 0; c < O.nclause; ++c) {
      const uint32_t len = O.clause_len[c];
      if ((D.clauses >> c & 1u) && pass) {
        bool one = false;
        for (uint32_t k = t; k < t + len && !one; ++k) {
          const mb_term &tm = O.terms[k];
          const uint64_t v = load_width(O.src[tm.src].col, d, O.src[tm.src].width);
          one = v >= tm.lo && v < tm.hi;
        }
        pass = one;
      }
      t += len;
    }
    const uint32_t m = __ballot_sync(0xffffffffu, pass);
    if (lane == 0) D.bits[w] = m;
    some |= m;
  }
  if (__syncthreads_or(some != 0) && threadIdx.x == 0) F.any[blockIdx.y] = 1u;
}

// Four consecutive elements of a W-byte column as its raw words: the vector load of all four,
// or one by one where the column is not aligned for it or the table ends.  Elements are taken
// out only when they are tested, so the loads of a tile's chunks are all in flight together.
template <int W>
struct Four {
  static constexpr int NW = W;  // 4 elements x W bytes / 4
  uint32_t w[NW];
  __device__ __forceinline__ void vec(const void *col, uint64_t r, bool on) {
    if (W == 1) {
      w[0] = on ? __ldg(reinterpret_cast<const uint32_t *>(col) + r / 4) : 0u;
    } else if (W == 2) {
      const uint2 t = on ? __ldg(reinterpret_cast<const uint2 *>(col) + r / 4) : make_uint2(0, 0);
      w[0] = t.x, w[1 % NW] = t.y;
    } else {
#pragma unroll
      for (int i = 0; i < W / 4; ++i) {
        const uint4 t = on ? __ldg(reinterpret_cast<const uint4 *>(col) + r / 4 * (W / 4) + i) : make_uint4(0, 0, 0, 0);
        w[(4 * i) % NW] = t.x, w[(4 * i + 1) % NW] = t.y, w[(4 * i + 2) % NW] = t.z, w[(4 * i + 3) % NW] = t.w;
      }
    }
  }
  __device__ __forceinline__ void one(const void *col, uint64_t r, uint32_t live) {
#pragma unroll
    for (int i = 0; i < NW; ++i) w[i] = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (!(live >> j & 1u)) continue;
      const uint64_t v = load_width(col, r + j, W);
      if (W == 8) w[(2 * j) % NW] = (uint32_t)v, w[(2 * j + 1) % NW] = (uint32_t)(v >> 32);
      else w[j * W / 4 % NW] |= (uint32_t)v << (8 * (j * W % 4));
    }
  }
};

template <int W>
__device__ __forceinline__ void screen_load(const Screen &S, uint64_t r0, uint32_t live, bool full,
                                            Four<W> (&x)[SC_CHUNKS]) {
  if (S.vec && full) {
#pragma unroll
    for (int c = 0; c < (int)SC_CHUNKS; ++c) x[c].vec(S.col, r0 + 128 * c, (live >> (4 * c) & 0xfu) != 0);
  } else {
#pragma unroll
    for (int c = 0; c < (int)SC_CHUNKS; ++c) x[c].one(S.col, r0 + 128 * c, live >> (4 * c) & 0xfu);
  }
}

// Screens return the live rows (bit 4c + j: row r0 + 128 c + j) that pass; full: all rows
// of the tile exist.  Each form spends as few instructions a row as it can, for the scan's issue
// slots are as scarce as its bytes: failures are shifted into one word, 16 or 32 rows
// of it, instead of set bit by bit.

// Key bits, from shared (staged) or global memory.
template <bool STAGED>
__device__ __forceinline__ uint32_t screen_keys(const Screen &S, uint64_t r0, uint32_t live, bool full,
                                                const uint32_t *bits) {
  Four<4> x[SC_CHUNKS];
  screen_load(S, r0, live, full, x);
  const uint32_t last = (uint32_t)(S.nkeys - 1);
  uint32_t m = 0;
#pragma unroll
  for (int i = 4 * (int)SC_CHUNKS - 1; i >= 0; --i) {
    const uint32_t k = x[i / 4].w[i % 4];
    uint32_t w = 0;
    if ((live >> i & 1u) && k <= last) w = STAGED ? bits[k >> 5] : __ldg(bits + (k >> 5));
    m = m + m + (w >> (k & 31) & 1u);
  }
  return m & live;
}

// A range on a 4-byte column: v - lo > span is the carry of (v - lo) + ~span.
__device__ __forceinline__ uint32_t screen_words(const Screen &S, uint64_t r0, uint32_t live, bool full) {
  const uint32_t lo = (uint32_t)S.lo, nspan = ~(uint32_t)S.span;
  Four<4> x[SC_CHUNKS];
  screen_load(S, r0, live, full, x);
  uint32_t f = 0;
#pragma unroll
  for (int i = 4 * (int)SC_CHUNKS - 1; i >= 0; --i) {
    uint32_t t;
    asm("add.cc.u32 %0, %2, %3;\n\taddc.u32 %1, %1, %1;" : "=&r"(t), "+r"(f) : "r"(x[i / 4].w[i % 4] - lo), "r"(nspan));
  }
  return ~f & live;
}

// A range on a 2-byte column, the two rows of a word at once: clamped to the range, a value
// outside changes; its 1 is shifted into the half's failures, which a perfect shuffle
// (Warren, Hacker's Delight, 2nd edition, section 7-2) brings into row order.
__device__ __forceinline__ uint32_t screen_halves(const Screen &S, uint64_t r0, uint32_t live, bool full) {
  static_assert(SC_CHUNKS == 8, "16 words of two rows");
  const uint32_t lo = (uint32_t)S.lo * 0x10001u, hi = (uint32_t)(S.lo + S.span) * 0x10001u;
  Four<2> x[SC_CHUNKS];
  screen_load(S, r0, live, full, x);
  uint32_t f = 0;  // bit i: even row of word i failed, bit 16 + i: the odd one
#pragma unroll
  for (int i = 2 * (int)SC_CHUNKS - 1; i >= 0; --i) {
    const uint32_t w = x[i / 2].w[i % 2];
    f = f + f + __vminu2(w ^ __vminu2(__vmaxu2(w, lo), hi), 0x10001u);
  }
  uint32_t t;
  t = (f ^ (f >> 8)) & 0x0000ff00u, f ^= t ^ (t << 8);
  t = (f ^ (f >> 4)) & 0x00f000f0u, f ^= t ^ (t << 4);
  t = (f ^ (f >> 2)) & 0x0c0c0c0cu, f ^= t ^ (t << 2);
  t = (f ^ (f >> 1)) & 0x22222222u, f ^= t ^ (t << 1);
  return ~f & live;
}

__device__ __forceinline__ uint32_t screen_longs(const Screen &S, uint64_t r0, uint32_t live, bool full) {
  Four<8> x[SC_CHUNKS];
  screen_load(S, r0, live, full, x);
  uint32_t m = 0;
#pragma unroll
  for (int i = 0; i < 4 * (int)SC_CHUNKS; ++i) {
    const uint64_t v = x[i / 4].w[2 * (i % 4)] | (uint64_t)x[i / 4].w[2 * (i % 4) + 1] << 32;
    if (v - S.lo <= S.span) m |= 1u << i;
  }
  return m & live;
}

// A range on a byte column, the four rows of a word at once: per byte d = x - lo mod 256
// (the top bits kept out of the borrow), then d <= span from the borrow of span - d and the
// two top bits; the four results are gathered by a multiply.
__device__ __forceinline__ uint32_t screen_bytes(const Screen &S, uint64_t r0, uint32_t live, bool full) {
  constexpr uint32_t H = 0x80808080u;
  const uint32_t lo = (uint32_t)S.lo * 0x01010101u, sp = (uint32_t)S.span * 0x01010101u;
  Four<1> x[SC_CHUNKS];
  screen_load(S, r0, live, full, x);
  uint32_t m = 0;
#pragma unroll
  for (int c = 0; c < (int)SC_CHUNKS; ++c) {
    const uint32_t w = x[c].w[0];
    const uint32_t d = ((w | H) - (lo & ~H)) ^ ((w ^ ~lo) & H);
    const uint32_t t = (sp | H) - (d & ~H);  // top bit: low 7 bits of d <= those of span
    const uint32_t ok = ((~d & sp) | (~(d ^ sp) & t)) & H;
    m |= ((ok >> 7) * 0x01020408u >> 24 & 0xfu) << (4 * c);
  }
  return m & live;
}

__device__ __forceinline__ uint32_t screen_rows(const Screen &S, uint64_t r0, uint32_t live, bool full,
                                                const uint32_t *stage) {
  switch (S.width) {
  case 0:
    return S.staged != ~0u ? screen_keys<true>(S, r0, live, full, stage + S.staged)
                           : screen_keys<false>(S, r0, live, full, S.bits);
  case 1: return screen_bytes(S, r0, live, full);
  case 2: return screen_halves(S, r0, live, full);
  case 4: return screen_words(S, r0, live, full);
  default: return screen_longs(S, r0, live, full);
  }
}

// The scan of one block: screens, compaction, drain of full batches.
template <int GS, class DR>
__device__ __forceinline__ void scan_body(uint64_t nrows, const DR &dr, const ScanArgs &A, uint32_t nr_grp,
                                          uint32_t grp_bytes, uint32_t stage_words, unsigned long long *out,
                                          unsigned long long *nqual, uint8_t *smem) {
  __shared__ uint64_t red[64];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint32_t t = 0; t < A.ntab; ++t)
    if (!A.any[t]) return;  // a dimension without a passing row: nothing qualifies
  const GrpCtx G = grp_init<GS>(smem, nr_grp, 0, out);
  uint32_t *stage = reinterpret_cast<uint32_t *>(smem + grp_bytes);
  uint32_t *queue = stage + stage_words + warp * SC_QCAP;
  for (uint32_t i = 0; i < A.ns; ++i) {
    const Screen &S = A.s[i];
    if (S.width || S.staged == ~0u) continue;
    const uint32_t nv = (uint32_t)((S.nkeys + 127) / 128);
    uint4 *dst = reinterpret_cast<uint4 *>(stage + S.staged);
    const uint4 *src = reinterpret_cast<const uint4 *>(S.bits);
    for (uint32_t k = threadIdx.x; k < nv; k += blockDim.x) dst[k] = src[k];
  }
  __syncthreads();
  int64_t acc = 0;
  uint32_t cnt = 0, qn = 0;
  const uint64_t ntiles = (nrows + SC_TILE - 1) / SC_TILE;
  // consecutive tiles go to different SMs, so that a small table uses all of them
  for (uint64_t t = (uint64_t)warp * gridDim.x + blockIdx.x; t < ntiles; t += (uint64_t)gridDim.x * SC_WARPS) {
    const uint64_t r0 = t * SC_TILE + 4 * lane;
    const bool full = (t + 1) * SC_TILE <= nrows;
    uint32_t live = 0xffffffffu >> (32 - 4 * SC_CHUNKS);
    if (!full) {
#pragma unroll
      for (int b = 0; b < (int)(4 * SC_CHUNKS); ++b)
        if (r0 + 128 * (b / 4) + (b & 3) >= nrows) live &= ~(1u << b);
    }
    for (uint32_t i = 0; i < A.ns; ++i) {
      live = screen_rows(A.s[i], r0, live, full, stage);
      if (!__any_sync(0xffffffffu, live != 0)) break;
    }
    // the queue takes 256 rows: all of a tile's survivors at once, or two chunks at a time
    uint32_t part = __reduce_add_sync(0xffffffffu, __popc(live)) <= 256 ? 0xffffffffu : 0xffu;
#pragma unroll 1
    for (; part; part = part == 0xffffffffu ? 0u : part << 8) {
      uint32_t m = live & part;
      if (!__any_sync(0xffffffffu, m != 0)) continue;
      const uint32_t pc = __popc(m);
      uint32_t incl = pc;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= (uint32_t)d) incl += y;
      }
      uint32_t *w = queue + (qn + incl - pc);
      const uint32_t rb = (uint32_t)r0;
      while (m) {
        const uint32_t b = __ffs(m) - 1;
        m &= m - 1;
        *w++ = rb + 128 * (b >> 2) + (b & 3);
      }
      qn += __shfl_sync(0xffffffffu, incl, 31);
      __syncwarp();
      while (qn >= 64) {  // from the end: the queue's order is irrelevant
        qn -= 64;
        dr.drain(queue + qn, 64, G, acc, cnt);
      }
      __syncwarp();
    }
  }
  if (qn) dr.drain(queue, qn, G, acc, cnt);
  __syncthreads();
  grp_flush<GS>(G, nr_grp, acc, cnt, nqual, red);
}

// Any op without the clauses that are screens, a row a lane (CHK: it still has some).
// Loading every source of two rows together instead: 1.1 to 1.9 times as long on
// interpreted ops (240M rows, half of them selected, 200 groups: 1,062 us here, 1,464).
template <int GS, bool CHK>
struct OpDrain {
  const mb_op &O;
  uint32_t nr_grp;
  __device__ __forceinline__ void drain(const uint32_t *q, uint32_t n, const GrpCtx &G, int64_t &acc,
                                        uint32_t &cnt) const {
#pragma unroll 1
    for (uint32_t i = threadIdx.x & 31; i < 64; i += 32) {
      bool kept = false;
      int64_t val = 0;
      uint32_t grp = 0;
      if (i < n) kept = op_eval(O, q[i], CHK, nr_grp, val, grp);
      cnt += kept ? 1u : 0u;
      aggregate<GS>(G, kept, grp, val, acc);
    }
  }
};

template <int GS, bool CHK>
__global__ void __launch_bounds__(SC_WARPS * 32, 1)
scan_kernel(uint64_t nrows, const __grid_constant__ mb_op O, const __grid_constant__ ScanArgs A, uint32_t nr_grp,
            uint32_t grp_bytes, uint32_t stage_words, unsigned long long *__restrict__ out,
            unsigned long long *__restrict__ nqual) {
  extern __shared__ __align__(16) uint8_t smem[];
  scan_body<GS>(nrows, OpDrain<GS, CHK>{O, nr_grp}, A, nr_grp, grp_bytes, stage_words, out, nqual, smem);
}

// A compiled op all of whose clauses are screens (shape.cuh).
template <int GS, int SH, bool NARROW, bool JOIN>
struct ScanShapeDrain {
  const ShapeArgs &S;
  __device__ __forceinline__ void drain(const uint32_t *q, uint32_t n, const GrpCtx &G, int64_t &acc,
                                        uint32_t &cnt) const {
    shape_rows<SH, NARROW, false, GS, 2, JOIN>(S, q, n, false, G, acc, cnt);
  }
};

template <int GS, int SH, bool NARROW, bool JOIN>
__global__ void __launch_bounds__(SC_WARPS * 32, 1)
scan_shape_kernel(uint64_t nrows, const __grid_constant__ ShapeArgs S, const __grid_constant__ ScanArgs A,
                  uint32_t nr_grp, uint32_t grp_bytes, uint32_t stage_words, unsigned long long *__restrict__ out,
                  unsigned long long *__restrict__ nqual) {
  extern __shared__ __align__(16) uint8_t smem[];
  scan_body<GS>(nrows, ScanShapeDrain<GS, SH, NARROW, JOIN>{S}, A, nr_grp, grp_bytes, stage_words, out, nqual, smem);
}

// ------------------------------------------------- rows through an interpreted op
// Clause c alone on one row, as op_eval evaluates it.
__device__ __forceinline__ bool clause_pass(const mb_op &O, uint32_t c, uint32_t t0, uint32_t row) {
  bool any = false;
  for (uint32_t k = 0; k < O.clause_len[c] && !any; ++k) {
    const mb_term &tm = O.terms[t0 + k];
    uint64_t v;
    any = src_value(O.src[tm.src], row, v) && v >= tm.lo && v < tm.hi;
  }
  return any;
}

constexpr uint32_t JOIN_WARPS = 8;
constexpr uint32_t JQ = 160;  // rows a warp queues between the screen and the op (31 + a 128-row chunk)

// Every row through the op.  A row first meets one clause (`screen`, first
// term `t0`; none if screen >= nclause), one row per lane; the rows that pass
// queue per warp, and each full warp of them runs the rest of the op, so the
// lanes of its loads and branches are all live rows.  The result equals
// op_eval on every row (the screen is one of the op's own clauses).
// Four consecutive values of a fact column of SW-byte elements from one
// vector load (the column 16-byte aligned, rows r .. r+3 inside it, r a
// multiple of 4).
template <int SW>
__device__ __forceinline__ void load4(const void *col, uint64_t r, uint64_t (&v)[4]) {
  if (SW == 1) {
    const uint32_t w = __ldg(reinterpret_cast<const uint32_t *>(col) + r / 4);
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = (w >> (8 * j)) & 0xffu;
  } else if (SW == 2) {
    const uint2 w = __ldg(reinterpret_cast<const uint2 *>(col) + r / 4);
    v[0] = w.x & 0xffffu, v[1] = w.x >> 16, v[2] = w.y & 0xffffu, v[3] = w.y >> 16;
  } else if (SW == 4) {
    const uint4 w = __ldg(reinterpret_cast<const uint4 *>(col) + r / 4);
    v[0] = w.x, v[1] = w.y, v[2] = w.z, v[3] = w.w;
  } else {
    const ulonglong2 a = __ldg(reinterpret_cast<const ulonglong2 *>(col) + r / 2),
                     b = __ldg(reinterpret_cast<const ulonglong2 *>(col) + r / 2 + 1);
    v[0] = a.x, v[1] = a.y, v[2] = b.x, v[3] = b.y;
  }
}

template <int GS, int SW>
__global__ void __launch_bounds__(256, 8)
join_grpby_kernel(uint64_t nrows, const __grid_constant__ mb_op O, uint32_t nr_grp, uint32_t grp_bytes, uint32_t screen, uint32_t t0, unsigned long long *__restrict__ out,
                  unsigned long long *__restrict__ nqual) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ uint64_t red[64];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  GrpCtx G = grp_init<GS>(smem, nr_grp, 0, out);
  uint32_t *queue = reinterpret_cast<uint32_t *>(smem + grp_bytes) + (size_t)warp * JQ;
  __syncthreads();
  int64_t acc = 0;
  uint32_t cnt = 0;
  uint32_t qn = 0;
  const uint32_t lt = (1u << lane) - 1u;
  auto drain = [&](uint32_t m) {  // the last m (<= 32) queued rows through the op
    bool kept = false;
    int64_t val = 0;
    uint32_t grp = 0;
    if (lane < m) kept = op_eval(O, queue[qn - m + lane], true, nr_grp, val, grp, screen);
    cnt += kept ? 1u : 0u;
    aggregate<GS>(G, kept, grp, val, acc);
    qn -= m;
    __syncwarp();
  };
  const uint64_t nchunks = (nrows + 31) / 32;
  if (screen >= O.nclause) {  // no screen (or no room for the queues): every row through the op
    for (uint64_t ch = (uint64_t)blockIdx.x * nw + warp; ch < nchunks; ch += (uint64_t)gridDim.x * nw) {
      const uint64_t row = ch * 32 + lane;
      bool kept = false;
      int64_t val = 0;
      uint32_t grp = 0;
      if (row < nrows) kept = op_eval(O, (uint32_t)row, true, nr_grp, val, grp);
      cnt += kept ? 1u : 0u;
      aggregate<GS>(G, kept, grp, val, acc);
    }
  } else if (SW == 0) {
    for (uint64_t ch = (uint64_t)blockIdx.x * nw + warp; ch < nchunks; ch += (uint64_t)gridDim.x * nw) {
      const uint64_t row = ch * 32 + lane;
      const bool pass = row < nrows && clause_pass(O, screen, t0, (uint32_t)row);
      const uint32_t bal = __ballot_sync(0xffffffffu, pass);
      if (pass) queue[qn + __popc(bal & lt)] = (uint32_t)row;
      qn += __popc(bal);  // at most 31 + 32 < JQ
      __syncwarp();
      if (qn >= 32) drain(32);
    }
    if (qn) drain(qn);
  } else {
    // the screen is one range on a fact column of SW-byte elements: four rows
    // a lane from one vector load; 128-row chunks, the last one partly by
    // scalar loads
    const mb_term &tm = O.terms[t0];
    const void *col = O.src[tm.src].col;
    const uint64_t lo = tm.lo, hi = tm.hi, nch4 = (nrows + 127) / 128;
    for (uint64_t ch = (uint64_t)blockIdx.x * nw + warp; ch < nch4; ch += (uint64_t)gridDim.x * nw) {
      const uint64_t r = ch * 128 + 4 * lane;
      uint64_t v[4] = {0, 0, 0, 0};
      if (ch * 128 + 128 <= nrows) {
        load4<SW>(col, r, v);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (r + j < nrows) v[j] = load_width(col, r + j, SW);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const bool pass = r + j < nrows && v[j] >= lo && v[j] < hi;
        const uint32_t bal = __ballot_sync(0xffffffffu, pass);
        if (pass) queue[qn + __popc(bal & lt)] = (uint32_t)(r + j);
        qn += __popc(bal);  // at most 31 + 128 < JQ
      }
      __syncwarp();
      while (qn >= 32) drain(32);
    }
    if (qn) drain(qn);
  }
  __syncthreads();
  grp_flush<GS>(G, nr_grp, acc, cnt, nqual, red);
}

// ------------------------------------------------------------------ host
struct ScanCall {
  uint64_t n;
  uint32_t nr_grp;
  unsigned long long *out, *nqual;
  cudaStream_t st;
};

// op: the kernel's argument that carries the op (one or two of them).
template <typename K, typename... OP>
static mb_status scan_launch(K kern, int gs, const ScanCall &C, ScanArgs &A, const OP &...op) {
  const DevInfo &di = dev_info();
  const size_t gb = (grp_smem_bytes(gs, C.nr_grp, 0) + 15) & ~(size_t)15, qb = (size_t)SC_WARPS * SC_QCAP * 4;
  // key bits are staged in screening order (the smaller dimensions first)
  uint32_t words = 0;
  for (uint32_t i = 0; i < A.ns; ++i) {
    Screen &S = A.s[i];
    if (S.width) continue;
    const uint64_t w = round_up(S.nkeys, 128) / 32;
    if ((words + w) * 4 > SC_STAGE_MAX || gb + qb + (words + w) * 4 + 1024 > (size_t)di.max_smem_optin) continue;
    S.staged = words;
    words += (uint32_t)w;
  }
  const size_t smem = gb + (size_t)words * 4 + qb;
  if (smem > (size_t)di.max_smem_optin) return fail(MB_ERR_INVALID, "scan: %zu bytes of shared memory", smem);
  MB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const uint64_t ntiles = (C.n + SC_TILE - 1) / SC_TILE;
  const unsigned grid = (unsigned)std::min<uint64_t>((uint64_t)di.sms, ntiles);
  kern<<<grid, SC_WARPS * 32, smem, C.st>>>(C.n, op..., A, C.nr_grp, (uint32_t)gb, words, C.out, C.nqual);
  MB_LAUNCH_CHECK("scan_kernel");
  return MB_OK;
}

template <int GS>
static mb_status scan_gs(const ScanCall &C, const mb_op &O, ScanArgs &A) {
  return O.nclause ? scan_launch(scan_kernel<GS, true>, GS, C, A, O) : scan_launch(scan_kernel<GS, false>, GS, C, A, O);
}

// The clause that screens rows in the no-index scan: the first whose terms
// read fact columns only (one load a row), else the first; nclause if none.
static uint32_t screen_clause(const mb_op &O, uint32_t *t0) {
  uint32_t t = 0, first_t = 0;
  for (uint32_t c = 0; c < O.nclause; ++c) {
    bool fact = true;
    for (uint32_t k = 0; k < O.clause_len[c]; ++k)
      if (O.src[O.terms[t + k].src].fk) fact = false;
    if (fact) {
      *t0 = t;
      return c;
    }
    t += O.clause_len[c];
  }
  *t0 = first_t;
  return 0;
}

template <int GS, int SW>
static mb_status join_launch(const ScanCall &C, const mb_op &O, uint32_t screen, uint32_t t0) {
  auto kern = join_grpby_kernel<GS, SW>;
  const DevInfo &di = dev_info();
  const size_t gb = (grp_smem_bytes(GS, C.nr_grp, 0) + 15) & ~(size_t)15, qbytes = (size_t)JOIN_WARPS * JQ * 4;
  // the row queues only where they cost no resident CTA (a large group
  // table in shared memory can leave no room for them)
  const size_t cap = (size_t)di.max_smem_optin - 1024;  // room for the kernel's static shared memory
  MB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)std::min(cap, gb + qbytes)));
  int with = 0, occ = 0;
  MB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, JOIN_WARPS * 32, gb));
  if (gb + qbytes <= cap) MB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&with, kern, JOIN_WARPS * 32, gb + qbytes));
  if (with < occ) screen = O.nclause;
  if (occ < 1) return fail(MB_ERR_INVALID, "kernel does not fit on an SM (smem %zu)", gb);
  const unsigned grid = (unsigned)std::min<uint64_t>((uint64_t)di.sms * occ, ceil_div(ceil_div(C.n, 32), JOIN_WARPS));
  kern<<<grid, JOIN_WARPS * 32, gb + (screen < O.nclause ? qbytes : 0), C.st>>>(C.n, O, C.nr_grp, (uint32_t)gb, screen,
                                                                               t0, C.out, C.nqual);
  MB_LAUNCH_CHECK("join_grpby_kernel");
  return MB_OK;
}

// The screen's shape picks the kernel: one range on a 16-byte-aligned fact
// column screens four rows a lane (its width a template argument).
template <int GS>
static mb_status join_gs(const ScanCall &C, const mb_op &O) {
  uint32_t t0 = 0;
  const uint32_t screen = screen_clause(O, &t0);
  uint32_t sw = 0;
  if (screen < O.nclause && O.clause_len[screen] == 1) {
    const mb_src &s = O.src[O.terms[t0].src];
    if (!s.fk && (reinterpret_cast<uintptr_t>(s.col) & 15) == 0) sw = s.width;
  }
  switch (sw) {
  case 1: return join_launch<GS, 1>(C, O, screen, t0);
  case 2: return join_launch<GS, 2>(C, O, screen, t0);
  case 4: return join_launch<GS, 4>(C, O, screen, t0);
  case 8: return join_launch<GS, 8>(C, O, screen, t0);
  default: return join_launch<GS, 0>(C, O, screen, t0);
  }
}

template <int SH>
static mb_status scan_shape(const ScanCall &C, const ShapeArgs &S, bool narrow, bool join, ScanArgs &A) {
  if constexpr (BSHAPES[SH].keym == 0) {
    return narrow ? scan_launch(scan_shape_kernel<GS_SCALAR, SH, true, false>, GS_SCALAR, C, A, S)
                  : scan_launch(scan_shape_kernel<GS_SCALAR, SH, false, false>, GS_SCALAR, C, A, S);
  } else {
    if (join)
      return narrow ? scan_launch(scan_shape_kernel<GS_SHARED, SH, true, true>, GS_SHARED, C, A, S)
                    : scan_launch(scan_shape_kernel<GS_SHARED, SH, false, true>, GS_SHARED, C, A, S);
    return narrow ? scan_launch(scan_shape_kernel<GS_SHARED, SH, true, false>, GS_SHARED, C, A, S)
                  : scan_launch(scan_shape_kernel<GS_SHARED, SH, false, false>, GS_SHARED, C, A, S);
  }
}

// The rest of the scan once the key screens are in A: `done` clauses (bit c) hold for
// every row that passes them, and the sources `keyed` (bit s) are read through a key that
// one of them has bounded.  A one-range clause on a fact column becomes a screen
// (before the key screens: its loads are plain streams); the others stay with the op.
static mb_status scan_rest(uint64_t n, const mb_op &op, uint32_t done, uint32_t keyed, ScanArgs &A, uint32_t nr_grp,
                           int64_t *out, uint64_t *nqual, cudaStream_t st) {
  mb_op O = op;
  O.nclause = 0;
  Screen range[MB_MAXCLAUSE];
  uint32_t nr = 0, t = 0, kept = 0;
  for (uint32_t c = 0; c < op.nclause; ++c) {
    const uint32_t len = op.clause_len[c];
    const mb_term &tm = op.terms[t];
    t += len;
    if (done >> c & 1u) continue;
    if (len == 1 && !op.src[tm.src].fk && tm.lo < tm.hi) {
      const mb_src &s = op.src[tm.src];
      const uint64_t top = s.width >= 8 ? ~0ull : (1ull << (8 * s.width)) - 1;
      if (tm.lo <= top) {
        Screen &S = range[nr++];
        memset(&S, 0, sizeof(S));
        S.col = s.col;
        S.width = s.width;
        S.lo = tm.lo;
        S.span = std::min(tm.hi - 1, top) - tm.lo;
        S.vec = (reinterpret_cast<uintptr_t>(s.col) & (s.width >= 4 ? 15u : 4u * s.width - 1)) == 0;
        continue;
      }
    }
    O.clause_len[O.nclause++] = len;
    for (uint32_t k = 0; k < len; ++k) O.terms[kept++] = op.terms[t - len + k];
  }
  memmove(A.s + nr, A.s, A.ns * sizeof(Screen));
  memcpy(A.s, range, nr * sizeof(Screen));
  A.ns += nr;
  const ScanCall C{n, nr_grp, reinterpret_cast<unsigned long long *>(out), reinterpret_cast<unsigned long long *>(nqual),
                   st};
  const int gs = pick_gs(nr_grp, MB_GRP_AUTO);
  ShapeArgs S;
  bool narrow = false;
  const int sh = O.nclause ? -1 : shape_of(op, nr_grp, ~0u, &S, &narrow, keyed);
  if (sh >= 0 && gs == (sh == 0 ? GS_SCALAR : GS_SHARED)) {
    const bool join = S.fk[0] || S.fk[1] || S.fk[2] || S.fk[3] || S.fk[4] || S.fk[5];
    if (sh == 0 && !join) return scan_shape<0>(C, S, narrow, join, A);
    if (sh == 1) return scan_shape<1>(C, S, narrow, join, A);
    if (sh == 2) return scan_shape<2>(C, S, narrow, join, A);
    if (sh == 3) return scan_shape<3>(C, S, narrow, join, A);
  }
  // An interpreted op goes through the screens where it has one, a range on a fact column or
  // a dimension's key bits, on tables of a tile a warp and more.  Else the row scan is the
  // faster.  Row scan / screens, us, 240M rows, 200 groups (6M, 300K in
  // brackets): half of the rows by one range 1,033 / 1,062 (36 / 41, 13 / 22), a tenth
  // 443 / 365 (26 / 18, 11 / 12), two ranges 1,292 / 646 (43 / 29, 12 / 17); no clause 1,398 /
  // 1,598 (42 / 60, 20 / 32), a dimension's clause 1,073 / 2,790 (39 / 96, 14 / 53), an OR
  // 1,435 / 2,987 (47 / 108, 14 / 53); 60M rows, an 8-byte value or clause 272 / 312 and 264 /
  // 326.  Where clauses are left for the rows that pass the screens, it depends on how many do:
  // a third and a dimension's clause 957 / 1,230 (36 / 45, 12 / 26); the benchmark's queries
  // over unindexed dimensions, 120M rows: flight 2 405 / 433, 338 / 312, 305 / 251, flight 3
  // 565 / 536, 233 / 176, 187 / 122, 173 / 89, flight 4 638 / 755, 544 / 302, 224 / 132.
  if (A.ntab == 0 && (nr == 0 || op_reads_wide(op) || n < (uint64_t)dev_info().sms * SC_WARPS * SC_TILE)) {
    switch (gs) {
    case GS_SCALAR: return join_gs<GS_SCALAR>(C, op);
    case GS_SHARED: return join_gs<GS_SHARED>(C, op);
    default: return join_gs<GS_GLOBAL>(C, op);
    }
  }
  switch (gs) {
  case GS_SCALAR: return scan_gs<GS_SCALAR>(C, O, A);
  case GS_SHARED: return scan_gs<GS_SHARED>(C, O, A);
  default: return scan_gs<GS_GLOBAL>(C, O, A);
  }
}

static mb_status scan_begin(const char *who, uint64_t nrows, const mb_op *op, uint32_t nr_grp, int64_t *out,
                            uint64_t *nqual) {
  if (!out || !nqual) return fail(MB_ERR_INVALID, "%s: NULL output", who);
  if (nr_grp == 0) return fail(MB_ERR_INVALID, "%s: nr_grp == 0", who);
  MB_CHECK(validate_op(op));
  if (nrows >= (1ull << 32)) return fail(MB_ERR_INVALID, "%s: rows >= 2^32", who);
  return MB_OK;
}

static mb_status scan_zero(uint32_t nr_grp, int64_t *out, uint64_t *nqual, cudaStream_t st) {
  MB_CUDA(cudaMemsetAsync(out, 0, (size_t)nr_grp * sizeof(int64_t), st));
  MB_CUDA(cudaMemsetAsync(nqual, 0, sizeof(uint64_t), st));
  return MB_OK;
}

}  // namespace mb

using namespace mb;

extern "C" mb_status mb_join_grpby(uint64_t nrows, const mb_op *op, uint32_t nr_grp, int64_t *out, uint64_t *nqual,
                                   void *stream) {
  MB_CHECK(scan_begin("mb_join_grpby", nrows, op, nr_grp, out, nqual));
  cudaStream_t st = as_stream(stream);
  MB_CHECK(scan_zero(nr_grp, out, nqual, st));
  if (nrows == 0) return MB_OK;
  ScanArgs A;
  memset(&A, 0, sizeof(A));
  return scan_rest(nrows, *op, 0, 0, A, nr_grp, out, nqual, st);
}

extern "C" mb_status mb_hash_join_grpby(uint64_t nrows, const mb_op *op, uint32_t nr_grp, int64_t *out,
                                        uint64_t *nqual, void *stream) {
  MB_CHECK(scan_begin("mb_hash_join_grpby", nrows, op, nr_grp, out, nqual));
  const mb_op &O = *op;
  // clauses whose terms all read one foreign key's dimension filter that dimension
  struct Dim {
    const uint32_t *fk;
    uint64_t n;
    uint32_t clauses, npay;
  } dim[HJ_MAXT];
  uint32_t nd = 0, done = 0, keyed = 0, t0 = 0;
  for (uint32_t c = 0; c < O.nclause; ++c) {
    const uint32_t *fk = nullptr;
    bool one = O.clause_len[c] > 0;
    for (uint32_t k = 0; k < O.clause_len[c]; ++k) {
      const mb_src &s = O.src[O.terms[t0 + k].src];
      if (!s.fk || s.dimsz == 0 || s.width > 4 || (fk && s.fk != fk)) one = false;
      fk = s.fk;
    }
    t0 += O.clause_len[c];
    if (!one) continue;
    uint32_t t = 0;
    while (t < nd && dim[t].fk != fk) ++t;
    if (t == nd) {
      if (nd == HJ_MAXT) continue;  // more keys than that: the clause stays with the op
      dim[nd++] = Dim{fk, ~0ull, 0u, 0u};
    }
    dim[t].clauses |= 1u << c;
    done |= 1u << c;
  }
  // a key's dimension ends where the shortest of its attributes does
  for (uint32_t t = 0; t < nd; ++t)
    for (uint32_t s = 0; s < O.nsrc; ++s) {
      if (O.src[s].fk != dim[t].fk) continue;
      if (O.src[s].width > 4 || dim[t].npay == HJ_PAY)
        return fail(MB_ERR_UNSUPPORTED, "mb_hash_join_grpby: more than %u attributes (or one over 4 bytes) on one key",
                    HJ_PAY);
      dim[t].n = std::min<uint64_t>(dim[t].n, O.src[s].dimsz ? O.src[s].dimsz : ~0ull);
      ++dim[t].npay;
      keyed |= 1u << s;
    }
  cudaStream_t st = as_stream(stream);
  MB_CHECK(scan_zero(nr_grp, out, nqual, st));
  if (nrows == 0) return MB_OK;
  ScanArgs A;
  memset(&A, 0, sizeof(A));
  if (nd == 0) return scan_rest(nrows, O, 0, 0, A, nr_grp, out, nqual, st);
  std::sort(dim, dim + nd, [](const Dim &a, const Dim &b) { return a.n < b.n; });
  uint64_t words = 0, most = 0;
  for (uint32_t t = 0; t < nd; ++t) {
    dim[t].n = std::min<uint64_t>(dim[t].n, 1ull << 32);  // keys have 32 bits
    words += round_up(dim[t].n, 128) / 32;
    most = std::max(most, dim[t].n);
  }
  Scratch sc(st);  // freed after the scan, in stream order
  uint32_t *bits;
  MB_CHECK(sc.get(&bits, words + HJ_MAXT));
  DimFilters F;
  memset(&F, 0, sizeof(F));
  F.any = bits + words;
  MB_CUDA(cudaMemsetAsync(F.any, 0, HJ_MAXT * 4, st));
  A.any = F.any;
  A.ntab = nd;
  for (uint32_t t = 0; t < nd; ++t) {
    F.d[t] = DimFilter{dim[t].n, bits, dim[t].clauses};
    Screen &S = A.s[A.ns++];
    S.col = dim[t].fk;
    S.bits = bits;
    S.nkeys = dim[t].n;
    S.vec = (reinterpret_cast<uintptr_t>(dim[t].fk) & 15) == 0;
    S.staged = ~0u;
    bits += round_up(dim[t].n, 128) / 32;
  }
  const unsigned gx = (unsigned)std::min<uint64_t>(ceil_div(most, 1024), (uint64_t)dev_info().sms * 2);
  dim_bits_kernel<<<dim3(gx ? gx : 1, nd), 256, 0, st>>>(O, F);
  MB_LAUNCH_CHECK("dim_bits_kernel");
  return scan_rest(nrows, O, done, keyed, A, nr_grp, out, nqual, st);
}
