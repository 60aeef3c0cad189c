// bitmap.cu - one-pass multi-bin bitmap-index creation (mb_bitmap_create).
//
// Reference: create_bin (bmpidx_create.cu:14-56) launching the multi-bin
// bmpcreate kernel (primitive.cuh:102-118): one thread per row, one
// __ballot_sync per (row-word, bin), lane 0 storing each word to HBM.
//
// Sorted, disjoint bins (an index level, a hierarchy of levels, one range) run
// in bitmap_planes_kernel (bitmap_planes.cuh): classes by table lookup, bit planes
// by transposition in registers, bitmaps as products of planes.  Overlapping,
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
#include "bitmap_planes.cuh"
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
// One level, or a hierarchy of two, over its own classes has its form; any
// other set of levels, and several levels over a wide domain, the general one.
static mb_status launch_planes(int mode, bool fine, const PlanePass &P) {
  const bool join = P.src->fk != nullptr;
  if (!fine || P.S.nlevels > (mode == BP_SEARCH ? 1u : 2u)) return join ? planes_any_join(mode, P) : planes_any_row(mode, P);
  if (mode == BP_SEARCH) return planes_search(P);
  if (join) return P.src->width <= 2 ? planes_join(P) : planes_wide(P);
  return P.src->width <= 4 ? planes_row(mode, P) : planes_wide(P);
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
      MB_CHECK(launch_planes(pmode, fine, PlanePass{PS, src, nrows, stride_words, st, LevelsJoinOut{nullptr, nullptr}}));
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
  return launch_planes(mode, fine, PlanePass{S, src, nrows, stride_words, st, LevelsJoinOut{dout, bad}});
}

extern "C" mb_status mb_bitmap_create_levels(const mb_src *src, uint64_t nrows, const mb_level *levels,
                                             uint32_t nlevels, uint64_t stride_words, void *stream) {
  return mb::bitmap_create_levels_join(src, nrows, levels, nlevels, stride_words, stream, nullptr, nullptr);
}
