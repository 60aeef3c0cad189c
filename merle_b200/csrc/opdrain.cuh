// opdrain.cuh - any op on a queue of rows, two rows a lane.
//
// The sources are loaded for both rows at once, foreign keys first and then
// every column / dimension value, keeping several independent gathers in flight
// per lane (op_eval, one row and one source at a time, waits for each).  Sources
// of up to 4 bytes.
#pragma once
#include "opeval.cuh"
#include "vbp.cuh"

namespace mb {

__device__ __forceinline__ uint32_t ld_w32(const void *p, uint64_t i, uint32_t w) {
  switch (w) {
  case 1: return __ldg(reinterpret_cast<const uint8_t *>(p) + i);
  case 2: return __ldg(reinterpret_cast<const uint16_t *>(p) + i);
  default: return __ldg(reinterpret_cast<const uint32_t *>(p) + i);
  }
}

// v[s] for a warp-uniform runtime s without dynamic register indexing.
__device__ __forceinline__ uint32_t pick(const uint32_t (&v)[MB_MAXSRC], uint32_t s) {
  uint32_t r = v[0];
#pragma unroll
  for (uint32_t i = 1; i < MB_MAXSRC; ++i) r = (s == i) ? v[i] : r;
  return r;
}

// Loads every needed source of one row: foreign keys first, then values.
// bad: bit s set if source s's key is out of its dimension.
__device__ __forceinline__ void load_row(const mb_op &O, uint32_t need, uint32_t row, uint32_t (&v)[MB_MAXSRC],
                                         uint32_t &bad) {
  uint32_t key[MB_MAXSRC];
#pragma unroll
  for (uint32_t s = 0; s < MB_MAXSRC; ++s) {
    key[s] = row;
    if (s < O.nsrc && ((need >> s) & 1u) && O.src[s].fk) key[s] = __ldg(O.src[s].fk + row);
  }
  bad = 0;
#pragma unroll
  for (uint32_t s = 0; s < MB_MAXSRC; ++s) {
    v[s] = 0;
    if (s < O.nsrc && ((need >> s) & 1u)) {
      const mb_src &S = O.src[s];
      if (S.fk && S.dimsz != 0 && key[s] >= S.dimsz) bad |= 1u << s;
      else v[s] = ld_w32(S.col, key[s], S.width);
    }
  }
}

// The op's filter over loaded values.
__device__ __forceinline__ bool filter_row(const mb_op &O, const uint32_t (&v)[MB_MAXSRC], uint32_t bad) {
  uint32_t t = 0;
  for (uint32_t c = 0; c < O.nclause; ++c) {
    bool any = false;
    const uint32_t len = O.clause_len[c];
    for (uint32_t k = 0; k < len; ++k, ++t) {
      const mb_term &tm = O.terms[t];
      const uint64_t x = pick(v, tm.src);
      any |= !((bad >> tm.src) & 1u) && x >= tm.lo && x < tm.hi;
    }
    if (!any) return false;
  }
  return true;
}

// The op over loaded values (the same semantics as op_eval in opeval.cuh).
__device__ __forceinline__ bool eval_row(const mb_op &O, const uint32_t (&v)[MB_MAXSRC], uint32_t bad, bool chk,
                                         uint32_t nr_grp, int64_t &value, uint32_t &group) {
  if (chk && !filter_row(O, v, bad)) return false;
  uint32_t g = 0;
  for (uint32_t k = 0; k < O.nkey; ++k) {
    const mb_key &kk = O.keys[k];
    if ((bad >> kk.src) & 1u) return false;
    uint32_t x = pick(v, kk.src);
    if (kk.xform == MB_X_DIV) x = x / kk.div;
    else if (kk.xform == MB_X_YEAR) x = date_to_year(x);
    g += kk.mul * (x - kk.base);
  }
  if (g >= nr_grp) return false;
  if (O.vkind == MB_V_ONE) {
    value = 1;
  } else {
    if ((bad >> O.va) & 1u) return false;
    const uint64_t a = pick(v, O.va);
    if (O.vkind == MB_V_COL) {
      value = (int64_t)a;
    } else {
      if ((bad >> O.vb) & 1u) return false;
      const uint64_t b = pick(v, O.vb);
      value = O.vkind == MB_V_MUL ? (int64_t)(a * b) : (int64_t)a - (int64_t)b;
    }
  }
  group = g;
  return true;
}

// Which queued rows the op's clauses are evaluated on: none (the entry is then the whole
// row id), those whose entry has bit 31 set.
enum { DR_NOCHK = 0, DR_FLAG = 1 };

// Runs the op over 64 queued rows (two per lane) and aggregates them.
template <int CHK, int GS>
__device__ __forceinline__ void drain64(const mb_op &O, const OpNeeds &N, const uint32_t *q, uint32_t nrows_avail,
                                        uint32_t nr_grp, const GrpCtx &G, int64_t &acc, uint32_t &cnt) {
  constexpr uint32_t ROW = CHK == DR_FLAG ? 0x7fffffffu : 0xffffffffu;
  const uint32_t lane = threadIdx.x & 31;
  const bool ok0 = lane < nrows_avail, ok1 = lane + 32 < nrows_avail;
  const uint32_t e0 = ok0 ? q[lane] : 0u, e1 = ok1 ? q[lane + 32] : 0u;
  const bool c0 = CHK == DR_FLAG && (e0 >> 31), c1 = CHK == DR_FLAG && (e1 >> 31);
  uint32_t v0[MB_MAXSRC], v1[MB_MAXSRC], bad0, bad1;
  load_row(O, ok0 ? (N.kv_mask | (c0 ? N.filt_mask : 0u)) : 0u, e0 & ROW, v0, bad0);
  load_row(O, ok1 ? (N.kv_mask | (c1 ? N.filt_mask : 0u)) : 0u, e1 & ROW, v1, bad1);
  int64_t val0 = 0, val1 = 0;
  uint32_t g0 = 0, g1 = 0;
  const bool k0 = ok0 && eval_row(O, v0, bad0, c0, nr_grp, val0, g0);
  const bool k1 = ok1 && eval_row(O, v1, bad1, c1, nr_grp, val1, g1);
  cnt += (k0 ? 1u : 0u) + (k1 ? 1u : 0u);
  aggregate<GS>(G, k0, g0, val0, acc);
  if (nrows_avail > 32) aggregate<GS>(G, k1, g1, val1, acc);
}

}  // namespace mb
