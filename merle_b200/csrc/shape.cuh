// shape.cuh - compiled forms of the query operator.
//
// A declarative op (mb_op) read as data costs several times its arithmetic:
// per row the evaluator walks sources, clauses and keys through uniform
// branches and selects its values by runtime index.  The engine's four query
// templates (s1op..s4op, ssb/lambdas.cuh:19-152) lower to four fixed forms;
// for these the op is compiled: which slots every row loads, which only
// uncertain rows load, the key transforms and the value are constants of the
// code, and the columns, bounds, divisors and multipliers are kernel
// parameters (constant-bank operands).  Any other op keeps the evaluators of
// opeval.cuh and fused.cu.
#pragma once
#include "batch.cuh"
#include "opeval.cuh"

namespace mb {

// Element bytes of each slot of a shape: the reference's ssb_schema widths
// (narrow) or 4-byte fact columns; the denormalised customer city (1) and part
// mfgr (2) either way.
constexpr uint8_t SHAPE_W[BNSHAPE][2][6] = {
    {{4, 4, 4, 4, 0, 0}, {2, 1, 1, 4, 0, 0}},  // date, discount, quantity, extendedprice
    {{4, 2, 4, 4, 0, 0}, {1, 2, 2, 4, 0, 0}},  // supplier city, mfgr, date, revenue
    {{4, 4, 1, 4, 0, 0}, {1, 2, 1, 4, 0, 0}},  // supplier city, date, customer city, revenue
    {{4, 4, 1, 2, 4, 4}, {1, 2, 1, 2, 4, 4}},  // supplier city, date, customer city, mfgr, revenue, supplycost
};

struct ShapeKey {
  uint32_t m, sh1, sh2;  // division magic (div_by_magic); year keys: unused
  uint32_t base, mul;
  uint32_t ident;        // 1: the key is the value itself
};

struct ShapeArgs {
  const void *col[6];
  const uint32_t *fk[6];  // the row's index into col, or NULL: the row itself (kernels with JOIN)
  uint32_t lo[6], hi[6];  // candidate-check bounds, inclusive
  ShapeKey key[4];        // by slot (key slots are 0..3)
  uint32_t ng;
  uint32_t fmask;         // filter slots to check (bit s); the others hold for every candidate row
};

// Host: the shape of an op (BSHAPES index, -1: none) with its arguments;
// *narrow selects the SHAPE_W row.  Sources through a foreign key (but `keyed`), widths of
// neither layout, clauses of several terms, ranges no value meets and keys
// sharing a source have no shape.
// sure: clauses (bit c) that every candidate row is known to satisfy.
// keyed: sources (bit s) whose foreign key lies inside its dimension on every
// candidate row; only those may be read through one.
int shape_of(const mb_op &O, uint32_t nr_grp, uint32_t sure, ShapeArgs *A, bool *narrow, uint32_t keyed = 0);

template <int W>
__device__ __forceinline__ uint32_t shape_load(const void *col, uint32_t row) {
  if (W == 1) return __ldg(reinterpret_cast<const uint8_t *>(col) + row);
  if (W == 2) return __ldg(reinterpret_cast<const uint16_t *>(col) + row);
  return __ldg(reinterpret_cast<const uint32_t *>(col) + row);
}

template <int SH, bool NARROW, int S>
struct ShapeSlot {
  static constexpr BShape sh = BSHAPES[SH];
  static constexpr bool used = (uint32_t)S < sh.ns;
  static constexpr bool kv = used && ((sh.kv >> S) & 1u);      // every row
  static constexpr bool filt = used && ((sh.filt >> S) & 1u);  // re-checked for uncertain rows
  static constexpr bool key = used && ((sh.keym >> S) & 1u);
  static constexpr bool year = used && ((sh.yearm >> S) & 1u);
  static constexpr int w = SHAPE_W[SH][NARROW ? 1 : 0][S];
};

// One row's slots, 0..5.  JOIN: slots may be read through a foreign key.
template <int SH, bool NARROW, bool JOIN>
struct ShapeVals {
  static constexpr BShape sh = BSHAPES[SH];
  uint32_t v[6];

  // Every row's slots that a filter reads too (rows of inactive lanes are row
  // 0, which exists).
  __device__ __forceinline__ void load_now(const ShapeArgs &A, uint32_t row) {
    n1<0>(A, row), n1<1>(A, row), n1<2>(A, row), n1<3>(A, row), n1<4>(A, row), n1<5>(A, row);
  }
  // Every row's other slots, if `on`.
  __device__ __forceinline__ void load_late(const ShapeArgs &A, uint32_t row, bool on) {
    l1<0>(A, row, on), l1<1>(A, row, on), l1<2>(A, row, on), l1<3>(A, row, on), l1<4>(A, row, on), l1<5>(A, row, on);
  }
  // The slots only the check of an uncertain row reads.
  __device__ __forceinline__ void load_filt(const ShapeArgs &A, uint32_t row, bool unc) {
    f1<0>(A, row, unc), f1<1>(A, row, unc), f1<2>(A, row, unc), f1<3>(A, row, unc), f1<4>(A, row, unc),
        f1<5>(A, row, unc);
  }
  __device__ __forceinline__ bool check(const ShapeArgs &A) const {
    return c1<0>(A) && c1<1>(A) && c1<2>(A) && c1<3>(A) && c1<4>(A) && c1<5>(A);
  }
  __device__ __forceinline__ uint32_t group(const ShapeArgs &A) const {
    return k1<0>(A) + k1<1>(A) + k1<2>(A) + k1<3>(A);
  }
  __device__ __forceinline__ int64_t value() const {
    if (sh.vk == MB_V_COL) return (int64_t)v[sh.va];
    if (sh.vk == MB_V_MUL) return (int64_t)((uint64_t)v[sh.va] * v[sh.vb]);
    return (int64_t)v[sh.va] - (int64_t)v[sh.vb];
  }

 private:
  template <int S>
  __device__ __forceinline__ uint32_t at(const ShapeArgs &A, uint32_t row) const {
    return JOIN && A.fk[S] ? __ldg(A.fk[S] + row) : row;
  }
  template <int S>
  __device__ __forceinline__ void n1(const ShapeArgs &A, uint32_t row) {
    using T = ShapeSlot<SH, NARROW, S>;
    if (T::kv && T::filt) v[S] = shape_load<T::w>(A.col[S], at<S>(A, row));
  }
  template <int S>
  __device__ __forceinline__ void l1(const ShapeArgs &A, uint32_t row, bool on) {
    using T = ShapeSlot<SH, NARROW, S>;
    if (T::kv && !T::filt && on) v[S] = shape_load<T::w>(A.col[S], at<S>(A, row));
  }
  template <int S>
  __device__ __forceinline__ void f1(const ShapeArgs &A, uint32_t row, bool unc) {
    using T = ShapeSlot<SH, NARROW, S>;
    if (T::filt && !T::kv && ((A.fmask >> S) & 1u) && unc) v[S] = shape_load<T::w>(A.col[S], at<S>(A, row));
  }
  template <int S>
  __device__ __forceinline__ bool c1(const ShapeArgs &A) const {
    using T = ShapeSlot<SH, NARROW, S>;
    return !T::filt || !((A.fmask >> S) & 1u) || v[S] - A.lo[S] <= A.hi[S] - A.lo[S];
  }
  template <int S>
  __device__ __forceinline__ uint32_t k1(const ShapeArgs &A) const {
    using T = ShapeSlot<SH, NARROW, S>;
    if (!T::key) return 0;
    const ShapeKey &K = A.key[S];
    uint32_t x = v[S];
    if (T::year) x = date_to_year(x);
    else if (!K.ident) x = div_by_magic(x, K.m, K.sh1, K.sh2);  // uniform branch
    return K.mul * (x - K.base);
  }
};

// The op on R rows per lane (32 R queued rows, n of them live; entry = row |
// uncertain << 31), with the aggregation.  All loads of the R rows issue
// before any value is used; with `late`, an uncertain row's value columns that
// no filter reads are loaded only once it has passed its check, which saves
// their sectors where selected rows are sparse and costs a second memory round
// trip where they are dense.
template <int SH, bool NARROW, bool CHK, int GS, int R, bool JOIN = false>
__device__ __forceinline__ void shape_rows(const ShapeArgs &A, const uint32_t *q, uint32_t n, bool late,
                                           const GrpCtx &G, int64_t &acc, uint32_t &cnt) {
  const uint32_t lane = threadIdx.x & 31;
  ShapeVals<SH, NARROW, JOIN> V[R];
  bool act[R], unc[R];
  uint32_t row[R];
#pragma unroll
  for (int j = 0; j < R; ++j) {
    const uint32_t i = lane + 32 * j;
    act[j] = i < n;
    // an inactive lane loads row 0, which exists; through a key, a live row (n > 0),
    // whose key is known to be inside its dimension
    const uint32_t e = act[j] ? q[i] : (JOIN ? q[0] : 0u);
    row[j] = CHK ? e & 0x7fffffffu : e;
    unc[j] = CHK && (e >> 31);
    V[j].load_now(A, row[j]);
    V[j].load_late(A, row[j], !(CHK && late && unc[j]));
  }
  if (CHK) {
    bool any = false;
#pragma unroll
    for (int j = 0; j < R; ++j) any = any || unc[j];
    if (__any_sync(0xffffffffu, any)) {
#pragma unroll
      for (int j = 0; j < R; ++j) V[j].load_filt(A, row[j], unc[j]);
#pragma unroll
      for (int j = 0; j < R; ++j) act[j] = act[j] && (!unc[j] || V[j].check(A));
      if (late) {
#pragma unroll
        for (int j = 0; j < R; ++j)
          if (act[j] && unc[j]) V[j].load_late(A, row[j], true);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < R; ++j) {
    bool keep = act[j];
    const uint32_t g = GS == GS_SCALAR ? 0u : V[j].group(A);
    if (GS != GS_SCALAR) keep = keep && g < A.ng;
    if (keep) {
      const int64_t val = V[j].value();
      ++cnt;
      if (GS == GS_SCALAR) acc += val;
      else if (GS == GS_SHARED) shared_add64(&G.lo[g], &G.hi[g], (uint64_t)val);
      else atomicAdd(&G.gout[g], (unsigned long long)val);
    }
  }
}

}  // namespace mb
