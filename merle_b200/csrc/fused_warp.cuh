// fused_warp.cuh - the warp-independent fused kernel
// (program -> compaction -> op -> group-by), over the drains of fused.cu (any
// op) and shape.cuh (compiled ops).
//
// Each warp walks tiles of 32 * V bitmap words on its own (no block barrier
// until the final flush): load the chain's words (V consecutive ones a lane)
// compact the selected rows into its queue, run the op on full batches of 64.
//
// What bounds it: the bitmap stream for selective queries (48-60 % of the
// measured copy rate at 120M-600M rows), the outstanding sparse sector reads of
// the op's columns at 1-10 % selected rows (DRAM fetches 64 bytes per 32-byte
// sector read, 4.3 TB/s), instruction issue above that.  Measured at 600M rows,
// 4-byte columns, 64 queries of selectivity 1e-6 to 0.5, one launch each: 102.2
// ms with the op interpreted and 2 words a lane, 43.8 ms compiled, 41.1 ms with 4
// words a lane; at 46 % selected rows 11.9 -> 2.0 ms.  Bounding the compiled kernels to 3
// CTAs an SM (85 registers; they take 56-60, so that 4 fit) beats bounding them to 4 (64, with
// spills) by 4 %.
#pragma once
#include "shape.cuh"
#include "vbp.cuh"

namespace mb {

constexpr uint32_t FW_THREADS = 256;
constexpr uint32_t FW_QCAP = 32 * 32 + 64;  // one 32-word chunk + fewer than 64 pending rows
constexpr size_t FW_STATIC = 64 * 8;        // shared memory of the final reduction
// Warps of a CTA, and its dynamic shared memory beside grp_bytes of group table.
inline uint32_t fw_warps(uint32_t asked) { return asked == 0 || asked > FW_THREADS / 32 ? FW_THREADS / 32 : asked; }
inline size_t fw_smem(size_t grp_bytes, uint32_t warps) {
  return ((grp_bytes + 15) & ~(size_t)15) + (size_t)fw_warps(warps) * FW_QCAP * 4;
}
// Selected rows of a 1,024-row chunk below which an uncertain row's value
// columns wait for its check (shape_rows): below about one row in eight most
// rows have a 32-byte sector to themselves, so a failing row's sectors are
// saved (120M rows, 0.8 % candidates of which 1 in 40 pass: 79 -> 42 us); above,
// the sectors are read for their other rows anyway.
constexpr uint32_t FW_LATE = 128;

// Words [w0, w0 + V) of a bitmap: one aligned vector load (w0 a multiple of V).
template <int V>
__device__ __forceinline__ void fw_load(const uint32_t *p, uint64_t w0, uint32_t (&x)[V]) {
  if (V == 4) {
    const uint4 t = __ldcs(reinterpret_cast<const uint4 *>(p + w0));
    x[0] = t.x, x[1 % V] = t.y, x[2 % V] = t.z, x[3 % V] = t.w;
  } else if (V == 2) {
    const uint2 t = __ldcs(reinterpret_cast<const uint2 *>(p + w0));
    x[0] = t.x, x[1 % V] = t.y;
  } else {
    x[0] = __ldcs(p + w0);
  }
}

// The conjunctive chain on words w0 + lane * V + k: p the selected rows, u the
// uncertain ones.  The chain's bitmaps are loaded in batches of independent
// loads; a lane whose finished conjuncts (most selective first) left no row in
// its words skips the later batches, so 32-byte sectors without a candidate
// are not fetched.
template <int V, bool CHK>
__device__ __forceinline__ void fw_chain(const DevPrg &P, uint64_t w0, uint32_t (&p)[V], uint32_t (&u)[V]) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t wl = w0 + lane * V;
  const bool full = wl + V <= P.nwords;
  uint32_t acc[V], cur[V], ce[V], unc[V];
#pragma unroll
  for (int k = 0; k < V; ++k) acc[k] = 0xffffffffu, cur[k] = ce[k] = unc[k] = 0;
  const uint32_t nb = P.ncnf;
  constexpr int B = V == 4 ? 4 : 8;  // bitmaps loaded together
  for (uint32_t b0 = 0; b0 < nb; b0 += B) {
    uint32_t x[B][V];
    uint32_t live = 0;
#pragma unroll
    for (int k = 0; k < V; ++k) live |= acc[k];
#pragma unroll
    for (int j = 0; j < B; ++j) {
#pragma unroll
      for (int k = 0; k < V; ++k) x[j][k] = 0;
      if (b0 + j < nb && live) {
        const uint32_t *src = P.cnf_ptr[b0 + j];
        if (full) {
          fw_load<V>(src, wl, x[j]);
        } else {
#pragma unroll
          for (int k = 0; k < V; ++k)
            if (wl + k < P.nwords) x[j][k] = __ldcs(src + wl + k);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < B; ++j) {
      if (b0 + j >= nb) break;
      const uint32_t f = P.cnf_flag[b0 + j];
#pragma unroll
      for (int k = 0; k < V; ++k) {
        cur[k] |= x[j][k];
        if (CHK && (f & CNF_EDGE)) ce[k] |= x[j][k];
      }
      if (f & CNF_END) {
#pragma unroll
        for (int k = 0; k < V; ++k) {
          acc[k] &= (f & CNF_NEG) ? ~cur[k] : cur[k];
          if (CHK && !(f & CNF_NEG)) unc[k] |= ce[k];
          cur[k] = ce[k] = 0;
        }
      }
    }
  }
  const uint32_t tail = (uint32_t)(P.nrows & 31u);
  const bool edge = w0 + 32 * V >= P.nwords;  // the table's last tile
#pragma unroll
  for (int k = 0; k < V; ++k) {
    p[k] = acc[k];
    if (edge) {
      const uint64_t w = wl + k;
      if (w >= P.nwords) p[k] = 0;
      else if (tail && w + 1 == P.nwords) p[k] &= (1u << tail) - 1u;
    }
    u[k] = CHK ? (unc[k] & p[k]) : 0u;
  }
}

// Appends the rows set in m (bit b: row rowbase + b; bit b of uw: uncertain) of
// every lane to the warp queue (qn rows pending), then drains full batches of
// 64 rows.  Queue entries are row ids with the uncertain flag in bit 31.
template <bool CHK, class DR>
__device__ __forceinline__ void fw_compact(const DR &dr, uint32_t *queue, uint32_t &qn, uint32_t rowbase, uint32_t m,
                                           uint32_t uw, const GrpCtx &G, int64_t &acc, uint32_t &cnt) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t pc = __popc(m);
  uint32_t incl = pc;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= (uint32_t)d) incl += y;
  }
  const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
  uint32_t *w = queue + (qn + incl - pc);
  while (m) {
    const uint32_t b = __ffs(m) - 1;
    m &= m - 1;
    uint32_t e = rowbase + b;
    if (CHK) e |= ((uw >> b) & 1u) << 31;
    *w++ = e;
  }
  qn += total;
  __syncwarp();
  while (qn >= 64) {  // drain from the end: the queue's order is irrelevant
    qn -= 64;
    dr.drain(queue + qn, 64, total, G, acc, cnt);
  }
  __syncwarp();
}

// CNF: the program is a conjunctive chain (fw_chain); else its instructions run
// one by one (vbp_eval) on the lane's words.  (A program with an OR and checked
// edges over 60M rows, 256 groups: 236 us in the kernel whose drain walks the op
// source by source, 163 us here with each row's loads issued together.)
template <int V, bool CHK, int GS, bool CNF, class DR>
__device__ __forceinline__ void fused_warp_body(const DevPrg &P, const DR &dr, uint32_t nr_grp, uint32_t hcap,
                                                unsigned long long *out, unsigned long long *nqual, uint8_t *smem) {
  __shared__ uint64_t red[FW_STATIC / 8];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const size_t gbytes = (grp_smem_bytes(GS, nr_grp, hcap) + 15) & ~(size_t)15;
  const GrpCtx G = grp_init<GS>(smem, nr_grp, hcap, out);
  uint32_t *queue = reinterpret_cast<uint32_t *>(smem + gbytes) + (size_t)warp * FW_QCAP;
  __syncthreads();
  int64_t acc = 0;
  uint32_t cnt = 0, qn = 0;
  constexpr uint32_t TW = 32 * V;
  const uint64_t ntiles = (P.nwords + TW - 1) / TW;
  for (uint64_t t = (uint64_t)blockIdx.x * nw + warp; t < ntiles; t += (uint64_t)gridDim.x * nw) {
    uint32_t p[V], u[V];
    if (CNF) fw_chain<V, CHK>(P, t * TW, p, u);
    else vbp_eval<V, CHK>(P, t * TW + lane * V, p, u);
    const uint32_t rb = (uint32_t)((t * TW + lane * V) * 32);
#pragma unroll
    for (int k = 0; k < V; ++k)
      if (__any_sync(0xffffffffu, p[k] != 0))
        fw_compact<CHK>(dr, queue, qn, rb + 32 * k, p[k], u[k], G, acc, cnt);
  }
  if (qn) dr.drain(queue, qn, 0, G, acc, cnt);
  __syncthreads();
  grp_flush<GS>(G, nr_grp, acc, cnt, nqual, red);
}

// A compiled op (shape.cuh) as the kernel's drain: n queued rows, of a 1,024-row chunk
// with `rows` selected ones.
template <int SH, bool NARROW, bool CHK, int GS>
struct ShapeDrain {
  const ShapeArgs &A;
  __device__ __forceinline__ void drain(const uint32_t *q, uint32_t n, uint32_t rows, const GrpCtx &G, int64_t &acc,
                                        uint32_t &cnt) const {
    shape_rows<SH, NARROW, CHK, GS, 2>(A, q, n, rows < FW_LATE, G, acc, cnt);
  }
};

template <int V, bool CHK, int GS, int SH, bool NARROW>
__global__ void __launch_bounds__(FW_THREADS, 3)
fused_shape_kernel(const __grid_constant__ DevPrg P, const __grid_constant__ ShapeArgs A, uint32_t nr_grp,
                   unsigned long long *__restrict__ out, unsigned long long *__restrict__ nqual) {
  extern __shared__ __align__(128) uint8_t smem[];
  fused_warp_body<V, CHK, GS, true>(P, ShapeDrain<SH, NARROW, CHK, GS>{A}, nr_grp, 0, out, nqual, smem);
}

// Launch of a warp-independent kernel of `warps` warps: persistent grid.
template <typename K, typename... Args>
mb_status fw_launch(K kern, uint32_t V, uint64_t nwords, size_t gbytes, uint32_t warps, uint32_t cps, cudaStream_t st,
                    Args &&...args) {
  const size_t smem = fw_smem(gbytes, warps);
  const DevInfo &di = dev_info();
  if (smem > (size_t)di.max_smem_optin) return fail(MB_ERR_INVALID, "fused: %zu bytes of shared memory", smem);
  MB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int occ = 0;
  MB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, (int)(warps * 32), smem));
  if (occ < 1) return fail(MB_ERR_INVALID, "fused: kernel does not fit on an SM");
  if (cps && (int)cps < occ) occ = (int)cps;
  const uint64_t ntiles = (nwords + 32 * V - 1) / (32 * V);
  uint64_t grid = (uint64_t)di.sms * occ;
  const uint64_t need = (ntiles + warps - 1) / warps;
  if (grid > need) grid = need ? need : 1;
  kern<<<(unsigned)grid, warps * 32, smem, st>>>(std::forward<Args>(args)...);
  MB_LAUNCH_CHECK("fused warp kernel");
  return MB_OK;
}

// The kernels of one shape (fused_shape1.cu .. fused_shape4.cu).
struct ShapeLaunch {
  uint32_t nr_grp, V, warps, cps;
  int gs;
  bool narrow;
  unsigned long long *out, *nqual;
  cudaStream_t st;
};
mb_status fused_shape1(const DevPrg &P, const ShapeArgs &A, const ShapeLaunch &L);
mb_status fused_shape2(const DevPrg &P, const ShapeArgs &A, const ShapeLaunch &L);
mb_status fused_shape3(const DevPrg &P, const ShapeArgs &A, const ShapeLaunch &L);
mb_status fused_shape4(const DevPrg &P, const ShapeArgs &A, const ShapeLaunch &L);

template <int SH, int V, bool CHK, int GS>
mb_status fused_shape_width(const DevPrg &P, const ShapeArgs &A, const ShapeLaunch &L) {
  const size_t gb = grp_smem_bytes(GS, L.nr_grp, 0);
  if (L.narrow)
    return fw_launch(fused_shape_kernel<V, CHK, GS, SH, true>, V, P.nwords, gb, L.warps, L.cps, L.st, P, A, L.nr_grp,
                     L.out, L.nqual);
  return fw_launch(fused_shape_kernel<V, CHK, GS, SH, false>, V, P.nwords, gb, L.warps, L.cps, L.st, P, A, L.nr_grp,
                   L.out, L.nqual);
}

// Shape 0 (SUM of a product) has one group; the others at least two (shape_of's
// callers see to it).
template <int SH, int V, bool CHK>
mb_status fused_shape_gs(const DevPrg &P, const ShapeArgs &A, const ShapeLaunch &L) {
  if constexpr (BSHAPES[SH].keym == 0) {
    return fused_shape_width<SH, V, CHK, GS_SCALAR>(P, A, L);
  } else {
    return L.gs == GS_SHARED ? fused_shape_width<SH, V, CHK, GS_SHARED>(P, A, L)
                             : fused_shape_width<SH, V, CHK, GS_GLOBAL>(P, A, L);
  }
}

template <int SH>
mb_status fused_shape_launch(const DevPrg &P, const ShapeArgs &A, const ShapeLaunch &L) {
  if (P.chk)
    return L.V == 4   ? fused_shape_gs<SH, 4, true>(P, A, L)
           : L.V == 2 ? fused_shape_gs<SH, 2, true>(P, A, L)
                      : fused_shape_gs<SH, 1, true>(P, A, L);
  return L.V == 4   ? fused_shape_gs<SH, 4, false>(P, A, L)
         : L.V == 2 ? fused_shape_gs<SH, 2, false>(P, A, L)
                    : fused_shape_gs<SH, 1, false>(P, A, L);
}

}  // namespace mb
