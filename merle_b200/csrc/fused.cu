// fused.cu - the fused kernels' evaluators of any op, and the TMA-staged kernel: program -> compaction -> op ->
// group-by, with every operand bitmap of a tile staged in shared memory.
//
// Reference: vprg_grpby (primitive.cuh:340-445).  The reference reads each
// operand word with a dependent chain of __ldcs loads per thread; here one
// thread per CTA streams the tile of EVERY bitmap of the program into shared
// memory with 1-D TMA bulk copies (cp.async.bulk, mbarrier completion, two
// stages), so HBM reads run ahead of the compute without occupying warps:
//
//   stage s ready -> phase A: all warps evaluate the program from shared
//   memory into a per-CTA result tile -> __syncthreads -> thread 0 refills
//   stage s with the tile after next -> phase B: each warp compacts 32-word
//   chunks of the result tile into its own row queue, while the other stage
//   streams in.
//
// A warp runs the op only on full 64-row batches of its queue (two rows per
// lane), carrying fewer than 64 rows over to the next chunk or tile, so lanes
// stay busy at any selectivity; sums commute, so the queue is drained from
// its end.  The op's sources are loaded for both rows at once, foreign keys
// first and then every column / dimension value, keeping several independent
// gathers in flight per lane; filter-only sources are read only for uncertain
// rows (chk), as the reference's functors do.
//
// Bounded waits: every mbarrier wait gives up after 2^20 tries, records the
// block in the device error word and leaves the loop block-uniformly.
#include <string.h>
#include "common.cuh"
#include "opdrain.cuh"
#include "opeval.cuh"
#include "tma.cuh"
#include "vbp.cuh"
#include "fused_warp.cuh"

namespace mb {

constexpr uint32_t FT_THREADS = 256;
constexpr uint32_t FT_WARPS = FT_THREADS / 32;

OpNeeds op_needs(const mb_op &O) {
  OpNeeds n{0, 0, false};
  for (uint32_t k = 0; k < O.nkey; ++k) n.kv_mask |= 1u << O.keys[k].src;
  if (O.vkind != MB_V_ONE) n.kv_mask |= 1u << O.va;
  if (O.vkind == MB_V_MUL || O.vkind == MB_V_SUB) n.kv_mask |= 1u << O.vb;
  uint32_t nt = 0;
  for (uint32_t c = 0; c < O.nclause; ++c) nt += O.clause_len[c];
  for (uint32_t t = 0; t < nt; ++t) n.filt_mask |= 1u << O.terms[t].src;
  for (uint32_t s = 0; s < O.nsrc; ++s)
    if ((n.kv_mask >> s & 1u) && O.src[s].fk && n.kv_mask != 1u << s) n.behind_key = true;
  return n;
}

bool op_reads_wide(const mb_op &O) {
  const OpNeeds n = op_needs(O);
  for (uint32_t s = 0; s < O.nsrc; ++s)
    if (((n.kv_mask | n.filt_mask) >> s & 1u) && O.src[s].width > 4) return true;
  return false;
}

// Word lw of bitmap b in the staged tile; words past the bulk-copied part of
// the last tile come from global memory, words past the bitmap are 0.
struct TileView {
  const uint32_t *stage;  // nb x T words
  uint32_t T, copied, valid;
  uint64_t w0;
};

// The stage holds all T words of every bitmap (the last tile's tail words are
// completed by the threads before phase A), so reads need no bounds checks.
__device__ __forceinline__ uint32_t tword(const DevPrg &P, const TileView &tv, uint32_t b, uint32_t lw) {
  (void)P;
  return tv.stage[b * tv.T + lw];
}

// The conjunctive form on word lw: p = AND of (negated) operand ORs,
// u = OR of the positive operands' edge bins, masked by p.
template <bool CHK>
__device__ __forceinline__ void cnf_eval(const DevPrg &P, const TileView &tv, uint32_t lw, uint32_t &p,
                                         uint32_t &u) {
  uint32_t acc = 0xffffffffu, unc = 0;
  for (uint32_t c = 0; c < MB_MAXCOLS; ++c) {
    if (!((P.cmask >> c) & 1u)) continue;
    const uint32_t first = P.off[c], nm = P.nmid[c], ne = P.nedge[c];
    uint32_t cm = 0, ce = 0;
    for (uint32_t b = 0; b < nm; ++b) cm |= tv.stage[(first + b) * tv.T + lw];
    for (uint32_t b = 0; b < ne; ++b) ce |= tv.stage[(first + nm + b) * tv.T + lw];
    if ((P.neg >> c) & 1u) {
      acc &= ~(cm | ce);
    } else {
      acc &= cm | ce;
      if (CHK) unc |= ce;
    }
  }
  const uint64_t w = tv.w0 + lw;
  uint32_t m = w < P.nwords ? 0xffffffffu : 0u;
  const uint32_t tail = (uint32_t)(P.nrows & 31u);
  if (tail && w + 1 == P.nwords) m = (1u << tail) - 1u;
  p = acc & m;
  u = CHK ? (unc & p) : 0u;
}

__device__ __forceinline__ void or_bins_s(const DevPrg &P, const TileView &tv, int first, int cnt, uint32_t lw,
                                          uint32_t &acc) {
  acc = 0;
  for (int b = 0; b < cnt; ++b) acc |= tword(P, tv, first + b, lw);
}

// The program on words lw[k] of the staged tile (same algebra as vbp_eval).
template <int V, bool CHK>
__device__ __forceinline__ void vbp_eval_staged(const DevPrg &P, const TileView &tv, const uint32_t (&lw)[V],
                                                uint32_t (&p)[V], uint32_t (&u)[V]) {
  Regs<V> R, U;
#pragma unroll
  for (int i = 0; i < MB_NREGS; ++i)
#pragma unroll
    for (int k = 0; k < V; ++k) R.r[i][k] = U.r[i][k] = 0;
  for (uint32_t i = 0; i < P.ninstr; ++i) {
    const mb_instr in = P.ins[i];
    uint32_t dp[V], du[V], sp[V], su[V];
    rget(R, in.dstreg, dp);
    if (CHK) rget(U, in.dstreg, du);
    switch (in.opcode) {
    case MB_AND:
      rget(R, in.src1, sp);
      if (CHK) rget(U, in.src1, su);
#pragma unroll
      for (int k = 0; k < V; ++k) {
        dp[k] &= sp[k];
        if (CHK) du[k] = (du[k] | su[k]) & dp[k];
      }
      break;
    case MB_OR:
      rget(R, in.src1, sp);
      if (CHK) rget(U, in.src1, su);
#pragma unroll
      for (int k = 0; k < V; ++k) {
        if (CHK) du[k] = (du[k] & ~(sp[k] & ~su[k])) | (su[k] & ~dp[k]);
        dp[k] |= sp[k];
      }
      break;
    case MB_NOT:
      rget(R, in.src1, sp);
#pragma unroll
      for (int k = 0; k < V; ++k) dp[k] = ~sp[k];
      if (CHK && in.dstreg != in.src1) rget(U, in.src1, du);
      break;
    case MB_ANDM:
    case MB_ORM: {
      const int c = in.src1;
#pragma unroll
      for (int k = 0; k < V; ++k) {
        uint32_t cm, ce;
        or_bins_s(P, tv, P.off[c], P.nmid[c], lw[k], cm);
        or_bins_s(P, tv, P.off[c] + P.nmid[c], P.nedge[c], lw[k], ce);
        if (in.opcode == MB_ANDM) {
          if (CHK) {
            const uint32_t np = dp[k] & (ce | cm);
            du[k] = dp[k] ? ((du[k] | ce) & np) : du[k];  // primitive.cuh:292
            dp[k] = np;
          } else {
            dp[k] &= (cm | ce);
          }
        } else {
          if (CHK) du[k] = (du[k] & ~cm) | (ce & ~dp[k]);
          dp[k] |= ce | cm;
        }
      }
      break;
    }
    default: break;
    }
    rset(R, in.dstreg, dp);
    if (CHK) rset(U, in.dstreg, du);
  }
  const uint32_t tail = (uint32_t)(P.nrows & 31u);
#pragma unroll
  for (int k = 0; k < V; ++k) {
    const uint64_t w = tv.w0 + lw[k];
    uint32_t m = w < P.nwords ? 0xffffffffu : 0u;
    if (tail && w + 1 == P.nwords) m = (1u << tail) - 1u;
    p[k] = R.r[0][k] & m;
    u[k] = CHK ? (U.r[0][k] & m) : 0u;
  }
}

constexpr uint32_t FT_QCAP = 32 * 32 + 64;  // one 32-word chunk + fewer than 64 pending rows

// Appends the set rows of one 32-word chunk (word w0 + lane of each lane,
// possible bits m, uncertain bits uw) to the warp queue (qn rows pending,
// warp-uniform), then drains full 64-row batches.  Queue entries are row ids
// with the uncertain flag in bit 31 (rows < 2^31).
template <bool CHK, int GS>
__device__ __forceinline__ void compact_chunk(const mb_op &O, const OpNeeds &N, uint32_t *queue, uint32_t &qn,
                                              uint64_t w0, uint32_t m, uint32_t uw, uint32_t nr_grp,
                                              const GrpCtx &G, int64_t &acc, uint32_t &cnt) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t pc = __popc(m);
  uint32_t incl = pc;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= (uint32_t)d) incl += y;
  }
  const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
  if (total == 0) return;
  uint32_t off = qn + incl - pc;
  const uint32_t rowbase = (uint32_t)((w0 + lane) * 32);
  while (m) {
    const uint32_t b = __ffs(m) - 1;
    m &= m - 1;
    uint32_t e = rowbase + b;
    if (CHK && ((uw >> b) & 1u)) e |= 0x80000000u;
    queue[off++] = e;
  }
  qn += total;
  __syncwarp();
  while (qn >= 64) {  // drain from the end: the queue's order is irrelevant
    qn -= 64;
    drain64<CHK ? DR_FLAG : DR_NOCHK, GS>(O, N, queue + qn, 64, nr_grp, G, acc, cnt);
  }
  __syncwarp();
}

// Any op as the warp-independent kernel's drain (fused_warp.cuh): n queued rows, of a
// 1,024-row chunk with `rows` selected ones.  Sparse rows wait for their sectors, and
// drain64 has two rows' loads in flight a lane; dense ones share sectors, and the
// instructions count: op_eval needs fewer, a row a lane.  120M rows without checks, 256
// groups, two words a lane: an OR over 30 % of the rows 328 -> 230 us, a chain over a third
// 488 -> 344, an OR over 0.5 % 89 -> 88.  From 16 rows a chunk on; 32 and 48 are slower by up to
// 1.2 and 1.4 times where the chunks of a table lie on both sides (an OR over 6 %, 240M
// rows: 190 us at 16, 228, 273).
// Several sources with one behind a foreign key keep drain64: op_eval would wait for the
// key, its dimension and each of the others in turn (120M rows, nearly all selected, a dimension key, a
// date and a value: 3,029 us, 3,475).
// With candidate checks drain64 alone: both in one kernel make the sparse cases 3 to 20 %
// slower, and op_eval on rows that fail their checks takes up to 1.46 times as long.
constexpr uint32_t ANY_DENSE = 16;
template <bool CHK, int GS, bool DENSE>
struct AnyDrain {
  const mb_op &O;
  OpNeeds N;
  uint32_t nr_grp;
  __device__ __forceinline__ void drain(const uint32_t *q, uint32_t n, uint32_t rows, const GrpCtx &G, int64_t &acc,
                                        uint32_t &cnt) const {
    if (!DENSE || rows < ANY_DENSE) {
      drain64<CHK ? DR_FLAG : DR_NOCHK, GS>(O, N, q, n, nr_grp, G, acc, cnt);
      return;
    }
#pragma unroll 1
    for (uint32_t i = threadIdx.x & 31; i < 64; i += 32) {
      int64_t val = 0;
      uint32_t grp = 0;
      const bool kept = i < n && op_eval(O, q[i], false, nr_grp, val, grp);
      cnt += kept ? 1u : 0u;
      aggregate<GS>(G, kept, grp, val, acc);
    }
  }
};

// DENSE: dense rows a row a lane (AnyDrain).  Such kernels name the CTAs an SM (64 registers a
// thread): left alone, the compiler takes 48 for most and spills, sparse programs up to
// 12 % slower (24M rows, an OR over 0.5 %: 21.8 -> 19.4 us).
template <int V, bool CHK, int GS, bool CNF, bool DENSE>
__global__ void __launch_bounds__(FW_THREADS, DENSE ? 4 : 0)
fused_warp_kernel(const __grid_constant__ DevPrg P, const __grid_constant__ mb_op O, OpNeeds N, uint32_t nr_grp,
                  uint32_t hcap, unsigned long long *__restrict__ out, unsigned long long *__restrict__ nqual) {
  extern __shared__ __align__(128) uint8_t smem[];
  fused_warp_body<V, CHK, GS, CNF>(P, AnyDrain<CHK, GS, DENSE>{O, N, nr_grp}, nr_grp, hcap, out, nqual, smem);
}

// T = FT_THREADS * V words per CTA tile.
template <bool CHK, int GS>
__global__ void __launch_bounds__(FT_THREADS, 2)
fused_tma_kernel(const __grid_constant__ DevPrg P, const __grid_constant__ mb_op O, OpNeeds N, uint32_t nb,
                 uint32_t T, uint32_t nr_grp, uint32_t hcap, unsigned long long *__restrict__ out,
                 unsigned long long *__restrict__ nqual, uint32_t *errw) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ uint64_t red[64];
  __shared__ __align__(8) uint64_t bars[2];
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const size_t stage_words = (size_t)nb * T;
  uint32_t *stages = reinterpret_cast<uint32_t *>(smem);
  uint32_t *ptile = stages + 2 * stage_words;      // the program's possible words of the tile
  uint32_t *utile = ptile + T;                      // ... and uncertain words (CHK)
  uint8_t *gsm = reinterpret_cast<uint8_t *>(utile + (CHK ? T : 0));
  const size_t gbytes = (grp_smem_bytes(GS, nr_grp, hcap) + 15) & ~(size_t)15;
  GrpCtx G = grp_init<GS>(gsm, nr_grp, hcap, out);
  uint32_t *queue = reinterpret_cast<uint32_t *>(gsm + gbytes) + (size_t)warp * FT_QCAP;
  if (tid == 0) {
    mbar_init(&bars[0], 1);
    mbar_init(&bars[1], 1);
    fence_mbar_init();
  }
  __syncthreads();

  const uint64_t ntiles = (P.nwords + T - 1) / T;
  auto valid_words = [&](uint64_t t) -> uint32_t {
    const uint64_t r = P.nwords - t * T;
    return (uint32_t)(r < T ? r : T);
  };
  auto issue = [&](uint64_t t, int s) {
    const uint32_t cw = valid_words(t) & ~3u;  // whole 16-byte chunks
    fence_proxy_async_smem();
    mbar_arrive_expect_tx(&bars[s], cw * 4 * nb);
    if (cw)
      for (uint32_t b = 0; b < nb; ++b)
        bulk_g2s(stages + s * stage_words + (size_t)b * T, P.ptr[b] + t * T, cw * 4, &bars[s]);
  };
  if (tid == 0) {
    if ((uint64_t)blockIdx.x < ntiles) issue(blockIdx.x, 0);
    if ((uint64_t)blockIdx.x + gridDim.x < ntiles) issue(blockIdx.x + gridDim.x, 1);
  }

  int64_t acc = 0;
  uint32_t cnt = 0;
  uint32_t qn = 0;  // rows pending in this warp's queue (warp-uniform)
  uint32_t it = 0;
  const uint32_t nchunks = T / 32;
  for (uint64_t t = blockIdx.x; t < ntiles; t += gridDim.x, ++it) {
    const int s = it & 1;
    const uint32_t parity = (it >> 1) & 1u;
    const bool arrived = mbar_wait_bounded(&bars[s], parity, errw, MB_DEVERR_TMA_WAIT);
    if (!__syncthreads_and(arrived)) {
      if (tid == 0) mbar_wait_bounded(&bars[s], parity, nullptr, 0, 1u << 16);
      break;
    }
    TileView tv;
    tv.stage = stages + s * stage_words;
    tv.T = T;
    tv.valid = valid_words(t);
    tv.copied = tv.valid & ~3u;
    tv.w0 = t * T;
    if (tv.copied < T) {  // last tile: tail words by plain loads, the rest zero
      uint32_t *st = stages + s * stage_words;
      const uint32_t span = T - tv.copied;
      for (uint32_t i = tid; i < nb * span; i += FT_THREADS) {
        const uint32_t b = i / span, lw = tv.copied + i % span;
        st[(size_t)b * T + lw] = lw < tv.valid ? __ldg(P.ptr[b] + tv.w0 + lw) : 0u;
      }
      __syncthreads();
    }
    // phase A: the program over the staged tile, one word per lane per chunk
    for (uint32_t c = warp; c < nchunks; c += FT_WARPS) {
      const uint32_t w = c * 32 + lane;
      uint32_t p1, u1;
      if (P.cnf) {
        cnf_eval<CHK>(P, tv, w, p1, u1);
      } else {
        uint32_t lw[1] = {w}, p[1], u[1];
        vbp_eval_staged<1, CHK>(P, tv, lw, p, u);
        p1 = p[0], u1 = u[0];
      }
      ptile[w] = p1;
      if (CHK) utile[w] = u1;
    }
    __syncthreads();  // stage s consumed, ptile complete
    if (tid == 0 && t + 2ull * gridDim.x < ntiles) issue(t + 2ull * gridDim.x, s);
    // phase B: compaction into the warp queue; the op runs on full 64-row batches
    for (uint32_t c = warp; c < nchunks; c += FT_WARPS)
      compact_chunk<CHK, GS>(O, N, queue, qn, tv.w0 + c * 32, ptile[c * 32 + lane], CHK ? utile[c * 32 + lane] : 0u,
                             nr_grp, G, acc, cnt);
  }
  if (qn) drain64<CHK ? DR_FLAG : DR_NOCHK, GS>(O, N, queue, qn, nr_grp, G, acc, cnt);
  __syncthreads();
  grp_flush<GS>(G, nr_grp, acc, cnt, nqual, red);
}

// ------------------------------------------------------------------ host
constexpr size_t FT_STAGE_TARGET = 24 * 1024;  // bytes of one stage when the tile can shrink

template <bool CHK, int GS>
static mb_status launch_ft(const DevPrg &P, const mb_op &O, uint32_t nb, uint32_t T, uint32_t nr_grp,
                           uint32_t hcap, int64_t *out, uint64_t *nq, uint32_t cps, cudaStream_t st) {
  auto kern = fused_tma_kernel<CHK, GS>;
  const size_t smem = 2 * (size_t)nb * T * 4 + (size_t)T * 4 * (CHK ? 2 : 1) +
                      ((grp_smem_bytes(GS, nr_grp, hcap) + 15) & ~(size_t)15) + (size_t)FT_WARPS * FT_QCAP * 4;
  const DevInfo &di = dev_info();
  if (smem > (size_t)di.max_smem_optin) return fail(MB_ERR_INVALID, "fused: %zu bytes of shared memory", smem);
  MB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int occ = 0;
  MB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, FT_THREADS, smem));
  if (occ < 1) return fail(MB_ERR_INVALID, "fused: kernel does not fit on an SM");
  if (cps && (int)cps < occ) occ = (int)cps;
  const uint64_t ntiles = (P.nwords + T - 1) / T;
  uint64_t grid = (uint64_t)di.sms * occ;
  if (grid > ntiles) grid = ntiles ? ntiles : 1;
  uint32_t *errw = device_error_word();
  if (!errw) return fail(MB_ERR_OOM, "fused: device error word");
  kern<<<(unsigned)grid, FT_THREADS, smem, st>>>(P, O, op_needs(O), nb, T, nr_grp, hcap,
                                                 reinterpret_cast<unsigned long long *>(out),
                                                 reinterpret_cast<unsigned long long *>(nq), errw);
  MB_LAUNCH_CHECK("fused_tma_kernel");
  return MB_OK;
}

template <bool CHK>
static mb_status ft_gs(int gs, const DevPrg &P, const mb_op &O, uint32_t nb, uint32_t T, uint32_t nr_grp,
                       uint32_t hcap, int64_t *out, uint64_t *nq, uint32_t cps, cudaStream_t st) {
  switch (gs) {
  case GS_SCALAR: return launch_ft<CHK, GS_SCALAR>(P, O, nb, T, nr_grp, hcap, out, nq, cps, st);
  case GS_SHARED: return launch_ft<CHK, GS_SHARED>(P, O, nb, T, nr_grp, hcap, out, nq, cps, st);
  case GS_GLOBAL: return launch_ft<CHK, GS_GLOBAL>(P, O, nb, T, nr_grp, hcap, out, nq, cps, st);
  default: return launch_ft<CHK, GS_HASH>(P, O, nb, T, nr_grp, hcap, out, nq, cps, st);
  }
}

// The staged kernel applies when every bitmap is 16-byte aligned (bulk
// copies), every op source is at most 4 bytes wide and the program reads at
// least one bitmap.
bool fused_tma_applies(const DevPrg &P, bool vec4, const mb_op &O) {
  uint32_t nb = 0;
  for (uint32_t c = 0; c < MB_MAXCOLS; ++c) nb += P.nmid[c] + P.nedge[c];
  if (!vec4 || nb == 0 || P.nrows == 0) return false;
  for (uint32_t s = 0; s < O.nsrc; ++s)
    if (O.src[s].width > 4) return false;
  return true;
}

static size_t ft_smem(uint32_t nb, uint32_t T, bool chk, int gs, uint32_t nr_grp, uint32_t hcap) {
  return 2 * (size_t)nb * T * 4 + (size_t)T * 4 * (chk ? 2 : 1) +
         ((grp_smem_bytes(gs, nr_grp, hcap) + 15) & ~(size_t)15) + (size_t)FT_WARPS * FT_QCAP * 4;
}

// V (words per thread of a tile; 0 = auto) sets the tile to 256 * V words:
// auto picks the widest tile whose stage stays near FT_STAGE_TARGET bytes;
// a tile that does not fit in shared memory shrinks.  Returns
// MB_ERR_UNSUPPORTED if even the narrowest tile does not fit.
mb_status fused_tma(const DevPrg &P, const mb_op &O, uint32_t nr_grp, int gs, uint32_t hcap, uint32_t V,
                    int64_t *out, uint64_t *nq, uint32_t cps, cudaStream_t st) {
  uint32_t nb = 0;
  for (uint32_t c = 0; c < MB_MAXCOLS; ++c) nb += P.nmid[c] + P.nedge[c];
  if (V == 0) V = nb * FT_THREADS * 4 * 4 <= FT_STAGE_TARGET ? 4 : nb * FT_THREADS * 2 * 4 <= FT_STAGE_TARGET ? 2 : 1;
  const size_t cap = (size_t)dev_info().max_smem_optin;
  while (V > 1 && ft_smem(nb, FT_THREADS * V, P.chk != 0, gs, nr_grp, hcap) > cap) V >>= 1;
  if (ft_smem(nb, FT_THREADS * V, P.chk != 0, gs, nr_grp, hcap) > cap)
    return fail(MB_ERR_UNSUPPORTED, "fused: %u bitmaps do not fit a staged tile", nb);
  const uint32_t T = FT_THREADS * V;
  return P.chk ? ft_gs<true>(gs, P, O, nb, T, nr_grp, hcap, out, nq, cps, st)
               : ft_gs<false>(gs, P, O, nb, T, nr_grp, hcap, out, nq, cps, st);
}

// ------------------------------------------------- warp-independent kernel
bool fused_warp_applies(const DevPrg &P, const mb_op &O, size_t grp_bytes, uint32_t warps) {
  // with candidate checks, bit 31 of a queued row says that it is uncertain
  if (P.nrows == 0 || P.nrows >= (P.chk ? 1ull << 31 : 1ull << 32)) return false;
  for (uint32_t s = 0; s < O.nsrc; ++s)
    if (O.src[s].width > 4) return false;
  // beside a group table near the limit (shared tables of 24,700 groups and more, on
  // request) a general program's row list of 2 or 4 KB a warp may fit where a queue does not
  return P.cnf || fw_smem(grp_bytes, warps) + FW_STATIC <= (size_t)dev_info().max_smem_optin;
}

template <int V, bool CHK, int GS>
static mb_status launch_fw(const DevPrg &P, const mb_op &O, uint32_t nr_grp, uint32_t hcap, int64_t *out,
                           uint64_t *nq, uint32_t warps, uint32_t cps, cudaStream_t st) {
  auto go = [&](auto kern) {
    return fw_launch(kern, V, P.nwords, grp_smem_bytes(GS, nr_grp, hcap), warps, cps, st, P, O, op_needs(O), nr_grp,
                     hcap, reinterpret_cast<unsigned long long *>(out), reinterpret_cast<unsigned long long *>(nq));
  };
  if constexpr (!CHK) {
    if (!op_needs(O).behind_key) {
      if constexpr (V < 4) {  // (general programs of four words run in the general kernel)
        if (!P.cnf) return go(fused_warp_kernel<V, CHK, GS, false, true>);
      }
      return go(fused_warp_kernel<V, CHK, GS, true, true>);
    }
  }
  if constexpr (V < 4) {
    if (!P.cnf) return go(fused_warp_kernel<V, CHK, GS, false, false>);
  }
  return go(fused_warp_kernel<V, CHK, GS, true, false>);
}

template <int V, bool CHK>
static mb_status fw_gs(int gs, const DevPrg &P, const mb_op &O, uint32_t nr_grp, uint32_t hcap, int64_t *out,
                       uint64_t *nq, uint32_t warps, uint32_t cps, cudaStream_t st) {
  switch (gs) {
  case GS_SCALAR: return launch_fw<V, CHK, GS_SCALAR>(P, O, nr_grp, hcap, out, nq, warps, cps, st);
  case GS_SHARED: return launch_fw<V, CHK, GS_SHARED>(P, O, nr_grp, hcap, out, nq, warps, cps, st);
  case GS_GLOBAL: return launch_fw<V, CHK, GS_GLOBAL>(P, O, nr_grp, hcap, out, nq, warps, cps, st);
  default: return launch_fw<V, CHK, GS_HASH>(P, O, nr_grp, hcap, out, nq, warps, cps, st);
  }
}

int shape_of(const mb_op &O, uint32_t nr_grp, uint32_t sure, ShapeArgs *A, bool *narrow, uint32_t keyed) {
  memset(A, 0, sizeof(*A));
  A->ng = nr_grp;
  if (O.nsrc > 6) return -1;
  const OpNeeds N = op_needs(O);
  uint32_t keym = 0, yearm = 0, termm = 0;
  for (uint32_t c = 0; c < O.nclause; ++c) {
    if (O.clause_len[c] != 1) return -1;
    const mb_term &t = O.terms[c];
    if ((termm >> t.src) & 1u || t.lo >= t.hi || t.lo > 0xffffffffull) return -1;
    termm |= 1u << t.src;
    if (!((sure >> c) & 1u)) A->fmask |= 1u << t.src;
    A->lo[t.src] = (uint32_t)t.lo;
    A->hi[t.src] = t.hi > 0x100000000ull ? 0xffffffffu : (uint32_t)(t.hi - 1);
  }
  for (uint32_t k = 0; k < O.nkey; ++k) {
    const mb_key &kk = O.keys[k];
    if (kk.src > 3 || (keym >> kk.src) & 1u) return -1;
    keym |= 1u << kk.src;
    ShapeKey &K = A->key[kk.src];
    if (kk.xform == MB_X_YEAR) yearm |= 1u << kk.src;
    const uint32_t d = kk.xform == MB_X_DIV ? kk.div : 1u;
    if (d == 0) return -1;
    const DivMagic m = div_magic(d);
    K = ShapeKey{m.m, m.sh1, m.sh2, kk.base, kk.mul, d == 1 ? 1u : 0u};
  }
  for (uint32_t i = 0; i < BNSHAPE; ++i) {
    const BShape &b = BSHAPES[i];
    if (b.ns != O.nsrc || b.kv != N.kv_mask || b.filt != N.filt_mask || b.filt != termm || b.keym != keym ||
        b.yearm != yearm || b.vk != O.vkind || b.va != O.va || (b.vk != MB_V_COL && b.vb != O.vb))
      continue;
    for (int nar = 0; nar < 2; ++nar) {
      bool same = true;
      for (uint32_t s = 0; s < b.ns && same; ++s) same = (!O.src[s].fk || (keyed >> s & 1u)) && O.src[s].width == SHAPE_W[i][nar][s];
      if (!same) continue;
      for (uint32_t s = 0; s < b.ns; ++s) A->col[s] = O.src[s].col, A->fk[s] = O.src[s].fk;
      *narrow = nar != 0;
      return (int)i;
    }
  }
  return -1;
}

mb_status fused_warp(const DevPrg &P, bool vec4, const mb_op &O, uint32_t sure, uint32_t nr_grp, int gs, uint32_t hcap,
                     uint32_t V, uint32_t warps, int64_t *out, uint64_t *nq, uint32_t cps, cudaStream_t st) {
  const bool chk = P.chk != 0;
  ShapeArgs A;
  bool narrow = false;
  const int sh = gs == GS_HASH || !P.cnf ? -1 : shape_of(O, nr_grp, sure, &A, &narrow);
  // a compiled op: one group in a register (shape 1), or several in a table
  const bool compiled = sh >= 0 && (sh == 0 ? gs == GS_SCALAR : gs != GS_SCALAR && nr_grp >= GRP_DIRECT_MIN);
  // Words a lane: wider tiles mean fewer, wider loads and fewer warps at work.
  // Device time in us at V = 1 / 2 / 4: 13 SSB queries, 1M rows 179 / 185 / 189; with a
  // 24-query spanning and a 24-query random mix beside them (narrow columns), back to back:
  //   60M      533 / 477 / 478     1,788 / 1,555 / 1,607    833 / 702 / 693
  //   120M     935 / 827 / 808     3,302 / 2,787 / 2,763  1,426 / 1,159 / 1,090
  //   200M   1,460 / 1,272 / 1,240  5,278 / 4,401 / 4,266  2,144 / 1,727 / 1,619
  // and V = 2 / 4 with the L2 flushed before each query:
  //   90M      792 / 786           2,408 / 2,408          1,076 / 1,034
  //   120M     972 / 968           3,022 / 2,995          1,324 / 1,263
  //   162M   1,232 / 1,214         3,946 / 3,834          1,677 / 1,584
  // (at 120M the densest query of the 13 still loses 7 % by four).
  // An interpreted op does not take four: 240M rows, 256 groups, a chain over 6 % of
  // the rows 196 / 189 / 197 us, over a third 640 / 656 / 662, with checks over 6 % 526 / 583
  // / 734 (over 0.1 % it gains 9 %: 79 / 69 / 63); a general program in this kernel, an OR
  // over 30 %, - / 429 / 736, with checks 1,510 / 1,609 / 3,367.
  if (V == 0) V = P.nrows < 4000000 ? 1 : !compiled || P.nrows < 150000000 ? 2 : 4;
  if (V == 4 && !P.cnf) V = 2;             // (no kernel of four; fused_grpby does not ask for it)
  warps = fw_warps(warps);
  if (!vec4) V = 1;                        // unaligned bitmaps: word loads
  if (compiled) {
    const ShapeLaunch L{nr_grp, V, warps, cps, gs, narrow, reinterpret_cast<unsigned long long *>(out),
                        reinterpret_cast<unsigned long long *>(nq), st};
    switch (sh) {
    case 0: return fused_shape1(P, A, L);
    case 1: return fused_shape2(P, A, L);
    case 2: return fused_shape3(P, A, L);
    default: return fused_shape4(P, A, L);
    }
  }
  if (V == 4) return chk ? fw_gs<4, true>(gs, P, O, nr_grp, hcap, out, nq, warps, cps, st)
                         : fw_gs<4, false>(gs, P, O, nr_grp, hcap, out, nq, warps, cps, st);
  if (V == 2) return chk ? fw_gs<2, true>(gs, P, O, nr_grp, hcap, out, nq, warps, cps, st)
                         : fw_gs<2, false>(gs, P, O, nr_grp, hcap, out, nq, warps, cps, st);
  return chk ? fw_gs<1, true>(gs, P, O, nr_grp, hcap, out, nq, warps, cps, st)
             : fw_gs<1, false>(gs, P, O, nr_grp, hcap, out, nq, warps, cps, st);
}

}  // namespace mb
