// Paged GQA decode / speculative-verify attention over FP8 KV on tcgen05, tokens on the TMEM lanes.
//
// With one (or a few) query tokens per sequence only `q_len * group` rows are live; putting them on the MMA's
// M dimension would leave 124 of 128 softmax rows idle and makes the exponential unit the bottleneck.  Here the
// problem is transposed:
//     S^T = K Q^T   : A = K tile [128 tokens x D] (smem, straight from the page pool), B = Q [NMAX rows x D]
//     O^T_t = V^T P^T : A = V^T tile [D x 128 tokens] (smem, from the pool), B = P [NMAX rows x 128 tokens]
// so every softmax thread owns one key position and touches only RMAX (2, 4, 8, 12 or 16) columns of tensor memory, and
// every accumulate thread owns one output dimension with RMAX running sums in registers.  Row maxima are
// exchanged across the four softmax warps once per tile; row sums are reduced once per work item.
//
// Work item = (sequence, kv head, block of NMAX rows); persistent CTAs; 320 threads (page loader warp, MMA warp, two sets
// of four softmax warps that take alternate tiles and are merged per work item); 2 CTAs per SM when at most 8 rows are
// live, else one CTA with a second loader warp.  Every wait is a bounded mbarrier wait.
//
// Loaders: keys and values have rings of their own, and a value slot is free two tiles after the key slot.  Two halves of one warp
// fill the rings where two CTAs share an SM; a half that waits holds up the other one, which the second CTA covers.  A single CTA
// has a warp for each ring: keys that came only as values were done with set the pace (1.5 us a tile).  64 sequences of 2400 tokens,
// 8 kv heads of 16 rows: 157 -> 114 us, 256 of 1200 tokens, 9 rows: 288 -> 204 us.
//
// Sharing out the work: with few sequences every item's keys are cut into `splits` equal runs of tiles (partial sums, which
// attn_decode_combine_kernel merges), and the runs are taken longest first, the second round from the other end: in the items'
// order the longest sequence's runs met others of their kind.  Six sequences of 6 K to 16 K tokens: 46 -> 34 us (with the loops below).
//
// What bounds it: the pages' bytes at 4 rows (85 % of copy bandwidth at 256 x 1.2 K tokens), the softmax warps at 8.  Their loops
// run over all RMAX rows without a test of how many are live (a branch per row kept the rows' chains of maximum, exponential
// and conversion from overlapping), tiles that no mask touches skip the masks, and what is done once per item is short: code
// that runs once per item comes from beyond the instruction caches.  256 sequences of 1.2 K tokens, 8 kv heads of 4 rows:
// 120 -> 113 us; 4 kv heads of 8 rows: 99 -> 77 us; 64 sequences, 8 kv heads of 8 rows: 52 -> 36 us; 16 sequences of 1.0 K to
// 2.1 K tokens with 20 rows: 86 -> 51 us (with the loaders).
// (Warp MMAs with the rows as M and probabilities in half precision need no word between warps until an item ends and took
// 43 us there, but 189 instead of 113 us for 4 rows; and a token verified in one kernel and decoded in the other would see its
// probabilities rounded differently.)
//
// Reference counterparts: kernels/src/cuda/mha_nvfp4.cu mha_decode_kernel :259 and mha_combine_kernel :572,
// kernels/src/cuda/mha_verify.cu verify_kernel :50.
#include "blaze/attn.cuh"
#include "blaze/host.h"

namespace blz {

constexpr int kOrdered = 64;          // sequences that a launch with splits takes by their length (more: as they come)

constexpr int NMAX = 16;              // MMA N: rows per work item

// RMAX = rows kept in registers by the softmax threads (2, 4, 8, 12 or 16, >= live rows).
template <int RMAX>
struct DecCfg {
  static constexpr int D = 128;
  static constexpr int PAGE_BYTES = 16 * D;
  static constexpr int TILE_BYTES = 8 * PAGE_BYTES;
  static constexpr bool V_WARP = RMAX > 8;           // values are loaded by a warp of their own
  static constexpr int THREADS = V_WARP ? 352 : 320;    // loader warp(s), MMA warp, two sets of four softmax warps
  static constexpr int CTAS_PER_SM = RMAX <= 8 ? 2 : 1;
  static constexpr int STAGES = CTAS_PER_SM == 2 ? 3 : 5;   // depth of the K ring and of the V ring (released separately)
  static constexpr int Q_BYTES = NMAX * D;
  static constexpr int P_BYTES = NMAX * 128;
  static constexpr int NB = 3;                       // S^T / P / O^T buffers (softmax runs up to two tiles ahead of the fold)
  static constexpr int TMEM_COLS = 128;
  static constexpr int SMEM = 2 * Q_BYTES + STAGES * 2 * TILE_BYTES + NB * P_BYTES + 128 + 640;
};

// The wait counters live in shared memory: thirteen 64-bit registers for a run that is not profiled would spill the others.
__device__ __forceinline__ bool timed_wait(long long* acc, bool on, uint64_t* bar, uint32_t par, volatile int* abort_flag,
                                           int* status) {
  if (!on) return mbar_wait(bar, par, abort_flag, status);
  const long long t = clock64();
  const bool r = mbar_wait(bar, par, abort_flag, status);
  if ((threadIdx.x & 31) == 0) *acc += clock64() - t;
  return r;
}

// What a CTA takes k-th of the work (sequence, row block, kv head, split), largest sequences first: CTA c takes c, then, in
// rounds, 2 ctas - 1 - c, 2 ctas + c, ... of the list.  `order`: the sequences by falling length (null: as they come).
__device__ __forceinline__ int kth_unit(int k, int cta, int ctas) { return k * ctas + ((k & 1) ? ctas - 1 - cta : cta); }

// Sums of every row over the warp's lanes, R rows per lane (a power of two, at most 16).  Each of the first steps halves the rows a
// lane carries, so it takes R - 1 + log2(32 / R) exchanges instead of 5 R; the sums are those of a butterfly from 16 down.  A lane
// gets the row whose bits, from the lowest, are its own from the highest.
template <int R>
__device__ __forceinline__ float sum_rows(float (&v)[R], int lane) {
  int bit = 16;
#pragma unroll
  for (int n = R / 2; n > 0; n >>= 1, bit >>= 1) {
    const bool hi = lane & bit;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const float give = hi ? v[2 * i] : v[2 * i + 1], keep = hi ? v[2 * i + 1] : v[2 * i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
    }
  }
  for (; bit > 0; bit >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], bit);
  return v[0];
}
template <int R>
__device__ __forceinline__ int row_of_lane(int lane) {        // -1: another lane has the row, too
  constexpr int BITS = R == 2 ? 1 : R == 4 ? 2 : R == 8 ? 3 : 4;
  return (lane & ((32 >> BITS) - 1)) ? -1 : (int)(__brev((unsigned)lane) >> 27) & (R - 1);
}

__device__ __forceinline__ void put_pair(float* p, float a, float b) { p[0] = a; p[1] = b; }      // (the caller's array: on 4 bytes)

// The first R columns of the lane's row in tensor memory (complete when it returns).
template <int R>
__device__ __forceinline__ void tmem_rows(uint32_t taddr, float (&v)[R]) {
  uint32_t a[R <= 4 ? 4 : R == 12 ? 8 : R], b[4] = {0, 0, 0, 0};
  if constexpr (R <= 4) tmem_ld4(taddr, a);
  else if constexpr (R == 8) tmem_ld8(taddr, a);
  else if constexpr (R == 12) { tmem_ld8(taddr, a); tmem_ld4(taddr + 8, b); }
  else tmem_ld16(taddr, a);
  tmem_ld_wait();
#pragma unroll
  for (int r = 0; r < R; ++r) v[r] = __uint_as_float(R == 12 && r >= 8 ? b[r & 3] : a[R == 12 ? r & 7 : r]);
}

// V (2 or 4) floats of shared memory.
template <int V>
__device__ __forceinline__ void load_some(const float* src, float (&v)[V]) {
  if constexpr (V == 4) {
    const float4 q = *reinterpret_cast<const float4*>(src);
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
  } else {
    const float2 q = *reinterpret_cast<const float2*>(src);
    v[0] = q.x; v[1] = q.y;
  }
}

template <int RMAX>
__global__ void __launch_bounds__(DecCfg<RMAX>::THREADS, (DecCfg<RMAX>::CTAS_PER_SM)) attn_decode_kernel(AttnParams p) {
  using Cfg = DecCfg<RMAX>;
  constexpr int VW = RMAX % 4 == 0 ? 4 : 2;          // rows per access of shared memory
  constexpr int ST = Cfg::STAGES, D = Cfg::D, NB = Cfg::NB;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
  uint8_t* sK = smem;
  uint8_t* sV = sK + ST * Cfg::TILE_BYTES;
  uint8_t* sQ = sV + ST * Cfg::TILE_BYTES;
  uint8_t* sP = sQ + 2 * Cfg::Q_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sP + NB * Cfg::P_BYTES);
  uint64_t* k_full = bars;                 // [ST]
  uint64_t* v_full = k_full + ST;          // [ST]
  uint64_t* k_empty = v_full + ST;         // [ST] released when S^T = K Q^T of the tile has completed
  uint64_t* v_empty = k_empty + ST;        // [ST] released when O^T = V^T P^T of the tile has completed
  uint64_t* s_full = v_empty + ST;         // [NB]
  uint64_t* s_empty = s_full + NB;         // [NB]
  uint64_t* p_full = s_empty + NB;         // [NB]
  uint64_t* o_full = p_full + NB;          // [NB]
  uint64_t* o_empty = o_full + NB;         // [NB]
  uint64_t* wm_bar = o_empty + NB;         // [NB] row-max exchange among the softmax warps
  uint64_t* q_full = wm_bar + NB;          // [2]
  uint64_t* q_empty = q_full + 2;          // [2]
  uint64_t* fin_bar = q_empty + 2;         // [1] both sets have published their partial results
  uint64_t* acc_free = fin_bar + 1;        // [1] set 0 has consumed set 1's partial results
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_free + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  __shared__ __align__(16) float s_c[2][NMAX];
  __shared__ int s_pos[2][NMAX];
  __shared__ uint16_t s_order[kOrdered];
  __shared__ int s_len[kOrdered];
  __shared__ long long s_prof[3][13];
  __shared__ uint32_t s_mask[2][NMAX];   // tree verify: which of the sequence's new tokens a row may see (bit per token)
  __shared__ __align__(16) float s_wmax[Cfg::NB][4][RMAX];
  __shared__ float s_l[2][4][RMAX];                  // [set][warp][row] partial row sums
  __shared__ float s_m[2][RMAX];                     // row maxima of the two sets
  __shared__ float2 s_f[4][RMAX];                    // [warp of set 0][row]: what the two sets' sums are multiplied by
  __shared__ float s_div[4][RMAX];                   // ... and divided by
  __shared__ int s_off[4][RMAX];                     // ... and the row (of the output, or of the piece) they go to
  __shared__ float s_acc[RMAX][128];                 // set 1's output sums

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < ST; ++i) { mbar_init(&k_full[i], 1); mbar_init(&v_full[i], 1); mbar_init(&k_empty[i], 1); mbar_init(&v_empty[i], 1); }
    for (int i = 0; i < NB; ++i) {
      mbar_init(&s_full[i], 1); mbar_init(&s_empty[i], 4); mbar_init(&p_full[i], 4);
      mbar_init(&o_full[i], 1); mbar_init(&o_empty[i], 4); mbar_init(&wm_bar[i], 4);
    }
    for (int i = 0; i < 2; ++i) { mbar_init(&q_full[i], 1); mbar_init(&q_empty[i], 1); }
    mbar_init(fin_bar, 8); mbar_init(acc_free, 4);
    *abort_flag = 0;
    mbar_fence_init();
  }
  for (int i = threadIdx.x; i < 2 * Cfg::Q_BYTES / 16; i += blockDim.x) reinterpret_cast<uint4*>(sQ)[i] = make_uint4(0, 0, 0, 0);
  fence_async_smem();
  if (warp == 1) tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_trigger();        // after the allocation (sm100.cuh)
  const uint32_t tmem = *tmem_slot;
  pdl_wait();          // the queries and this step's K/V rows come from the kernel before this one

  const int group = p.Hq / p.Hkv;
  int g = 0, item_it = 0;
  const bool prof = p.prof != nullptr && blockIdx.x < 8 && warp < 3;
  long long* pc = s_prof[prof ? warp : 0];
  if (prof && lane == 0) {
    for (int i = 0; i < 12; ++i) pc[i] = 0;
    pc[12] = -clock64();
  }
#define TW(cat, bar, par) timed_wait(&pc[cat], prof, bar, par, abort_flag, p.status)

  const int total = p.num_items * p.Hkv * p.row_blocks * p.splits;
  const bool ordered = p.splits > 1 && p.num_items > 1 && p.num_items <= kOrdered;
  if (ordered) {
    // the sequences by falling length (every thread ranks its own; there are few)
    const int mine = threadIdx.x;
    if (mine < p.num_items) s_len[mine] = p.ctx_len[mine];
    __syncthreads();
    if (mine < p.num_items) {
      const int len = s_len[mine];
      int rank = 0;
      for (int j = 0; j < p.num_items; ++j) { const int l = s_len[j]; rank += l > len || (l == len && j < mine); }
      s_order[rank] = mine;
    }
    __syncthreads();
  }
  for (int k = 0; ; ++k) {
    const int u = p.splits > 1 ? kth_unit(k, blockIdx.x, gridDim.x) : k * (int)gridDim.x + (int)blockIdx.x;
    if (k * (int)gridDim.x >= total) break;
    if (u >= total) continue;
    const int split = u % p.splits;
    const int rb = (u / p.splits) % p.row_blocks;
    const int kh = (u / (p.splits * p.row_blocks)) % p.Hkv;
    int b = u / (p.splits * p.row_blocks * p.Hkv);
    if (ordered) b = s_order[b];
    const int w = ((b * p.Hkv + kh) * p.row_blocks + rb) * p.splits + split;      // where a run's partial sums go
    const int r0 = p.q_start[b], qlen = p.q_start[b + 1] - r0;
    const int rows_total = qlen * group;
    if (rows_total < p.min_rows || rows_total > p.max_rows) continue;
    const int row0 = rb * NMAX;
    const int nrows = min(NMAX, rows_total - row0);
    if (nrows <= 0) continue;
    const int ctx = p.ctx_len[b];
    const int kv_end = ctx - qlen + (row0 + nrows - 1) / group + 1;       // keys visible to the block's last row
    const int tiles_all = (kv_end + 127) >> 7;
    const int per = (tiles_all + p.splits - 1) / p.splits;
    const int t0 = split * per;
    const int n = max(min(tiles_all, t0 + per) - t0, 0);
    const int slot = p.slots[b];
    if (n == 0) {
      // a run without a tile: nothing to add.  (Without splits there is nowhere to say so: rows that see no key are left alone.)
      if (p.splits > 1 && warp == 2)
        for (int r = lane; r < nrows; r += 32)
          put_pair(&p.part_ml[((size_t)w * NMAX + r) * 2], -INFINITY, 0.f);
      continue;
    }

    const int* bt = p.block_table + (size_t)slot * p.bt_stride;
    const int npages = (kv_end + 15) >> 4;
    // V^T tiles of the item: sixteen lanes, lane vl of which takes page vl of a tile
    auto load_values = [&](int vl, uint32_t mask) {
      int page = 0;
      if (vl < 8) { const int pidx = t0 * 8 + vl; page = pidx < npages ? bt[pidx] : 0; }
      for (int i = 0; i < n; ++i) {
        const int gi = g + i, s = gi % ST;
        int next = 0;
        if (vl < 8 && i + 1 < n) { const int pidx = (t0 + i + 1) * 8 + vl; next = pidx < npages ? bt[pidx] : 0; }
        if (!mbar_wait(&v_empty[s], ((gi / ST) & 1) ^ 1, abort_flag, p.status)) break;
        if (vl == 0) mbar_expect_tx(&v_full[s], Cfg::TILE_BYTES);
        __syncwarp(mask);
        if (vl < 8) {
          const uint8_t* src = p.pool + (size_t)page * p.page_stride + (size_t)kh * p.head_stride + Cfg::PAGE_BYTES;
          bulk_load(sV + s * Cfg::TILE_BYTES + vl * Cfg::PAGE_BYTES, src, Cfg::PAGE_BYTES, &v_full[s]);
        }
        __syncwarp(mask);
        page = next;
      }
    };
    if (warp == 0) {
      // -------------------------------------------------------------- page loader
      {
        // ---- this item's Q rows → e4m3 in the K-major core-matrix layout, plus the per-row constants
        // Items of at most 8 live rows (plain decode at group 4 or 8, two verify rows) are prepared by the K half of the
        // warp alone, 4 or 2 lanes per row: the two halves then never meet, and this half moves on to the next item's Q
        // rows and K tiles while the V half is still waiting for ring slots of this one.  (The rows beyond RMAX of both Q
        // buffers are zeroed once, before the loop.)
        constexpr bool HALF = RMAX <= 8;
        constexpr int LPR = RMAX <= 4 ? 4 : 2;              // lanes per row
        constexpr int DPL = D / LPR;                               // dims per lane
        constexpr uint32_t QMASK = HALF ? 0x0000FFFFu : 0xFFFFFFFFu;
        if (!HALF || lane < 16) {
        const int qb = item_it & 1;
        const int rr = lane / LPR, part = lane % LPR;
        const int R = row0 + rr;
        const bool live = rr < nrows;
        const int tq = R / group, hq = kh * group + R % group;
        uint4 raw[DPL / 8];
        float amax = 0.f;
        if (live) {
          const __nv_bfloat16* qrow = p.q + ((size_t)(r0 + tq) * p.Hq + hq) * D + part * DPL;
#pragma unroll
          for (int j = 0; j < DPL / 8; ++j) raw[j] = *reinterpret_cast<const uint4*>(qrow + j * 8);
#pragma unroll
          for (int j = 0; j < DPL / 8; ++j) {
            const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(&raw[j]);
#pragma unroll
            for (int k = 0; k < 8; ++k) amax = fmaxf(amax, fabsf(bf2f(e[k])));
          }
        }
        if (LPR >= 2) amax = fmaxf(amax, __shfl_xor_sync(QMASK, amax, 1));
        if (LPR == 4) amax = fmaxf(amax, __shfl_xor_sync(QMASK, amax, 2));
        const float qscale = fmaxf(amax, 1e-12f) / 448.f;
        const float qinv = 1.f / qscale;
        if (!TW(10, &q_empty[qb], ((item_it >> 1) & 1) ^ 1)) break;
        uint8_t* qdst = sQ + qb * Cfg::Q_BYTES + (rr >> 3) * (8 * D) + (rr & 7) * 16 + (part * DPL / 16) * 128;
#pragma unroll
        for (int j = 0; j < DPL / 16; ++j) {
          uint4 o = make_uint4(0, 0, 0, 0);
          if (live) {
            const __nv_bfloat16* e0 = reinterpret_cast<const __nv_bfloat16*>(&raw[2 * j]);
            const __nv_bfloat16* e1 = reinterpret_cast<const __nv_bfloat16*>(&raw[2 * j + 1]);
            o.x = pack_e4m3x4(bf2f(e0[0]) * qinv, bf2f(e0[1]) * qinv, bf2f(e0[2]) * qinv, bf2f(e0[3]) * qinv);
            o.y = pack_e4m3x4(bf2f(e0[4]) * qinv, bf2f(e0[5]) * qinv, bf2f(e0[6]) * qinv, bf2f(e0[7]) * qinv);
            o.z = pack_e4m3x4(bf2f(e1[0]) * qinv, bf2f(e1[1]) * qinv, bf2f(e1[2]) * qinv, bf2f(e1[3]) * qinv);
            o.w = pack_e4m3x4(bf2f(e1[4]) * qinv, bf2f(e1[5]) * qinv, bf2f(e1[6]) * qinv, bf2f(e1[7]) * qinv);
          }
          *reinterpret_cast<uint4*>(qdst + j * 128) = o;
        }
        if (part == 0) {
          s_c[qb][rr] = p.scale_log2 * qscale;
          s_pos[qb][rr] = live ? ctx - qlen + tq : -1;
          if constexpr (RMAX > 4) s_mask[qb][rr] = (live && p.tree_mask) ? (uint32_t)p.tree_mask[r0 + tq] : 0xFFFFFFFFu;
        }
        fence_async_smem();
        __syncwarp(QMASK);
        if (lane == 0) mbar_arrive(&q_full[qb]);
        }
      }
      // The lower half of the warp streams K tiles, the upper half V^T tiles: the two rings are released at different
      // times (K after S^T = K Q^T, V two tiles later after O^T = V^T P^T), so each half waits only for its own ring
      // (and, for plain decode items, runs through the work items at its own pace).
      // (the page number of the next tile is fetched before the wait for its ring slot, off the critical path)
      if (lane < 16) {
        int page = 0;
        if (lane < 8) { const int pidx = t0 * 8 + lane; page = pidx < npages ? bt[pidx] : 0; }
        for (int i = 0; i < n; ++i) {
          const int gi = g + i, s = gi % ST;
          int next = 0;
          if (lane < 8 && i + 1 < n) { const int pidx = (t0 + i + 1) * 8 + lane; next = pidx < npages ? bt[pidx] : 0; }
          if (!TW(0, &k_empty[s], ((gi / ST) & 1) ^ 1)) break;
          if (lane == 0) mbar_expect_tx(&k_full[s], Cfg::TILE_BYTES);
          __syncwarp(0x0000FFFFu);
          if (lane < 8) {
            const uint8_t* src = p.pool + (size_t)page * p.page_stride + (size_t)kh * p.head_stride;   // page 0 = zero scratch page
            bulk_load(sK + s * Cfg::TILE_BYTES + lane * Cfg::PAGE_BYTES, src, Cfg::PAGE_BYTES, &k_full[s]);
          }
          __syncwarp(0x0000FFFFu);
          page = next;
        }
      } else if constexpr (!Cfg::V_WARP) {
        load_values(lane - 16, 0xFFFF0000u);
      }
      if constexpr (RMAX > 8) __syncwarp();
    } else if (warp == 1) {
      // -------------------------------------------------------------- MMA issuer
      if (lane == 0) {
        bool ok = TW(6, &q_full[item_it & 1], (item_it >> 1) & 1);
        tc_fence_after();
        const uint32_t q_addr = smem_u32(sQ + (item_it & 1) * Cfg::Q_BYTES);
        auto issue_pv = [&](int gj) -> bool {
          const int s = gj % ST, pb = gj % NB;
          if (!TW(3, &v_full[s], (gj / ST) & 1)) return false;
          if (!TW(4, &p_full[pb], (gj / NB) & 1)) return false;
          if (!TW(5, &o_empty[pb], ((gj / NB) & 1) ^ 1)) return false;
          tc_fence_after();
          const uint32_t pa = smem_u32(sP + pb * Cfg::P_BYTES), va = smem_u32(sV + s * Cfg::TILE_BYTES);
#pragma unroll
          for (int ks = 0; ks < 4; ++ks)
            mma_f8(tmem + NB * NMAX + pb * NMAX,
                   make_smem_desc(va + ks * 2 * Cfg::PAGE_BYTES, Cfg::PAGE_BYTES, 128, kSwzNone),
                   make_smem_desc(pa + ks * 256, 128, 1024, kSwzNone), make_idesc(0, 0, 128, NMAX), ks > 0);
          mma_commit(&o_full[pb]);
          mma_commit(&v_empty[s]);
          return true;
        };
        for (int i = 0; i < n && ok; ++i) {
          const int gi = g + i, s = gi % ST, sb = gi % NB;
          if (!TW(1, &k_full[s], (gi / ST) & 1)) { ok = false; break; }
          if (!TW(2, &s_empty[sb], ((gi / NB) & 1) ^ 1)) { ok = false; break; }
          tc_fence_after();
          const uint32_t ka = smem_u32(sK + s * Cfg::TILE_BYTES);
#pragma unroll
          for (int ks = 0; ks < D / 32; ++ks)
            mma_f8(tmem + sb * NMAX, make_smem_desc(ka + ks * 256, 128, 8 * D, kSwzNone),
                   make_smem_desc(q_addr + ks * 256, 128, 8 * D, kSwzNone), make_idesc(0, 0, 128, NMAX), ks > 0);
          mma_commit(&s_full[sb]);
          mma_commit(&k_empty[s]);
          if (i > 1) ok = issue_pv(gi - 2);
        }
        if (ok && n > 1) ok = issue_pv(g + n - 2);
        if (ok) ok = issue_pv(g + n - 1);
        if (ok) mma_commit(&q_empty[item_it & 1]);
      }
    } else if (Cfg::V_WARP && warp == 10) {
      if (lane < 16) load_values(lane, 0x0000FFFFu);
      __syncwarp();
    } else {
      // -------------------------------------------------------------- softmax (thread = key position) and
      //                                                                accumulate (thread = output dimension)
      const int qd = warp & 3;
      const int set = (warp - 2) >> 2;                     // two softmax warp sets take alternate tiles
      const int t = qd * 32 + lane;
      const uint32_t lane_bits = (uint32_t)(qd * 32) << 16;
      float m_run[RMAX], l_part[RMAX], acc[RMAX];
#pragma unroll
      for (int i = 0; i < RMAX; ++i) { m_run[i] = -INFINITY; l_part[i] = 0.f; acc[i] = 0.f; }
      bool ok = true;
      const int qb = item_it & 1;
      if (!TW(6, &q_full[qb], (item_it >> 1) & 1)) break;     // per-row constants are published with Q
      // add tile gj's O^T (relative to this set's row maxima at tile gj) to the running sums
      auto fold = [&](int gj) -> bool {
        const int ob = gj % NB;
        if (!TW(9, &o_full[ob], (gj / NB) & 1)) return false;
        tc_fence_after();
        // only the first RMAX columns hold live rows: a plain decode step reads 4 of the 16
        float o[RMAX];
        tmem_rows<RMAX>(tmem + NB * NMAX + ob * NMAX + lane_bits, o);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&o_empty[ob]);
#pragma unroll
        for (int r = 0; r < RMAX; ++r) acc[r] += o[r];
        return true;
      };
      // All rows are computed, dead ones (beyond nrows: their Q rows are zero) too: nothing of them is written.
      const int first_new = ctx - qlen;                  // keys before it are visible to every row
      int last = -1;
      for (int i = set; i < n && ok; i += 2) {
        const int gi = g + i, sb = gi % NB;
        if (!TW(7, &s_full[sb], (gi / NB) & 1)) { ok = false; break; }
        tc_fence_after();
        float x[RMAX];
        tmem_rows<RMAX>(tmem + sb * NMAX + lane_bits, x);
        const int key0 = (t0 + i) * 128, key = key0 + t;
#pragma unroll
        for (int r = 0; r < RMAX; r += VW) {
          float c[VW];
          load_some<VW>(&s_c[qb][r], c);
#pragma unroll
          for (int k = 0; k < VW; ++k) x[r + k] *= c[k];
        }
        if (key0 + 127 >= first_new) {
#pragma unroll
          for (int r = 0; r < RMAX; ++r) {
            bool vis = key <= s_pos[qb][r];
            if constexpr (RMAX > 4) {
              // tree verify: among the sequence's own new tokens (keys from ctx - qlen on) a row sees its ancestors only
              // (a word covers the first 32 new tokens; plain causal rows - no tree mask - may be longer and are not masked)
              const int j = key - first_new;
              if (p.tree_mask != nullptr && j >= 0 && j < 32) vis = vis && ((s_mask[qb][r] >> j) & 1u);
            }
            if (!vis) x[r] = -INFINITY;
          }
        }
        float wm[RMAX];
#pragma unroll
        for (int r = 0; r < RMAX; ++r) wm[r] = warp_max_redux(x[r]);
        if (lane == 0) {
#pragma unroll
          for (int r = 0; r < RMAX; r += VW) {
            if constexpr (VW == 4) *reinterpret_cast<float4*>(&s_wmax[sb][qd][r]) = make_float4(wm[r], wm[r + 1], wm[r + 2], wm[r + 3]);
            else *reinterpret_cast<float2*>(&s_wmax[sb][qd][r]) = make_float2(wm[r], wm[r + 1]);
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&wm_bar[sb]);
        // fold this set's previous tile while the other warps of the set catch up
        if (last >= 0 && !fold(last)) { ok = false; break; }
        if (!TW(8, &wm_bar[sb], (gi / NB) & 1)) { ok = false; break; }
        // A row may see no key so far (an earlier chain row when the new tokens straddle a tile boundary): its maximum stays
        // -inf, and 0 stands for it in the differences.
        bool grew = false;
#pragma unroll
        for (int r = 0; r < RMAX; r += VW) {
          float m[VW];
          load_some<VW>(&s_wmax[sb][0][r], m);
#pragma unroll
          for (int k = 1; k < 4; ++k) {
            float o[VW];
            load_some<VW>(&s_wmax[sb][k][r], o);
#pragma unroll
            for (int j = 0; j < VW; ++j) m[j] = fmaxf(m[j], o[j]);
          }
#pragma unroll
          for (int j = 0; j < VW; ++j) { wm[r + j] = m[j]; grew |= m[j] > m_run[r + j]; }
        }
        if (grew) {                                      // the same in every warp of the set
#pragma unroll
          for (int r = 0; r < RMAX; ++r) {
            const float m_new = fmaxf(m_run[r], wm[r]);
            wm[r] = ex2(m_run[r] - (m_new == -INFINITY ? 0.f : m_new));     // ex2(-inf) = 0 on the first visible keys
            acc[r] *= wm[r];
            m_run[r] = m_new;
          }
        } else {
#pragma unroll
          for (int r = 0; r < RMAX; ++r) wm[r] = 1.f;
        }
        uint8_t* pdst = sP + sb * Cfg::P_BYTES + (t >> 4) * 128 + (t & 15);
#pragma unroll
        for (int r = 0; r < RMAX; r += 2) {
          const float ma = m_run[r] == -INFINITY ? 0.f : m_run[r], mb = m_run[r + 1] == -INFINITY ? 0.f : m_run[r + 1];
          const float pa = ex2(x[r] - ma + 8.f), pb = ex2(x[r + 1] - mb + 8.f);      // masked keys: ex2(-inf) = 0; P scaled by 2^8
          l_part[r] = fmaf(l_part[r], wm[r], pa);
          l_part[r + 1] = fmaf(l_part[r + 1], wm[r + 1], pb);
          const uint32_t two = __nv_cvt_float2_to_fp8x2(make_float2(pa, pb), __NV_SATFINITE, __NV_E4M3);
          pdst[(r >> 3) * 1024 + (r & 7) * 16] = (uint8_t)two;
          pdst[(r >> 3) * 1024 + (r & 7) * 16 + 16] = (uint8_t)(two >> 8);
        }
        fence_async_smem();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) { mbar_arrive(&s_empty[sb]); mbar_arrive(&p_full[sb]); }
        last = gi;
      }
      if (ok && last >= 0) ok = fold(last);
      if (!ok) break;
      // ---- merge the two sets and the four warps of each: row sums, maxima, output sums
      // the exchange buffers are single: set 1 writes them only after set 0 has read the previous item's
      if (set == 1 && !TW(11, acc_free, (item_it & 1) ^ 1)) break;
      constexpr int RP = RMAX == 12 ? 16 : RMAX;           // (a power of two)
      float lp[RP];
#pragma unroll
      for (int r = 0; r < RP; ++r) lp[r] = r < RMAX ? l_part[r < RMAX ? r : 0] : 0.f;
      const float ls = sum_rows<RP>(lp, lane);
      if (const int lr = row_of_lane<RP>(lane); lr >= 0 && lr < RMAX) s_l[set][qd][lr] = ls;
      if (t == 0) {
#pragma unroll
        for (int r = 0; r < RMAX; ++r) s_m[set][r] = m_run[r];
      }
      if (set == 1) {
#pragma unroll
        for (int r = 0; r < RMAX; ++r) s_acc[r][t] = acc[r];
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(fin_bar);
      if (!TW(11, fin_bar, item_it & 1)) break;
      if (set == 0) {
        // Lane r works out what row r needs, once per warp: the code per row and thread stays short.  (It runs once per item and
        // does not stay in the instruction caches: divisions and exponentials unrolled per row took longer than the tiles.)
        if (lane < RMAX) {
          const int r = lane;
          const float ma = s_m[0][r], mb = s_m[1][r];
          const float m = fmaxf(ma, mb);
          // (a set that saw no visible key of the row has maximum -inf and contributes nothing)
          const float fa = ma == -INFINITY ? 0.f : ex2(ma - m), fb = mb == -INFINITY ? 0.f : ex2(mb - m);
          const float l = (s_l[0][0][r] + s_l[0][1][r] + s_l[0][2][r] + s_l[0][3][r]) * fa +
                          (s_l[1][0][r] + s_l[1][1][r] + s_l[1][2][r] + s_l[1][3][r]) * fb;
          s_div[qd][r] = l;
          if (p.splits == 1) {
            const int tq = (row0 + r) / group;
            s_off[qd][r] = (r0 + tq) * p.Hq + kh * group + (row0 + r - tq * group);
          } else {
            s_off[qd][r] = w * NMAX + r;
            if (qd == 0 && r < nrows) put_pair(&p.part_ml[((size_t)w * NMAX + r) * 2], m, l);
          }
          s_f[qd][r] = make_float2(fa, fb);
        }
        __syncwarp();
#pragma unroll
        for (int r = 0; r < RMAX; ++r) {
          const float2 f = s_f[qd][r];
          const float o = acc[r] * f.x + s_acc[r][t] * f.y;
          const size_t at = (size_t)s_off[qd][r] * D + t;
          if (r < nrows) {
            const float l = s_div[qd][r];
            if (p.splits == 1) p.out[at] = __float2bfloat16(l > 0.f ? o * p.v_scale / l : 0.f);
            else p.part_o[at] = o;
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(acc_free);
      }
    }
    g += n;
    ++item_it;
    if (*abort_flag) break;
  }
#undef TW
  if (prof && lane == 0) {
    pc[12] += clock64();
    for (int i = 0; i < 13; ++i) p.prof[((size_t)blockIdx.x * 3 + warp) * 16 + i] = pc[i];
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, Cfg::TMEM_COLS);
  }
}

// Merge an item's runs: one block per (sequence, kv head, row block), a warp per row, four dims per lane.  The lanes weigh the runs
// side by side, and the runs' sums are added up (in their order) by loads that do not wait for one another; with a thread per
// dim, a row after the other and a branch around every run it took 10.5 us for 48 items of 8 runs, now 5.3.
// WIDE: the caller's arrays and output lie on 16 bytes (else they are read and written by elements).
template <bool WIDE>
__global__ void __launch_bounds__(512) attn_decode_combine_kernel(AttnParams p) {
  pdl_trigger();
  pdl_wait();
  constexpr int D = 128;
  const int rb = blockIdx.x % p.row_blocks;
  const int kh = (blockIdx.x / p.row_blocks) % p.Hkv;
  const int b = blockIdx.x / (p.row_blocks * p.Hkv);
  const int group = p.Hq / p.Hkv;
  const int r0 = p.q_start[b], qlen = p.q_start[b + 1] - r0;
  const int rows_total = qlen * group;
  if (rows_total < p.min_rows || rows_total > p.max_rows) return;
  const int row0 = rb * NMAX, nrows = min(NMAX, rows_total - row0);
  const int lane = threadIdx.x & 31;
  for (int r = threadIdx.x >> 5; r < nrows; r += blockDim.x >> 5) {
    auto at = [&](int i) { return ((size_t)blockIdx.x * p.splits + i) * NMAX + r; };
    auto max_sum = [&](int i) {
      const float* ml = &p.part_ml[at(i < p.splits ? i : 0) * 2];
      const float2 v = WIDE ? *reinterpret_cast<const float2*>(ml) : make_float2(ml[0], ml[1]);
      return i < p.splits ? v : make_float2(-INFINITY, 0.f);
    };
    float m = -INFINITY, l = 0.f;
    for (int i = lane; i < p.splits; i += 32) { const float2 ml = max_sum(i); if (ml.y > 0.f) m = fmaxf(m, ml.x); }
    m = warp_max(m);
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int i0 = 0; i0 < p.splits; i0 += 32) {
      const float2 ml = max_sum(i0 + lane);
      const float mine = ml.y > 0.f ? exp2f(ml.x - m) : 0.f, sum = ml.y > 0.f ? ml.y : 0.f;
      const int here = min(32, p.splits - i0);
#pragma unroll 8
      for (int i = 0; i < here; ++i) {
        const float f = __shfl_sync(0xffffffffu, mine, i), ls = __shfl_sync(0xffffffffu, sum, i);
        // (a run without a visible key has written no outputs; one whose sum is not a number, for a key that is none, does not count)
        const float* po = &p.part_o[at(i0 + i) * D + lane * 4];
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (ls > 0.f) x = WIDE ? *reinterpret_cast<const float4*>(po) : make_float4(po[0], po[1], po[2], po[3]);
        l = fmaf(ls, f, l);
        o.x = fmaf(x.x, f, o.x); o.y = fmaf(x.y, f, o.y); o.z = fmaf(x.z, f, o.z); o.w = fmaf(x.w, f, o.w);
      }
    }
    const int R = row0 + r, tq = R / group, hq = kh * group + R % group;
    auto fin = [&](float v) { return l > 0.f ? v * p.v_scale / l : 0.f; };
    __nv_bfloat16* dst = &p.out[((size_t)(r0 + tq) * p.Hq + hq) * D + lane * 4];
    if constexpr (WIDE) {
      *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16x2(fin(o.x), fin(o.y)), pack_bf16x2(fin(o.z), fin(o.w)));
    } else {
      const float v[4] = {fin(o.x), fin(o.y), fin(o.z), fin(o.w)};
#pragma unroll
      for (int j = 0; j < 4; ++j) dst[j] = __float2bfloat16(v[j]);
    }
  }
}

template <typename Cfg, typename K>
static cudaError_t launch_form(K kernel, PerDeviceOnce& configured, const AttnParams& p, int max_ctas, cudaStream_t stream) {
  cudaError_t e = configured.smem_limit(kernel, Cfg::SMEM);
  if (e != cudaSuccess) return e;
  const int items = p.num_items * p.Hkv * p.row_blocks, cap = Cfg::CTAS_PER_SM * sm_count();
  int grid = items * p.splits < cap ? items * p.splits : cap;
  if (max_ctas > 0 && grid > max_ctas) grid = max_ctas;
  e = launch_pdl(kernel, dim3(grid), dim3(Cfg::THREADS), Cfg::SMEM, stream, p);
  if (e != cudaSuccess || p.splits == 1) return e;
  const bool wide = !((reinterpret_cast<uintptr_t>(p.part_o) | reinterpret_cast<uintptr_t>(p.part_ml) | reinterpret_cast<uintptr_t>(p.out)) & 15);
  return launch_pdl(wide ? attn_decode_combine_kernel<true> : attn_decode_combine_kernel<false>, dim3(items), dim3(p.max_rows <= 4 ? 128 : p.max_rows <= 8 ? 256 : 512), 0, stream, p);
}

// The most rows of any work item choose the kernel (16 rows an item).  Draft trees need the mask that those of up to 4 rows leave out.
// Rows that no query has are computed, too, so there are forms for the numbers of rows that heads and short chains make: with those of
// 4, 8 and 16 rows alone, 256 sequences of 1.2 K tokens with 8 kv heads of 9 rows took 310 us instead of 251 by loops over the live
// rows (now 204), 16 of 1.1 K with 8 kv heads of 1 row 21.1 instead of 19.6 (now 20.1).
template <int RMAX>
static cudaError_t launch_rows(const AttnParams& p, int max_ctas, cudaStream_t stream) {
  static PerDeviceOnce configured;
  return launch_form<DecCfg<RMAX>>(attn_decode_kernel<RMAX>, configured, p, max_ctas, stream);
}
static cudaError_t launch_decode(const AttnParams& p, int max_ctas, cudaStream_t stream) {
  if (p.max_rows <= 2 && !p.tree_mask) return launch_rows<2>(p, max_ctas, stream);
  if (p.max_rows <= 4 && !p.tree_mask) return launch_rows<4>(p, max_ctas, stream);
  if (p.max_rows <= 8) return launch_rows<8>(p, max_ctas, stream);
  if (p.max_rows <= 12) return launch_rows<12>(p, max_ctas, stream);
  return launch_rows<16>(p, max_ctas, stream);
}

}  // namespace blz

// Decode / verify attention for every sequence with min_rows <= q_len * (Hq / Hkv) <= max_rows.
// nmax: 16 or 32; row_blocks = ceil(max rows of any processed sequence / nmax).  (Work items have 16 rows either way.)
// Scratch for splits > 1: part_o = B*Hkv*row_blocks*splits*nmax*128 floats, part_ml = ...*nmax*2 floats.
// tree_mask (optional, [T] int32, indexed like q's rows): bit j of row i's word = row i may attend to the j-th new token
// of its sequence (itself and its ancestors in a draft tree; at most 32 new tokens per sequence).  Null = causal rows.
// Plain decode work items (at most 4 live rows per KV head) ignore it: a single new token sees only itself.
BLZ_API int blz_attn_decode_tree(const void* q, void* out, const void* pool, const int* block_table, const int* slots,
                            const int* q_start, const int* ctx_len, int num_seqs, int Hq, int Hkv, int D, int bt_stride, long long page_stride, long long head_stride,
                            float scale, float k_scale, float v_scale, int nmax, int row_blocks, int min_rows,
                            int max_rows, int splits, float* part_o, float* part_ml, int max_ctas, long long* prof,
                            const int* tree_mask, cudaStream_t stream) {
  using namespace blz;
  if (num_seqs <= 0) return 0;
  if (D != 128 || Hq % Hkv || (nmax != 16 && nmax != 32) || row_blocks < 1 || splits < 1 ||
      (splits > 1 && (!part_o || !part_ml)))
    return (int)cudaErrorInvalidValue;
  // every processed sequence has at most max_rows rows per kv head: the row blocks must cover them, or rows would be skipped
  if (max_rows < (1 << 29) && (long long)row_blocks * nmax < max_rows) return (int)cudaErrorInvalidValue;
  AttnParams p;
  p.q = (const __nv_bfloat16*)q; p.out = (__nv_bfloat16*)out; p.pool = (const uint8_t*)pool;
  p.page_stride = page_stride > 0 ? page_stride : (long long)Hkv * 2 * 16 * D;
  p.head_stride = head_stride > 0 ? head_stride : (long long)2 * 16 * D;
  p.block_table = block_table; p.slots = slots; p.q_start = q_start; p.ctx_len = ctx_len;
  p.item_seq = nullptr; p.item_q0 = nullptr; p.part_o = part_o; p.part_ml = part_ml;
  p.num_items = num_seqs; p.Hq = Hq; p.Hkv = Hkv; p.bt_stride = bt_stride; p.splits = splits;
  p.scale_log2 = scale * 1.4426950408889634f * k_scale; p.v_scale = v_scale;
  p.tokens_per_block = 0; p.min_rows = min_rows; p.max_rows = max_rows; p.row_blocks = row_blocks * (nmax / 16);
  p.status = status_word();
  p.prof = prof;
  p.tree_mask = tree_mask;
  return (int)launch_decode(p, max_ctas, stream);
}

BLZ_API int blz_attn_decode(const void* q, void* out, const void* pool, const int* block_table, const int* slots,
                            const int* q_start, const int* ctx_len, int num_seqs, int Hq, int Hkv, int D, int bt_stride, long long page_stride, long long head_stride,
                            float scale, float k_scale, float v_scale, int nmax, int row_blocks, int min_rows,
                            int max_rows, int splits, float* part_o, float* part_ml, int max_ctas, long long* prof,
                            cudaStream_t stream) {
  return blz_attn_decode_tree(q, out, pool, block_table, slots, q_start, ctx_len, num_seqs, Hq, Hkv, D, bt_stride, page_stride,
                              head_stride, scale, k_scale, v_scale, nmax, row_blocks, min_rows, max_rows, splits, part_o, part_ml,
                              max_ctas, prof, nullptr, stream);
}

// ------------------------------------------------------------------------------------------------------------------
// Allocation-free variant (see blaze/attn_noalloc.h): the split-KV partials live in a library-owned device array.
#include <cstdio>
#include <mutex>

#include "blaze/attn_noalloc.h"

namespace {
// partial outputs [work][16][128] floats followed by (max, sum) pairs [work][16][2] floats
static __device__ __align__(256) unsigned char g_noalloc_scratch[BLZ_ATTN_NOALLOC_SCRATCH_BYTES];
static __device__ int g_noalloc_status;

struct NoAllocDev {
  bool ready = false;
  float* scratch = nullptr;     // device address of g_noalloc_scratch on that device
  int* status = nullptr;
};
NoAllocDev g_noalloc_dev[64];
std::mutex g_noalloc_mu;          // guards the first-call set-up of a device
thread_local char g_noalloc_err[256] = "";
}  // namespace

// Reads and clears the status word that blz_attn_decode_noalloc's kernels report into on the current device (0 = fine,
// 1 = a bounded wait inside the kernel ran out and the call's output is not valid).  Synchronises the device; returns -1
// when no call has been made on this device yet or the copy fails.  Allocates nothing.
extern "C" __attribute__((visibility("default"))) int blz_attn_decode_noalloc_status(void) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -1;
  {
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_dev[dev].ready) return -1;
  }
  int h = 0;
  if (cudaMemcpyFromSymbol(&h, g_noalloc_status, sizeof(int)) != cudaSuccess) return -1;
  if (h != 0) {
    const int zero = 0;
    if (cudaMemcpyToSymbol(g_noalloc_status, &zero, sizeof(int)) != cudaSuccess) return -1;
  }
  return h;
}

extern "C" __attribute__((visibility("default"))) const char* blz_attn_decode_noalloc_error(void) { return g_noalloc_err; }

extern "C" __attribute__((visibility("default"))) long long blz_attn_decode_noalloc_bytes(int num_seqs, int Hkv, int row_blocks,
                                                                                          int splits) {
  const long long work = (long long)num_seqs * Hkv * row_blocks * splits;
  return work * 16 * (128 + 2) * (long long)sizeof(float);
}

extern "C" __attribute__((visibility("default"))) int blz_attn_decode_noalloc(
    const void* q, void* out, const void* pool, const int* block_table, const int* slots, const int* q_start, const int* ctx_len,
    int num_seqs, int Hq, int Hkv, int D, int bt_stride, long long page_stride, long long head_stride, float scale, float k_scale, float v_scale, int row_blocks, int min_rows,
    int max_rows, int splits, int max_ctas, cudaStream_t stream) {
  using namespace blz;
  g_noalloc_err[0] = 0;
  if (num_seqs <= 0) return 0;
  if (D != 128 || Hkv <= 0 || Hq % Hkv || row_blocks < 1 || splits < 1) {
    snprintf(g_noalloc_err, sizeof(g_noalloc_err), "unsupported shape: head_dim %d, heads %d/%d, row_blocks %d, splits %d", D, Hq,
             Hkv, row_blocks, splits);
    return (int)cudaErrorInvalidValue;
  }
  if (max_rows < (1 << 29) && (long long)row_blocks * 16 < max_rows) {
    snprintf(g_noalloc_err, sizeof(g_noalloc_err), "row_blocks %d x 16 rows do not cover max_rows %d: rows would be skipped",
             row_blocks, max_rows);
    return (int)cudaErrorInvalidValue;
  }
  const long long need = blz_attn_decode_noalloc_bytes(num_seqs, Hkv, row_blocks, splits);
  if (splits > 1 && need > (long long)BLZ_ATTN_NOALLOC_SCRATCH_BYTES) {
    snprintf(g_noalloc_err, sizeof(g_noalloc_err),
             "split-KV scratch of %lld bytes (%d seqs x %d kv heads x %d row blocks x %d splits) exceeds the built-in %u bytes; "
             "use fewer splits or blz_attn_decode with caller-owned scratch",
             need, num_seqs, Hkv, row_blocks, splits, (unsigned)BLZ_ATTN_NOALLOC_SCRATCH_BYTES);
    return (int)cudaErrorInvalidValue;
  }
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= 64) {
    snprintf(g_noalloc_err, sizeof(g_noalloc_err), "cudaGetDevice failed (%d)", (int)e);
    return (int)(e != cudaSuccess ? e : cudaErrorInvalidDevice);
  }
  NoAllocDev& d = g_noalloc_dev[dev];
  std::unique_lock<std::mutex> setup_lock(g_noalloc_mu);
  if (!d.ready) {
    // first call on this device, with this device current: resolve the device addresses of the library-owned arrays.
    // In host code the array names are host-side stand-ins, never device pointers.
    void* p_scratch = nullptr;
    void* p_status = nullptr;
    e = cudaGetSymbolAddress(&p_scratch, g_noalloc_scratch);
    if (e == cudaSuccess) e = cudaGetSymbolAddress(&p_status, g_noalloc_status);
    if (e != cudaSuccess) {
      snprintf(g_noalloc_err, sizeof(g_noalloc_err), "cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
      return (int)e;
    }
    d.scratch = reinterpret_cast<float*>(p_scratch);
    d.status = reinterpret_cast<int*>(p_status);
    d.ready = true;
  }
  setup_lock.unlock();
  AttnParams p;
  p.q = (const __nv_bfloat16*)q; p.out = (__nv_bfloat16*)out; p.pool = (const uint8_t*)pool;
  p.page_stride = page_stride > 0 ? page_stride : (long long)Hkv * 2 * 16 * D;
  p.head_stride = head_stride > 0 ? head_stride : (long long)2 * 16 * D;
  p.block_table = block_table; p.slots = slots; p.q_start = q_start; p.ctx_len = ctx_len;
  p.item_seq = nullptr; p.item_q0 = nullptr;
  const long long work = (long long)num_seqs * Hkv * row_blocks * splits;
  p.part_o = d.scratch;
  p.part_ml = d.scratch + work * 16 * 128;
  p.num_items = num_seqs; p.Hq = Hq; p.Hkv = Hkv; p.bt_stride = bt_stride; p.splits = splits;
  p.scale_log2 = scale * 1.4426950408889634f * k_scale; p.v_scale = v_scale;
  p.tokens_per_block = 0; p.min_rows = min_rows; p.max_rows = max_rows; p.row_blocks = row_blocks;
  p.status = d.status;
  p.prof = nullptr;
  e = launch_decode(p, max_ctas, stream);
  if (e != cudaSuccess) snprintf(g_noalloc_err, sizeof(g_noalloc_err), "launch failed: %s", cudaGetErrorString(e));
  return (int)e;
}
