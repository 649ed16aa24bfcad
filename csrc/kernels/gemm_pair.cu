// GEMM on CTA pairs, for any number of rows, and experts' products:  C[tokens, features] = X[tokens, K] · W[features, K]^T.
//
// A pair (a cluster of two CTAs on neighbouring SMs) computes 256 features x up to 256 tokens with one tcgen05.mma.cta_group::2 per
// K step: features are the MMA lanes (128 in each CTA), tokens its columns, half of their rows in either CTA's shared memory.  Per 128
// bytes of K an SM so fetches 16 KB of weights and at most 16 KB of activations, where a CTA by itself fetches 16 + 32 KB for a tile of
// the same work (128 x 256): the path from L2 to shared memory, about 64 bytes per clock and SM, is what bounds these products, not
// the tensor pipe.  Tokens as columns: a tile is as wide as the rows need (a multiple of 64), features are whole tiles in practice.
//
// Two accumulators per CTA, so that the epilogue of a tile runs beside the next tile's MMAs.  Scale factors of the block-scaled kinds take
// 48 (NVFP4) or 12 columns of tensor memory (copied anew for every stage: copies and MMAs of one issuer run in order), so at 256
// columns the two accumulators share as many: the epilogue reads the shared ones first, and the next tile waits for those alone.
//
// Few tiles and a long K: a cluster of up to four pairs shares a tile's K, and the CTAs of one rank exchange their partial sums through
// distributed shared memory (each owns some columns and adds the parts up in the pairs' order, so results do not depend on timing).
//
// Few tokens: tiles of 64 or 128 columns take less of a stage, so that more of a weight that is read once is in flight (NVFP4 x 4096 x
// 4096, 64 rows 12.7 -> 9.1 us); where MMAs are short (64 columns, experts) a stage holds two K blocks, since its waits and commits cost
// some 450 clocks.  Experts: a tile is a run of one expert's routed rows.
//
// 448 threads: warp 0 = TMA producer (one per CTA, its own half of the tile), warp 1 = MMA issuer (first CTA of the pair only), warps
// 2-13 = epilogue.  Persistent, one pair per two SMs.  Barriers: `full` lives in the first CTA and counts both CTAs' bytes; `empty` and
// `acc_full` are in both and raised by multicast commits; `acc_early` and `acc_free` are in the first and count both CTAs' epilogue
// warps.  Every wait is bounded; the hardware cluster barrier is used at the start and, by all threads, at the end.  No load is multicast.
//
// Measured against one CTA per tile of 128 x 256 (gemm_wide.cu, gemm_tc.cu; back to back in a graph, inputs from memory): 8192 rows, NVFP4
// x 4096 x 12288 177 -> 126 us (6.6 PFLOP/s), x 6144 x 4096 115 -> 75, x 24576 x 4096 with the gated activation 380 -> 306; bf16 x
// 6144 x 4096 328 -> 249; MXFP8 x 12352 x 2048 266 -> 142.  In a long run the chip's power limit takes a part of that back.  What the
// stages of the loop cost: of an NVFP4 K block at 256 columns (360 ns) the MMAs and scale copies alone need 350.  One thread that built
// each descriptor anew issued a block in 330 ns whatever its columns (gated 371 -> 350 us).  Arrivals that release global stores to the
// cluster made every warp wait for its stores twice per tile, some 1200 clocks each, and 64-bit addresses and exchanges per store
// another 1800 per 32 columns, so that short tiles hung on the epilogue (gated 350 -> 309 us, K 512 x 2048 27.5 -> 16.6).  Twelve
// epilogue warps: eight did not keep up with a gated tile, sixteen have too few registers.
//
// Counterpart in the reference: the tiled kernels of kernels/src/cuda/nvfp4_gemm.cu.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <atomic>

#include "blaze/glu.cuh"
#include "blaze/host.h"
#include "blaze/sm100.cuh"

namespace blz {

bool gemm_oneshot_take_unsupported();   // gemm_tc.cu

struct PairParams {
  int M, N, K;                // tokens, features, elements
  void* C;                    // [tokens, ldc] bf16 or fp32
  long long ldc;
  int out_f32;
  const float* row_scale;     // per token, or null
  const float* alpha;         // per feature, or null
  const __nv_bfloat16* bias;  // per feature, or null
  int sf_col_tiles;           // 4-column scale tiles per 128-row tile
  int cn;                     // columns (tokens) of a tile
  int ks;                     // pairs that share a tile's K (split kernel), else 1
  int acc1;                   // first tensor-memory column of the second accumulator
  const int4* heads;          // experts (grouped kernel): [0].x = number of tiles, then {first row, live rows, expert, 0} of each
  int act;                    // 1, 2: rows of W are [16 gate | 16 up] groups; C = gated activation, bf16 [tokens, N/2]
  float act_limit;            // act 2: the clamp of glu.cuh
  int* status;
};

template <int KIND> struct PKind;
template <> struct PKind<0> { static constexpr int KMMA = 16, SF_ATOMS = 0; };
template <> struct PKind<1> { static constexpr int KMMA = 64, SF_ATOMS = 4; };
template <> struct PKind<2> { static constexpr int KMMA = 32, SF_ATOMS = 1; };

// MODE: one weight, the routed rows of several experts, or one weight with K split over the pairs of a cluster.
enum { kPairDense = 0, kPairExperts = 1, kPairSplit = 2 };

// CN: most columns of a tile (64, 128 or 256).  Narrow tiles leave room for more stages: what a weight that is read once needs.
template <int KIND, int CN, int MODE>
struct PairCfg {
  static constexpr int KMMA = PKind<KIND>::KMMA;
  static constexpr int BK = KMMA * 4;                       // 128 bytes of K per row and stage
  static constexpr int SF_ATOMS = PKind<KIND>::SF_ATOMS;
  static constexpr int A_BYTES = 128 * 128, B_BYTES = CN * 64;
  static constexpr int GROUPS = CN > 128 ? 2 : 1;           // 128-row scale tiles under a tile's tokens
  static constexpr int SF_BYTES = SF_ATOMS * 512;           // scales of 128 rows and one stage
  // K blocks per stage.  Waits and commits cost as much as the products of 64 columns (one / two blocks: NVFP4 64 x 4096 x 12288 17.3 / 15.1
  // us, MXFP8 64 x 2048 x 4096 12.5 / 10.7); at 128 the stages are worth more (17.6 / 18.4, bf16 45 / 48), but for experts, whose tiles
  // are mostly not full (512 MXFP8 experts, both products of 256 tokens 314 / 307).
  static constexpr int UB = CN == 64 || (CN == 128 && MODE == kPairExperts) ? 2 : 1;
  static constexpr int STAGE_BYTES = UB * (A_BYTES + B_BYTES + (1 + GROUPS) * SF_BYTES);
  static constexpr int STAGES = (216 * 1024) / STAGE_BYTES;
  static constexpr int SF_COLS = SF_ATOMS * 4 * 3;
  static constexpr int SF_COL0 = 512 - SF_COLS;
  static constexpr int SMEM = STAGES * STAGE_BYTES + 1024 + 512 + 2 * 256 * 4;
  static constexpr int EPI = 12;                            // epilogue warps
  static constexpr int THREADS = 64 + EPI * 32;
  static_assert((2 * STAGES + 9) * 8 + 8 <= 512 && STAGES <= 32 && SMEM <= 227 * 1024, "shared memory");
  static_assert(SF_COLS <= 64, "the accumulators may share two chunks of 32 columns at most");
};

// (x * s) * a + b of two neighbours at once, each rounded as by fmaf(x * s, a, b): token scale first, as in gemm_tc.cu; the narrow kernel
// of moe_gemm.cu multiplies by the feature's first, which may round the other way
__device__ __forceinline__ void scale_pair(uint32_t x0, uint32_t x1, float s0, float s1, float a, float b, float& y0, float& y1) {
  asm("{\n\t.reg .b64 x, s, a, b;\n\t"
      "mov.b64 x, {%2, %3};\n\tmov.b64 s, {%4, %5};\n\tmov.b64 a, {%6, %6};\n\tmov.b64 b, {%7, %7};\n\t"
      "mul.rn.f32x2 x, x, s;\n\tfma.rn.f32x2 x, x, a, b;\n\tmov.b64 {%0, %1}, x;\n\t}\n"
      : "=f"(y0), "=f"(y1)
      : "r"(x0), "r"(x1), "f"(s0), "f"(s1), "f"(a), "f"(b));
}

// A tile as its roles see it.
struct PairTile {
  int frow;      // first row of W
  int feat;      // first feature
  int t0;        // first token (row of X and of C)
  int cn;        // columns: live tokens, rounded up to 64
  int end;       // first row past the live ones
  int wbase;     // first row of W of the tile's expert (0 for one weight)
};

template <int KIND, int CN, int MODE>
__global__ void __launch_bounds__(PairCfg<KIND, CN, MODE>::THREADS, 1) gemm_pair_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX,
                                                            const __grid_constant__ CUtensorMap tmSW, const __grid_constant__ CUtensorMap tmSX,
                                                            const PairParams p) {
  using Cfg = PairCfg<KIND, CN, MODE>;
  constexpr int STAGES = Cfg::STAGES, BK = Cfg::BK, ATOMS = Cfg::SF_ATOMS, UB = Cfg::UB;
  constexpr bool GROUPED = MODE == kPairExperts, SPLIT = MODE == kPairSplit;
  extern __shared__ uint8_t smem_raw[];
  // both CTAs of a pair round the same way: dynamic shared memory starts at the same offset in each
  uint8_t* base = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* sA = base;
  uint8_t* sB = sA + STAGES * UB * Cfg::A_BYTES;
  uint8_t* sSFA = sB + STAGES * UB * Cfg::B_BYTES;
  uint8_t* sSFB = sSFA + STAGES * UB * Cfg::SF_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(sSFB + STAGES * UB * Cfg::GROUPS * Cfg::SF_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* acc_full = empty + STAGES;      // [2]
  uint64_t* acc_early = acc_full + 2;       // [2] an accumulator has been read as far as the two overlap
  uint64_t* acc_free = acc_early + 2;       // [2] and altogether
  uint64_t* drain = acc_free + 2;
  uint64_t* ring_free = drain + 1;          // every CTA of the split is done with its operands (its ring may be written)
  uint64_t* part_ready = ring_free + 1;     // and has handed out its partial sums
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(part_ready + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* s_rs = reinterpret_cast<float*>(full + 64);        // [2][256] row scales of a tile's tokens (after 512 bytes of barriers)

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // warp-uniform to the compiler
  const uint32_t crank = cluster_ctarank(), rank = crank & 1, lead = crank & ~1u;       // lead: the pair's first CTA
  const int ks = SPLIT ? p.ks : 1, kp = SPLIT ? (int)(crank >> 1) : 0;                   // this pair's share of K
  const int pair = blockIdx.x / (2 * ks), pairs = gridDim.x / (2 * ks);
  const int tiles_f = (p.N + 255) / 256;
  const int k_tiles = (p.K + BK * UB - 1) / (BK * UB);      // stages along K
  const int kb0 = kp * k_tiles / ks, kb1 = (kp + 1) * k_tiles / ks;

  if (threadIdx.x == 0) {
    for (int i = 0; i < STAGES; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_early[i], 2 * Cfg::EPI); mbar_init(&acc_free[i], 2 * Cfg::EPI); }
    mbar_init(drain, 1);
    mbar_init(ring_free, ks);
    mbar_init(part_ready, ks);
    *abort_flag = 0;
    mbar_fence_init();
    prefetch_tmap(&tmW);
    prefetch_tmap(&tmX);
    if (ATOMS) { prefetch_tmap(&tmSW); prefetch_tmap(&tmSX); }
  }
  __syncwarp();
  if (warp == 1) tmem_alloc_pair(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  cluster_arrive();                         // the peer's barriers are initialised before anything signals them
  cluster_wait();
  tc_fence_after();
  pdl_trigger();        // after the allocation (sm100.cuh)
  const uint32_t tmem = *tmem_slot;
  pdl_wait();

  const int tiles_t = GROUPED ? p.heads[0].x : (p.M + p.cn - 1) / p.cn;
  const int tiles = tiles_f * tiles_t;
  // Tile u.  One weight: bands of eight token tiles, so that the pairs at work at one time share both operands in L2.  Experts: all
  // features of a run of rows, then the next.  The roles ask for a tile while they are at the one before it.
  auto tile_at = [&](int u) {
    PairTile t = {0, 0, 0, 64, 0, 0};
    if (u >= tiles) return t;
    int ft;
    if constexpr (GROUPED) {
      const int h = u / tiles_f;
      ft = u - h * tiles_f;
      const int4 e = __ldg(p.heads + 1 + h);
      t.t0 = e.x;
      t.cn = (e.y + 63) & ~63;
      t.end = t.t0 + e.y;
      t.wbase = e.z * p.N;
    } else {
      const int per_band = 8 * tiles_f, band = u / per_band, in = u - band * per_band;
      const int width = min(8, tiles_t - band * 8);
      ft = in / width;
      t.t0 = (band * 8 + in - ft * width) * p.cn;
      t.cn = p.cn;
      t.end = p.M;
    }
    t.feat = ft * 256;
    t.frow = t.wbase + t.feat;
    return t;
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ producer: this CTA's half of the operands
    if (lane == 0) {
      int s = 0; uint32_t ph = 0;
      uint32_t used = 0, last = 0;          // stages filled so far, and the parity of their latest fill
      bool ok = true;
      PairTile next = tile_at(pair);
      for (int u = pair; u < tiles && ok; u += pairs) {
        const PairTile t = next;
        next = tile_at(u + pairs);
        const int frow = t.frow + (int)rank * 128, trow = t.t0 + (int)rank * (t.cn >> 1);
        const int groups = t.cn > 128 ? 2 : 1;      // tiles of 64 and 192 may start in the middle of a scale tile, but not end past the second
        for (int kt = kb0; kt < kb1; ++kt) {
          if (!mbar_wait(&empty[s], ph ^ 1, abort_flag, p.status)) { ok = false; break; }
          const uint32_t bar = mapa_shared(smem_u32(&full[s]), lead);
          if (rank == 0) mbar_expect_tx(&full[s], 2u * UB * (Cfg::A_BYTES + (uint32_t)t.cn * 64u + (uint32_t)(1 + groups) * Cfg::SF_BYTES));
#pragma unroll
          for (int h = 0; h < UB; ++h) {         // (a block beyond K is filled with zeros and not used)
            const int kk = kt * UB + h, kc = KIND == 0 ? kk * BK : kk * 128, sh = s * UB + h;
            tma_load_2d_pair(sA + sh * Cfg::A_BYTES, &tmW, kc, frow, bar);
            if constexpr (GROUPED) {
              for (int r = 0; r < t.cn >> 1; r += 32) tma_load_2d_pair(sB + sh * Cfg::B_BYTES + r * 128, &tmX, kc, trow + r, bar);
            } else {
              tma_load_2d_pair(sB + sh * Cfg::B_BYTES, &tmX, kc, trow, bar);
            }
            if constexpr (ATOMS > 0) {
              tma_load_3d_pair(sSFA + sh * Cfg::SF_BYTES, &tmSW, 0, kk * ATOMS, frow >> 7, bar);
              tma_load_3d_pair(sSFB + sh * Cfg::GROUPS * Cfg::SF_BYTES, &tmSX, 0, kk * ATOMS, t.t0 >> 7, bar);
              if (GROUPED && Cfg::GROUPS == 2 && groups == 2)
                tma_load_3d_pair(sSFB + (sh * 2 + 1) * Cfg::SF_BYTES, &tmSX, 0, kk * ATOMS, (t.t0 >> 7) + 1, bar);
            }
          }
          used |= 1u << s;
          last = (last & ~(1u << s)) | (ph << s);
          if (++s == STAGES) { s = 0; ph ^= 1; }
        }
      }
      if (!ok && rank == 0)                 // no copy of either CTA is in flight when the pair leaves
        for (int i = 0; i < STAGES; ++i)
          if (used >> i & 1) mbar_drain(&full[i], last >> i & 1);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer of the pair.  The whole warp walks the loop, so that
    // the descriptors stay in uniform registers, and one thread issues; they are built from their lower halves, which alone change.
    if (rank == 0) {
      int s = 0; uint32_t ph = 0;
      int it = 0;
      bool ok = true;
      const bool leader = elect_one();
      const uint32_t a_lo0 = (uint32_t)desc_sw128(smem_u32(sA)), b_lo0 = (uint32_t)desc_sw128(smem_u32(sB));
      const uint32_t sa_lo0 = (uint32_t)make_smem_desc(smem_u32(sSFA), 0, 128, kSwzNone);
      const uint32_t sb_lo0 = (uint32_t)make_smem_desc(smem_u32(sSFB), 0, 128, kSwzNone);
      constexpr uint32_t OP_HI = (1024u >> 4) | 1u << 14 | (uint32_t)kSwz128 << 29, SF_HI = (128u >> 4) | 1u << 14;
      auto desc = [](uint32_t lo, uint32_t hi) { return (uint64_t)hi << 32 | lo; };
      PairTile next = tile_at(pair);
      int before = 0;                       // columns of the tile before
      for (int u = pair; u < tiles && ok; u += pairs, ++it) {
        const PairTile t = next;
        next = tile_at(u + pairs);
        const int b = it & 1;
        const uint32_t idesc = KIND == 0 ? make_idesc(1, 1, 256, t.cn) : make_idesc_bs(KIND == 1, KIND == 1, KIND == 2, 256, t.cn);
        // this accumulator has been read by the tile before the last, and where it reaches into the other one, that by the last
        if (it >= 2 && !mbar_wait_cluster(&acc_free[b], ((it >> 1) - 1) & 1, abort_flag, p.status)) { ok = false; break; }
        if (it >= 1 && (b ? before : t.cn) > p.acc1 && !mbar_wait_cluster(&acc_early[b ^ 1], ((it - 1) >> 1) & 1, abort_flag, p.status)) { ok = false; break; }
        before = t.cn;
        tc_fence_after();
        const uint32_t d = tmem + (b ? p.acc1 : 0);
        const uint32_t sfa = tmem + Cfg::SF_COL0, sfb = sfa + ATOMS * 4, sfb0 = sfb + ((t.t0 & 127) >> 5);
        for (int kt = kb0; kt < kb1; ++kt) {
          if (!mbar_wait(&full[s], ph, abort_flag, p.status)) { ok = false; break; }
          tc_fence_after();
          if (leader) {
#pragma unroll
            for (int u2 = 0; u2 < UB; ++u2) {
              const int kk = kt * UB + u2, sh = s * UB + u2;
              const int nblk = min(4, (p.K - kk * BK + Cfg::KMMA - 1) / Cfg::KMMA);
              if (nblk <= 0) break;
              const uint32_t a_lo = a_lo0 + sh * (Cfg::A_BYTES >> 4), b_lo = b_lo0 + sh * (Cfg::B_BYTES >> 4);
              if constexpr (ATOMS > 0) {
                const uint32_t sa_lo = sa_lo0 + sh * (Cfg::SF_BYTES >> 4), sb_lo = sb_lo0 + sh * (Cfg::GROUPS * Cfg::SF_BYTES >> 4);
#pragma unroll
                for (int a = 0; a < ATOMS; ++a) {
                  tmem_cp_sf_pair(sfa + a * 4, desc(sa_lo + a * 32, SF_HI));
                  tmem_cp_sf_pair(sfb + a * 8, desc(sb_lo + a * 32, SF_HI));
                }
                if (Cfg::GROUPS == 2 && t.cn > 128) {
#pragma unroll
                  for (int a = 0; a < ATOMS; ++a) tmem_cp_sf_pair(sfb + a * 8 + 4, desc(sb_lo + (ATOMS + a) * 32, SF_HI));
                }
              }
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                if (j < nblk) {
                  const uint64_t da = desc(a_lo + j * 2, OP_HI), db = desc(b_lo + j * 2, OP_HI);
                  const uint32_t acc = (kt > kb0 || u2 > 0 || j > 0) ? 1u : 0u;
                  if constexpr (KIND == 0) mma_f16_pair(d, da, db, idesc, acc);
                  else if constexpr (KIND == 1) mma_nvfp4_pair(d, da, db, idesc, sfa + j * 4, sfb0 + j * 8, acc);
                  else mma_mxf8_pair(d, da, db, idesc | make_idesc_bs(0, 0, 0, 0, 0, j, j), sfa, sfb0, acc);
                }
              }
            }
            mma_commit_pair(&empty[s], lead);
          }
          __syncwarp();
          if (++s == STAGES) { s = 0; ph ^= 1; }
        }
        if (ok && leader) mma_commit_pair(&acc_full[it & 1], lead);
        __syncwarp();
      }
      if (!ok && leader) {                  // the MMAs in flight end before their operands' memory goes
        mma_commit_pair(drain, lead);
        mbar_drain(drain, 0);
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue: lane = feature, column = token
    const int q = warp & 3, part = (warp - 2) >> 2, etid = threadIdx.x - 64;
    const uint32_t quad = (uint32_t)(q * 32) << 16;
    const bool odd = lane & 1, hi = lane >= 16;
    const uint32_t pick = odd ? 0x3276u : 0x5410u;      // even lanes: both lower halves, odd lanes: both upper halves
    bool ok = true;
    int it = 0;
    PairTile next = tile_at(pair);
    for (int u = pair; u < tiles; u += pairs, ++it) {
      const PairTile t = next;
      next = tile_at(u + pairs);
      const int b = it & 1, t0 = t.t0, cn = t.cn;
      float* rs = s_rs + b * 256;
      if (etid < cn) rs[etid] = (p.row_scale && t0 + etid < t.end) ? __ldg(p.row_scale + t0 + etid) : 1.0f;
      const int fl = (int)rank * 128 + q * 32 + lane, feat = t.feat + fl;
      const bool feat_ok = feat < p.N;
      const float al = (p.alpha && feat_ok) ? __ldg(p.alpha + t.frow + fl) : 1.0f;
      const float bs = (p.bias && feat_ok) ? bf2f(p.bias[feat]) : 0.0f;
      // sums of the columns [c, c + NC) of the tile, as they come from tensor memory: scales, bias, activation, store
      auto finish = [&](const auto& r, int c) {
        constexpr int NC = sizeof(r) / sizeof(r[0]);
        const int tc = t0 + c;              // token of the first column
        float v[NC];
#pragma unroll
        for (int j = 0; j < NC; j += 4) {
          const float4 s4 = *reinterpret_cast<const float4*>(rs + c + j);
          scale_pair(r[j], r[j + 1], s4.x, s4.y, al, bs, v[j], v[j + 1]);
          scale_pair(r[j + 2], r[j + 3], s4.z, s4.w, al, bs, v[j + 2], v[j + 3]);
        }
        if (p.out_f32) {
          float* C = reinterpret_cast<float*>(p.C) + feat;
#pragma unroll
          for (int j = 0; j < NC; ++j)
            if (feat_ok && tc + j < t.end) C[(size_t)(tc + j) * p.ldc] = v[j];
        } else if (p.act) {
          // lanes 0-15 hold the gates and 16-31 the up values of 16 features: one exchange gives the lower lanes a token and the upper
          // ones the next, a second one pairs two features per store
          const int first = tc + (odd ? 2 : 0) + (hi ? 1 : 0), left = feat_ok ? t.end - first : 0;
          __nv_bfloat16* C = reinterpret_cast<__nv_bfloat16*>(p.C) + (size_t)first * p.ldc + ((t.feat + (int)rank * 128 + q * 32) >> 1) + (lane & 14);
          const size_t step = (size_t)p.ldc * 4;
          auto gated = [&](auto act) {
#pragma unroll
            for (int j = 0; j < NC; j += 4) {
              float a[2];
#pragma unroll
              for (int k = 0; k < 2; ++k) {
                const float lo = v[j + 2 * k], up = v[j + 2 * k + 1];
                const float got = __shfl_xor_sync(0xffffffffu, hi ? lo : up, 16);
                a[k] = act(hi ? got : lo, hi ? up : got);
              }
              const uint32_t own = pack_bf16x2(a[0], a[1]);
              const uint32_t two = __byte_perm(own, __shfl_xor_sync(0xffffffffu, own, 1), pick);
              if (j < left) *reinterpret_cast<uint32_t*>(C) = two;
              C += step;
            }
          };
          if (p.act == 2) {
            gated([&](float gf, float uf) { return clamped_glu_fast(gf, uf, p.act_limit); });
          } else {
            gated([](float gf, float uf) {
              const float g = bf2f(__float2bfloat16(gf)), up = bf2f(__float2bfloat16(uf));
              return silu(g) * up;
            });
          }
        } else {
          // neighbouring lanes trade every other token so that each writes two adjacent features at once
          const int first = tc + (odd ? 1 : 0), left = feat_ok ? t.end - first : 0;
          __nv_bfloat16* C = reinterpret_cast<__nv_bfloat16*>(p.C) + (size_t)first * p.ldc + (feat & ~1);
          const size_t step = (size_t)p.ldc * 2;
#pragma unroll
          for (int j = 0; j < NC; j += 2) {
            const uint32_t own = pack_bf16x2(v[j], v[j + 1]);
            const uint32_t two = __byte_perm(own, __shfl_xor_sync(0xffffffffu, own, 1), pick);
            if (j < left) *reinterpret_cast<uint32_t*>(C) = two;
            C += step;
          }
        }
      };
      // the row scales are complete, and the warps agree on whether a wait ran out, so that none is left at a barrier
      if (!bar_red_and(1, Cfg::EPI * 32, ok)) break;
      ok = mbar_wait(&acc_full[b], (it >> 1) & 1, abort_flag, p.status);
      ok = __all_sync(0xffffffffu, ok);
      constexpr int PARTS = Cfg::EPI / 4;
      if constexpr (SPLIT) {
        // The CTAs of one rank exchange their partial sums: of the tile's groups of 16 columns pair i owns [i * ng / ks, (i + 1) * ng /
        // ks), whose sums all pairs push into its ring (free once all are done with theirs), slot [source][group][quad of columns]
        // [feature]; it adds them up in the pairs' order.  A CTA whose wait ran out still arrives, so that none waits for it.
        const int ng = cn >> 4, most = (ng + ks - 1) / ks, f = q * 32 + lane;
        if (etid == 0)
          for (int i = 0; i < ks; ++i) mbar_arrive_remote(mapa_shared(smem_u32(ring_free), 2 * i + rank));
        ok = __all_sync(0xffffffffu, mbar_wait_cluster(ring_free, 0, abort_flag, p.status)) && ok;
        if (ok) {
          tc_fence_after();
          for (int ch = part; ch < cn >> 5; ch += PARTS) {
            uint32_t r[32];
            tmem_ld32(tmem + ch * 32 + quad, r);
            tmem_ld_wait();
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int g = ch * 2 + h, owner = (g * ks + ks - 1) / ng, gl = g - owner * ng / ks;
              const uint32_t dst = mapa_shared(smem_u32(base) + (uint32_t)(((kp * most + gl) * 4 * 128 + f) * 16), 2 * owner + rank);
#pragma unroll
              for (int k = 0; k < 4; ++k)
                st_dsmem_f4(dst + k * 2048, __uint_as_float(r[h * 16 + k * 4]), __uint_as_float(r[h * 16 + k * 4 + 1]),
                            __uint_as_float(r[h * 16 + k * 4 + 2]), __uint_as_float(r[h * 16 + k * 4 + 3]));
            }
          }
        }
        fence_acq_rel_cluster();
        bar_sync(2, Cfg::EPI * 32);
        if (etid == 0)
          for (int i = 0; i < ks; ++i) mbar_arrive_remote(mapa_shared(smem_u32(part_ready), 2 * i + rank));
        ok = __all_sync(0xffffffffu, mbar_wait_cluster(part_ready, 0, abort_flag, p.status)) && ok;
        if (!ok || *abort_flag) break;
        const int g0 = kp * ng / ks, g1 = (kp + 1) * ng / ks;
        for (int g = g0 + part; g < g1; g += PARTS) {
          uint32_t r[16];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int i = 0; i < ks; ++i) {
              const float4 v = reinterpret_cast<const float4*>(base)[((i * most + g - g0) * 4 + k) * 128 + f];
              a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
            }
            r[4 * k] = __float_as_uint(a.x); r[4 * k + 1] = __float_as_uint(a.y);
            r[4 * k + 2] = __float_as_uint(a.z); r[4 * k + 3] = __float_as_uint(a.w);
          }
          finish(r, g * 16);
        }
      } else {
        if (!ok) continue;
        tc_fence_after();
        // chunks of 32 columns, a round of one per warp at a time, the end that the accumulators share first
        const int chunks = cn >> 5, rounds = (chunks + PARTS - 1) / PARTS;
        for (int i = 0; i < rounds; ++i) {
          const int ch = b ? i * PARTS + part : chunks - 1 - i * PARTS - part;
          const bool mine = ch >= 0 && ch < chunks;
          uint32_t r[32];
          if (mine) {
            tmem_ld32(tmem + (b ? p.acc1 : 0) + ch * 32 + quad, r);
            tmem_ld_wait();
          }
          if (i == 0 || i == rounds - 1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0 && i == 0) mbar_arrive_remote_tmem(mapa_shared(smem_u32(&acc_early[b]), lead));
            if (lane == 0 && i == rounds - 1) mbar_arrive_remote_tmem(mapa_shared(smem_u32(&acc_free[b]), lead));
          }
          if (!mine) break;
          finish(r, ch * 32);
        }
      }
    }
  }
  tc_fence_before();
  __syncwarp();
  cluster_arrive();                         // neither CTA leaves while the other still reads its memory or signals its barriers
  cluster_wait();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem, 512);
  }
}

template <int KIND, int CN, int MODE>
static cudaError_t launch_pair(const CUtensorMap& tmW, const CUtensorMap& tmX, const CUtensorMap& tmSW, const CUtensorMap& tmSX,
                               const PairParams& p, int tiles, int max_ctas, cudaStream_t stream) {
  using Cfg = PairCfg<KIND, CN, MODE>;
  auto kern = gemm_pair_kernel<KIND, CN, MODE>;
  static PerDeviceOnce configured;
  cudaError_t e = configured.smem_limit(kern, Cfg::SMEM);
  if (e != cudaSuccess) return e;
  int pairs = sm_count() / 2;
  if (max_ctas > 1 && pairs > max_ctas / 2) pairs = max_ctas / 2;
  if (MODE != kPairExperts && pairs > tiles) pairs = tiles;          // the experts' tiles are counted on the device
  if (MODE == kPairSplit) pairs = tiles * p.ks;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(pairs * 2));
  cfg.blockDim = dim3(Cfg::THREADS);
  cfg.dynamicSmemBytes = Cfg::SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2 * p.ks;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  // The set-up (barriers, tensor memory, tensor maps, cluster) runs while the kernel before this one ends; nothing is read before
  // pdl_wait.  With it 8b decode steps of 1, 256 and 80 rows take 1109, 2652, 1617 us, without 1146, 2688, 1674.  Fetching the first
  // weights ahead into L2 as well cost 3 % (the copy engine serves those first), and the same attribute on the norms and quantisers
  // gained 2 % at one row and lost as much elsewhere.
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_pairs() ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kern, tmW, tmX, tmSW, tmSX, p);
}

template <int MODE>
static cudaError_t launch_pair_kind(int kind, int most, const CUtensorMap& tmW, const CUtensorMap& tmX, const CUtensorMap& tmSW,
                                    const CUtensorMap& tmSX, const PairParams& p, int tiles, int max_ctas, cudaStream_t stream) {
#define BLZ_PAIR_CASE(KD, CN) \
  if (kind == KD && most <= CN) return launch_pair<KD, CN, MODE>(tmW, tmX, tmSW, tmSX, p, tiles, max_ctas, stream);
  if constexpr (MODE != kPairExperts) { BLZ_PAIR_CASE(0, 64) BLZ_PAIR_CASE(1, 64) BLZ_PAIR_CASE(2, 64) }
  BLZ_PAIR_CASE(0, 128) BLZ_PAIR_CASE(1, 128) BLZ_PAIR_CASE(2, 128)
  BLZ_PAIR_CASE(0, 256) BLZ_PAIR_CASE(1, 256) BLZ_PAIR_CASE(2, 256)
#undef BLZ_PAIR_CASE
  return cudaErrorInvalidValue;
}

static PairParams pair_params(int kind, int N, int K, void* C, long long ldc, const float* row_scale, const float* alpha, int act, float act_limit) {
  PairParams p = {};
  p.N = N; p.K = K; p.C = C; p.ldc = ldc; p.ks = 1;
  p.row_scale = row_scale; p.alpha = alpha;
  p.sf_col_tiles = kind == 1 ? (K + 63) / 64 : kind == 2 ? (K + 127) / 128 : 0;
  p.acc1 = (kind == 0 ? PairCfg<0, 256, kPairDense>::SF_COL0 : kind == 1 ? PairCfg<1, 256, kPairDense>::SF_COL0 : PairCfg<2, 256, kPairDense>::SF_COL0) - 256;
  p.act = act; p.act_limit = act_limit;
  p.status = status_word();
  return p;
}

// Clusters of `ctas` CTAs that run at the same time on the current device (whole within a GPC each; one CTA fits an SM, whatever the kind).
// 0 for all with BLAZE_GEMM_PAIR=0: products then take the kernels of single CTAs, as in a context without room for a pair.  The number is
// that of the first context that asks on a device.
int pair_cluster_room(int ctas) {
  static std::atomic<int> cache[64][9];
  static const bool off = [] { const char* e = getenv("BLAZE_GEMM_PAIR"); return e && e[0] == '0'; }();
  if (off) return 0;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || ctas < 2 || ctas > 8) return 0;
  if (cache[dev][ctas]) return cache[dev][ctas] - 1;
  auto kern = gemm_pair_kernel<1, 64, kPairSplit>;
  static PerDeviceOnce configured;
  if (configured.smem_limit(kern, PairCfg<1, 64, kPairSplit>::SMEM) != cudaSuccess) return 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(ctas * sm_count()));
  cfg.blockDim = dim3(PairCfg<1, 64, kPairSplit>::THREADS);
  cfg.dynamicSmemBytes = PairCfg<1, 64, kPairSplit>::SMEM;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned)ctas;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) return 0;
  cache[dev][ctas] = n + 1;
  return n;
}

// Columns of a tile (a multiple of 64) and pairs that share its K: the least rounds x time of a round.  Nanoseconds per K block measured at
// 8192 x 4096 x 12288 (NVFP4 and bf16, 64 columns: 64 rows; more columns than the MMAs of a block can hide behind its bytes and its issue
// cost little), a microsecond per tile for the accumulators' hand-over, and some six for the exchange of a split, which only pays where
// all clusters run at once: us of one pair per tile / of two / of three, 64 rows: NVFP4 4096 x 12288 15.1 / 14.1 / 14.5 (over a
// cluster of single CTAs 20), 4096 x 4096 8.6 / 9.9 / 10.5, bf16 4096 x 12288 41 / 32 / 31, 4096 x 4096 16.3 / 15.1 / 15.0; 16 tiles
// of 4 pairs do not fit the chip at once: 24.3.
static void pair_shape(int kind, int M, int N, int K, int* cn, int* ks) {
  static const int scaled[] = {230, 313, 338, 387}, plain[] = {195, 255, 296, 385};
  const int tiles_f = (N + 255) / 256, sms = sm_count(), pairs = sms / 2 > 0 ? sms / 2 : 1;
  const int k_tiles = (K + (kind == 0 ? 63 : kind == 1 ? 255 : 127)) / (kind == 0 ? 64 : kind == 1 ? 256 : 128);
  long best = 1L << 60;
  int best_cn = 256, best_ks = 1;
  for (int c = 256; c >= 64; c -= 64) {
    if (*cn && c != *cn) continue;
    const long tiles = (long)tiles_f * ((M + c - 1) / c);
    const long block = (kind ? scaled : plain)[c / 64 - 1];
    for (int k = 1; k <= 4 && k <= (k_tiles + 1) / 2; ++k) {
      if (*ks && k != *ks) continue;
      if (k > 1 && !*ks && (tiles * k > pairs || tiles > pair_cluster_room(2 * k))) continue;
      const long cost = k == 1 ? ((tiles + pairs - 1) / pairs) * (k_tiles * block + 1000) : (k_tiles + k - 1) / k * block + 1300 + 2000 * k + 10 * c;
      if (cost < best) { best = cost; best_cn = c; best_ks = k; }
    }
  }
  *cn = best_cn;
  *ks = best_ks;
}

}  // namespace blz

// How many clusters of `ctas` CTAs (2 - 8) run at once on the current device; for 2: whether products can take pairs at all.
BLZ_API int blz_pair_room(int ctas) { return blz::pair_cluster_room(ctas); }

// C[M, N] = X[M, K] · W[N, K]^T with the operand conventions of blz_gemm_tc (ldx / ldw in BYTES, ldc in elements).  kind: 0 bf16,
// 1 NVFP4, 2 MXFP8.  N even, or a multiple of 32 with act (bf16 out, [M, N/2]).  cn: tokens per tile, 64 / 128 / 192 / 256, and
// ks: pairs that share a tile's K, 1 - 4 (at most one per two K blocks); 0 to choose.
BLZ_API int blz_gemm_pair(int kind, const void* X, long long ldx, const void* W, long long ldw, void* C, long long ldc, int M, int N,
                          int K, const float* row_scale, const float* alpha, const void* bias, const void* sfx, const void* sfw,
                          int out_f32, int cn, int ks, int max_ctas, int act, float act_limit, cudaStream_t stream) {
  using namespace blz;
  // this kernel has no fused all-reduce / peer-wait / arg-max epilogue: a call armed for one is refused (and disarmed)
  if (gemm_oneshot_take_unsupported()) return (int)cudaErrorNotSupported;
  if (M <= 0 || N <= 0 || K <= 0 || kind < 0 || kind > 2 || cn < 0 || cn > 256 || cn % 64 || ks < 0 || ks > 4) return (int)cudaErrorInvalidValue;
  const int kmma = kind == 0 ? 16 : kind == 1 ? 64 : 32;
  if (K % kmma || (ks > 1 && ks > (K + 8 * kmma - 1) / (8 * kmma))) return (int)cudaErrorInvalidValue;
  if (kind && (!sfx || !sfw)) return (int)cudaErrorInvalidValue;
  if (act < 0 || act > 2 || (act && (out_f32 || N % 32))) return (int)cudaErrorInvalidValue;
  if (!out_f32 && ((N & 1) || (ldc & 1) || (reinterpret_cast<uintptr_t>(C) & 3))) return (int)cudaErrorInvalidValue;
  PairParams p = pair_params(kind, N, K, C, ldc, row_scale, alpha, act, act_limit);
  p.M = M; p.out_f32 = out_f32;
  p.bias = reinterpret_cast<const __nv_bfloat16*>(bias);
  if (max_ctas > 0) ks = 1;                  // a split is one round of clusters
  pair_shape(kind, M, N, K, &cn, &ks);
  p.cn = cn; p.ks = ks;
  p.acc1 = p.acc1 + 256 - p.cn < 256 ? p.acc1 + 256 - p.cn : 256;               // narrower tiles overlap less
  CUtensorMap tmW, tmX, tmSW, tmSX;
  const int es = kind == 0 ? 2 : 1;                                   // bytes per tensor-map element
  const uint64_t inner = kind == 1 ? (uint64_t)K / 2 : (uint64_t)K;
  cudaError_t e = encode_tmap(&tmW, W, es, inner, N, ldw, 128 / es, 128, 3);
  if (e == cudaSuccess) e = encode_tmap(&tmX, X, es, inner, M, ldx, 128 / es, p.cn / 2, 3);
  if (e != cudaSuccess) return (int)e;
  tmSW = tmW; tmSX = tmX;
  if (kind) {
    // with copies of 2 KB on barriers of each CTA, or a map of 256-byte rows with a load per row tile, 8192 x 4096 x 12288 in NVFP4 took
    // 275 and 166 us, so 141
    const uint32_t atoms = kind == 1 ? 4 : 1;
    e = encode_sf_tmap(&tmSW, sfw, (uint64_t)((N + 127) / 128), p.sf_col_tiles, atoms);
    if (e == cudaSuccess) e = encode_sf_tmap(&tmSX, sfx, (uint64_t)((M + 127) / 128), p.sf_col_tiles, atoms, p.cn > 128 ? 2 : 1);
    if (e != cudaSuccess) return (int)e;
  }
  const int tiles = ((N + 255) / 256) * ((M + p.cn - 1) / p.cn);
  if (p.ks > 1) return (int)launch_pair_kind<kPairSplit>(kind, p.cn, tmW, tmX, tmSW, tmSX, p, tiles, max_ctas, stream);
  return (int)launch_pair_kind<kPairDense>(kind, p.cn, tmW, tmX, tmSW, tmSX, p, tiles, max_ctas, stream);
}

// The routed rows of `experts` experts: X and C are in the padded row space of moe.cu (row_tiles x 128 rows), `heads` comes from
// blz_moe_plan_runs with the same `run` (128 or 256 rows at most per tile), W holds the experts' weights one after the other,
// [experts * N, K].  N % 256 == 0; act 0, or 1 (rows of each expert's W in [16 gate | 16 up] groups).
BLZ_API int blz_gemm_pair_experts(int kind, const void* X, long long ldx, const void* W, long long ldw, void* C, long long ldc, int row_tiles,
                                  int N, int K, int experts, const float* row_scale, const float* alpha, const void* sfx, const void* sfw,
                                  const void* heads, int run, int act, cudaStream_t stream) {
  using namespace blz;
  if (row_tiles <= 0) return 0;
  if (N <= 0 || N % 256 || K <= 0 || kind < 0 || kind > 2 || experts <= 0 || !heads || (run != 128 && run != 256) || act < 0 || act > 1) return (int)cudaErrorInvalidValue;
  const int kmma = kind == 0 ? 16 : kind == 1 ? 64 : 32;
  if (K % kmma || (kind && (!sfx || !sfw)) || (ldc & 1) || (reinterpret_cast<uintptr_t>(C) & 3)) return (int)cudaErrorInvalidValue;
  if ((long long)experts * N > 0x7fffffffLL) return (int)cudaErrorInvalidValue;
  PairParams p = pair_params(kind, N, K, C, ldc, row_scale, alpha, act, 0.f);
  p.heads = reinterpret_cast<const int4*>(heads);
  CUtensorMap tmW, tmX, tmSW, tmSX;
  const int es = kind == 0 ? 2 : 1;
  const uint64_t inner = kind == 1 ? (uint64_t)K / 2 : (uint64_t)K;
  cudaError_t e = encode_tmap(&tmW, W, es, inner, (uint64_t)experts * N, ldw, 128 / es, 128, 3);
  if (e == cudaSuccess) e = encode_tmap(&tmX, X, es, inner, (uint64_t)row_tiles * 128, ldx, 128 / es, 32, 3);
  tmSW = tmW; tmSX = tmX;
  const uint32_t atoms = kind == 1 ? 4 : 1;
  if (e == cudaSuccess && kind) e = encode_sf_tmap(&tmSW, sfw, (uint64_t)experts * N / 128, p.sf_col_tiles, atoms);
  if (e == cudaSuccess && kind) e = encode_sf_tmap(&tmSX, sfx, row_tiles, p.sf_col_tiles, atoms);
  if (e != cudaSuccess) return (int)e;
  return (int)launch_pair_kind<kPairExperts>(kind, run, tmW, tmX, tmSW, tmSX, p, 0, 0, stream);
}
