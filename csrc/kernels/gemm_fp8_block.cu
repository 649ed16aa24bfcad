// Exact FP8 GEMM for checkpoints with 128x128 fp32 weight block scales and 1x128 fp32 activation group scales:
//     C[m, n] = sum_kb  sa[kb, m] * sb[n / 128, kb] * ( A8[m, kb*128 : kb*128+128] . B8[n, kb*128 : kb*128+128] )  (+ bias[n])
// A8 / B8 are e4m3.  The hardware block-scaled MMA modes only take power-of-two (e8m0) scales per 32 elements, so a
// checkpoint's fp32 block scales cannot ride along with the operands.  Instead every 128-deep K block is multiplied on
// the tensor cores into its own TMEM accumulator (tcgen05.mma kind::f8f6f4, fp32 accumulate, overwrite mode), and the
// epilogue warps promote it: read the 128x128 partial from TMEM, multiply by the block's (row scale x tile scale)
// and add it to fp32 accumulators held in registers (64 per thread: one output row, 64 columns).  Two TMEM buffers
// take turns, so the tensor cores compute block kb+1 while block kb is being promoted (four buffers measured the same; so
// did polling instead of the suspended barrier wait, which was slower: the spinning warps take issue slots): per block the MMA needs about
// 256 cycles and the promotion (split over eight warps) about 100 of issue plus its TMEM load latency.
//
// 320 threads: warp 0 = TMA producer (one 128-byte-swizzled 128x128 e4m3 tile of A and of B per stage, 6 stages), warp 1
// = MMA issuer, warps 2-9 = promotion + store: two warps per TMEM lane quadrant, each owning 64 of the 128 columns, so that
// every scheduler has two promotion warps and the latency of one warp's TMEM loads hides behind the other's FMAs (with one
// warp per scheduler the tensor pipe sat at 32 % and the FMA pipe at 19 %).  Every wait is a bounded mbarrier wait that
// reports through the status word.  No TMA load is cluster-multicast.
//
// Both products here are what calls take that gemm_fp8_pair.cu does not (see blz_gemm_fp8_block): this one where the token scales are off 16
// bytes, and where no pair fits the context or pairs are off (BLAZE_GEMM_PAIR=0), the one of few rows below among them.
//
// Reference counterpart: the FP8 block-scale linear of kernels/src/cuda/fp8_linear.cu (fp8_block_* kernels: dequantise to
// bf16 and run a bf16 GEMM, or 1x128-quantised activations with per-block fp32 rescale on mma.sync), routed from
// crates/blaze/src/linear.rs (Fp8Block variants).
#include "blaze/glu.cuh"
#include "blaze/host.h"
#include "blaze/sm100.cuh"

namespace blz {

cudaError_t gemm_fp8_pair(const void* A, long long lda, const void* B, long long ldb, void* C, long long ldc, int M, int N, int K,
                          const float* sa, long long ld_sa, const float* sb, const void* bias, int out_f32, int cn, int ks, cudaStream_t stream);   // gemm_fp8_pair.cu
int pair_cluster_room(int ctas);           // gemm_pair.cu

struct FbParams {
  int M, N, K;
  void* C;                   // bf16 or fp32 [M, N]
  long long ldc;             // elements
  int out_f32;
  const float* sa;           // [K / 128, ld_sa]: activation scale of (k block, row)
  long long ld_sa;
  const float* sb;           // [ceil(N / 128), K / 128]: weight scale of (n block, k block)
  const __nv_bfloat16* bias; // [N] or null
  int* status;
};

struct FbCfg {
  static constexpr int BM = 128, BN = 128, BK = 128;
  static constexpr int A_BYTES = BM * BK, B_BYTES = BN * BK;
  static constexpr int STAGES = 6;
  static constexpr int NBUF = 2;                       // partial accumulators in flight (128 TMEM columns each)
  static constexpr int TMEM_COLS = NBUF * 128;
  static constexpr int SMEM = STAGES * (A_BYTES + B_BYTES) + 1024 /*align*/ + 256 /*barriers*/;
  static_assert(SMEM <= 227 * 1024, "shared memory budget");
};

__global__ void __launch_bounds__(320, 1)
gemm_fp8_block_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, FbParams p) {
  using Cfg = FbCfg;
  constexpr int BM = Cfg::BM, BN = Cfg::BN, STAGES = Cfg::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sA = smem;
  uint8_t* sB = sA + STAGES * Cfg::A_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sB + STAGES * Cfg::B_BYTES);
  uint64_t* full = bars;                      // [STAGES] operands of a k block have landed
  uint64_t* empty = bars + STAGES;            // [STAGES] the MMAs reading a stage have completed
  constexpr int NBUF = Cfg::NBUF;
  uint64_t* part_full = bars + 2 * STAGES;    // [NBUF] a k block's partial products are complete in TMEM buffer b
  uint64_t* part_empty = part_full + NBUF;    // [NBUF] the promotion warps have read buffer b (8 arrivals)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(part_empty + NBUF);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles_m = (p.M + BM - 1) / BM;
  const int mt = blockIdx.x % tiles_m, nt = blockIdx.x / tiles_m;     // consecutive CTAs share a weight tile through L2
  const int nkb = p.K / Cfg::BK;

  if (threadIdx.x == 0) {
    for (int i = 0; i < STAGES; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    for (int i = 0; i < NBUF; ++i) { mbar_init(&part_full[i], 1); mbar_init(&part_empty[i], 8); }
    *abort_flag = 0;
    mbar_fence_init();
    prefetch_tmap(&tmA);
    prefetch_tmap(&tmB);
  }
  if (warp == 1) tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_trigger();        // after the allocation (sm100.cuh)
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------------ producer
    if (lane == 0) {
      const int pre = min(STAGES, nkb);
      // weights do not depend on the kernel before this one: their first tiles go out before the dependency wait
      for (int i = 0; i < pre; ++i) {
        mbar_expect_tx(&full[i], Cfg::A_BYTES + Cfg::B_BYTES);
        tma_load_2d(sB + i * Cfg::B_BYTES, &tmB, i * Cfg::BK, nt * BN, &full[i]);
      }
      pdl_wait();
      int s = 0; uint32_t ph = 0;
      for (int i = 0; i < nkb; ++i) {
        if (i >= pre) {
          if (!mbar_wait(&empty[s], ph ^ 1, abort_flag, p.status)) break;
          mbar_expect_tx(&full[s], Cfg::A_BYTES + Cfg::B_BYTES);
          tma_load_2d(sB + s * Cfg::B_BYTES, &tmB, i * Cfg::BK, nt * BN, &full[s]);
        }
        tma_load_2d(sA + s * Cfg::A_BYTES, &tmA, i * Cfg::BK, mt * BM, &full[s]);
        if (++s == STAGES) { s = 0; ph ^= 1; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      int s = 0; uint32_t ph = 0;
      for (int i = 0; i < nkb; ++i) {
        const int b = i % NBUF;
        // buffer b was last filled for block i - NBUF: its promotion is completion number (i / NBUF - 1) of part_empty[b]
        if (i >= NBUF && !mbar_wait(&part_empty[b], (uint32_t)((i / NBUF - 1) & 1), abort_flag, p.status)) break;
        if (!mbar_wait(&full[s], ph, abort_flag, p.status)) break;
        tc_fence_after();
        const uint32_t a_addr = smem_u32(sA + s * Cfg::A_BYTES), b_addr = smem_u32(sB + s * Cfg::B_BYTES);
#pragma unroll
        for (int j = 0; j < 4; ++j)
          mma_f8(tmem + b * BN, desc_sw128(a_addr + j * 32), desc_sw128(b_addr + j * 32), make_idesc(0, 0, BM, BN), j > 0 ? 1u : 0u);
        mma_commit(&empty[s]);
        mma_commit(&part_full[b]);
        if (++s == STAGES) { s = 0; ph ^= 1; }
      }
    }
  } else {
    // ------------------------------------------------------------------ promotion + store (256 threads)
    const int q = warp & 3;                 // TMEM lane quadrant this warp may read
    const int half = (warp - 2) >> 2;       // which 64 columns of the tile this warp owns
    const int rl = q * 32 + lane;
    const int row = mt * BM + rl;
    const bool in_range = row < p.M;
    const float* sb = p.sb + (size_t)nt * nkb;
    constexpr int HC = BN / 2;
    float acc[HC];
#pragma unroll
    for (int i = 0; i < HC; ++i) acc[i] = 0.f;
    pdl_wait();                             // the activation scales come from the kernel before this one
    float sa_next = in_range ? p.sa[row] : 0.f;
    bool ok = true;
#pragma unroll 1
    for (int i = 0; i < nkb; ++i) {
      const int b = i % NBUF;
      const float s = sa_next * __ldg(sb + i);
      if (i + 1 < nkb) sa_next = in_range ? p.sa[(size_t)(i + 1) * p.ld_sa + row] : 0.f;
      // tcgen05.ld is warp-collective: the outcome of the wait is made warp-uniform before any lane loads
      ok = __all_sync(0xffffffffu, mbar_wait(&part_full[b], (uint32_t)((i / NBUF) & 1), abort_flag, p.status));
      if (!ok) break;
      tc_fence_after();
      const uint32_t t0 = tmem + b * BN + half * HC + ((uint32_t)(q * 32) << 16);
      uint32_t r0[32], r1[32];
      tmem_ld32(t0, r0);
      tmem_ld32(t0 + 32, r1);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        acc[j] = fmaf(__uint_as_float(r0[j]), s, acc[j]);
        acc[32 + j] = fmaf(__uint_as_float(r1[j]), s, acc[32 + j]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&part_empty[b]);
    }
    if (ok && in_range) {
#pragma unroll
      for (int c = 0; c < HC / 8; ++c) {
        const int col0 = nt * BN + half * HC + c * 8;
        if (col0 >= p.N) break;
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          v[j] = acc[c * 8 + j];
          if (p.bias && col0 + j < p.N) v[j] += bf2f(p.bias[col0 + j]);
        }
        const bool whole = col0 + 8 <= p.N;
        if (p.out_f32) {
          float* dst = reinterpret_cast<float*>(p.C) + (size_t)row * p.ldc + col0;
          if (whole && (p.ldc & 3) == 0) {
            *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
            *reinterpret_cast<float4*>(dst + 4) = make_float4(v[4], v[5], v[6], v[7]);
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              if (col0 + j < p.N) dst[j] = v[j];
          }
        } else {
          __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(p.C) + (size_t)row * p.ldc + col0;
          if (whole && (p.ldc & 7) == 0) {
            *reinterpret_cast<uint4*>(dst) = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]),
                                                        pack_bf16x2(v[6], v[7]));
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              if (col0 + j < p.N) dst[j] = __float2bfloat16(v[j]);
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, Cfg::TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------------------------------------------------
// The same product for at most 64 rows (decoding): features on the MMA's 128 lanes, the rows, rounded up to 32, on its columns, so
// that a k block costs 16 KB of weights and 8 of activations, and half the tensor and promotion time.  A small layer has few
// feature tiles (40 of the 148 SMs worked on 5120 x 8192): the K range is split over a cluster of `ks` CTAs, whose fp32 sums meet
// in distributed shared memory; CTA r owns row-column groups [r * ng / ks, (r + 1) * ng / ks) and adds the parts in rank order.
// 192 threads (producer, MMA issuer, four promotion warps: lane = feature, column = row of X), two CTAs per SM.  A k block's 64
// activation scales ride behind the operands in a ring of their own, since they outlive the operand stage.  A slot is free once all
// promotion warps have read it.  The producer knows that of the blocks before i - STAGES - NBUF only, when it fills the slot of block
// i: it has seen the MMA of block i - STAGES complete, which waited until the accumulator of block i - STAGES - NBUF was handed back,
// and a warp hands that back before it reads the block's scales, but after those of the block before.  Weight bytes bound it.
struct FrCfg {
  static constexpr int W_BYTES = 128 * 128, X_BYTES = 64 * 128, STAGES = 4;
  static constexpr int NBUF = 4, TMEM_COLS = NBUF * 64;
  static constexpr int SA_SLOTS = 16, SA_BYTES = 64 * 4;
  static constexpr int RING = STAGES * (W_BYTES + X_BYTES);
  static constexpr int SMEM = RING + SA_SLOTS * SA_BYTES + 1024 /*align*/ + 384 /*barriers*/;
  static constexpr int GROUP = 8;                      // row columns that change hands together in the reduction
  static_assert(2 * (SMEM + 1024) <= 228 * 1024, "two CTAs per SM");
  static_assert((2 * STAGES + 2 * NBUF + SA_SLOTS + 2) * 8 + 8 <= 384, "barriers");
  static_assert(STAGES + NBUF < SA_SLOTS, "a scale slot is read before it is filled again");
};

__global__ void __launch_bounds__(192, 2)
gemm_fp8_rows_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, FbParams p, int ks) {
  using Cfg = FrCfg;
  constexpr int STAGES = Cfg::STAGES, NBUF = Cfg::NBUF, GW = Cfg::GROUP;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sW = smem;
  uint8_t* sX = sW + STAGES * Cfg::W_BYTES;
  float* sSA = reinterpret_cast<float*>(smem + Cfg::RING);            // [SA_SLOTS][64]
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + Cfg::RING + Cfg::SA_SLOTS * Cfg::SA_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* part_full = empty + STAGES;    // [NBUF] a k block's products are complete in TMEM buffer b
  uint64_t* part_empty = part_full + NBUF; // [NBUF] the promotion warps have read it (4 arrivals)
  uint64_t* sa_full = part_empty + NBUF;   // [SA_SLOTS]
  uint64_t* ring_free = sa_full + Cfg::SA_SLOTS;       // every CTA of the cluster has finished its main loop (ks remote arrivals)
  uint64_t* part_ready = ring_free + 1;    // every CTA of the cluster has parked its sums here
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(part_ready + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kr = ks > 1 ? (int)cluster_ctarank() : 0;
  const int nt = blockIdx.x / ks;
  const int nkb_all = p.K / 128;
  const int kb0 = (int)((long long)kr * nkb_all / ks), nkb = (int)((long long)(kr + 1) * nkb_all / ks) - kb0;      // >= 1: ks <= nkb_all
  const int ncols = (p.M + 31) & ~31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < STAGES; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    for (int i = 0; i < NBUF; ++i) { mbar_init(&part_full[i], 1); mbar_init(&part_empty[i], 4); }
    for (int i = 0; i < Cfg::SA_SLOTS; ++i) mbar_init(&sa_full[i], 1);
    mbar_init(ring_free, ks);
    mbar_init(part_ready, ks);
    *abort_flag = 0;
    mbar_fence_init();
    prefetch_tmap(&tmW);
    prefetch_tmap(&tmX);
  }
  if (warp == 1) tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_trigger();
  if (ks > 1) cluster_arrive();            // the peers' barriers are initialised before anyone arrives on them remotely
  const uint32_t tmem = *tmem_slot;
  int issued = 0;                          // thread 0: blocks whose copies have been started

  if (warp == 0) {
    if (lane == 0) {
      const int pre = min(STAGES, nkb);
      const uint32_t sa_bytes = (uint32_t)((p.M + 3) & ~3) * 4u;
      auto weights = [&](int s, int i) {
        mbar_expect_tx(&full[s], Cfg::W_BYTES + (uint32_t)ncols * 128u);
        tma_load_2d(sW + s * Cfg::W_BYTES, &tmW, (kb0 + i) * 128, nt * 128, &full[s]);
      };
      for (int i = 0; i < pre; ++i) weights(i, i);     // they do not depend on the kernel before this one
      pdl_wait();
      int s = 0; uint32_t ph = 0;
      for (int i = 0; i < nkb; ++i) {
        if (i >= pre) {
          if (!mbar_wait(&empty[s], ph ^ 1, abort_flag, p.status)) break;
          weights(s, i);
        }
        for (int c = 0; c < ncols; c += 32) tma_load_2d(sX + s * Cfg::X_BYTES + c * 128, &tmX, (kb0 + i) * 128, c, &full[s]);
        const int slot = i % Cfg::SA_SLOTS;
        mbar_expect_tx(&sa_full[slot], sa_bytes);
        bulk_load(sSA + slot * 64, p.sa + (size_t)(kb0 + i) * p.ld_sa, sa_bytes, &sa_full[slot]);
        if (++s == STAGES) { s = 0; ph ^= 1; }
        issued = i + 1;
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      int s = 0; uint32_t ph = 0;
      for (int i = 0; i < nkb; ++i) {
        const int b = i % NBUF;
        if (i >= NBUF && !mbar_wait(&part_empty[b], (uint32_t)((i / NBUF - 1) & 1), abort_flag, p.status)) break;
        if (!mbar_wait(&full[s], ph, abort_flag, p.status)) break;
        tc_fence_after();
        const uint32_t w_addr = smem_u32(sW + s * Cfg::W_BYTES), x_addr = smem_u32(sX + s * Cfg::X_BYTES);
#pragma unroll
        for (int j = 0; j < 4; ++j)
          mma_f8(tmem + b * 64, desc_sw128(w_addr + j * 32), desc_sw128(x_addr + j * 32), make_idesc(0, 0, 128, ncols), j > 0 ? 1u : 0u);
        mma_commit(&empty[s]);
        mma_commit(&part_full[b]);
        if (++s == STAGES) { s = 0; ph ^= 1; }
      }
    }
  }
  __syncwarp();
  if (ks > 1) cluster_wait();              // all threads, unconditionally (pairs with cluster_arrive above)
  if (warp >= 2) {
    const int q = warp & 3, fl = q * 32 + lane, f = nt * 128 + fl;
    float acc[64];
#pragma unroll
    for (int j = 0; j < 64; ++j) acc[j] = 0.f;
    const float* sb = p.sb + (size_t)nt * nkb_all + kb0;
    bool ok = true;
    float sb_next = __ldg(sb);
#pragma unroll 1
    for (int i = 0; i < nkb; ++i) {
      const int b = i % NBUF, slot = i % Cfg::SA_SLOTS;
      const float sbv = sb_next;
      if (i + 1 < nkb) sb_next = __ldg(sb + i + 1);
      // tcgen05.ld is warp-collective: the outcome of the waits is made warp-uniform before any lane loads
      ok = __all_sync(0xffffffffu, mbar_wait(&sa_full[slot], (uint32_t)((i / Cfg::SA_SLOTS) & 1), abort_flag, p.status) &&
                                       mbar_wait(&part_full[b], (uint32_t)((i / NBUF) & 1), abort_flag, p.status));
      if (!ok) break;
      tc_fence_after();
      const float4* sa = reinterpret_cast<const float4*>(sSA + slot * 64);
      const uint32_t t0 = tmem + b * 64 + ((uint32_t)(q * 32) << 16);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (h * 32 >= ncols) break;
        uint32_t r[32];
        tmem_ld32(t0 + h * 32, r);
        tmem_ld_wait();
        if ((h + 1) * 32 >= ncols) {       // the products are in registers: hand the buffer back
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&part_empty[b]);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float4 s4 = sa[h * 8 + j];
          float* a = acc + h * 32 + j * 4;
          a[0] = fmaf(__uint_as_float(r[4 * j]), s4.x * sbv, a[0]);
          a[1] = fmaf(__uint_as_float(r[4 * j + 1]), s4.y * sbv, a[1]);
          a[2] = fmaf(__uint_as_float(r[4 * j + 2]), s4.z * sbv, a[2]);
          a[3] = fmaf(__uint_as_float(r[4 * j + 3]), s4.w * sbv, a[3]);
        }
      }
    }
    const float bias = p.bias && f < p.N ? bf2f(p.bias[f]) : 0.f;
    auto store = [&](int row, float v) {
      if (row >= p.M || f >= p.N) return;
      if (p.out_f32) reinterpret_cast<float*>(p.C)[(size_t)row * p.ldc + f] = v + bias;
      else reinterpret_cast<__nv_bfloat16*>(p.C)[(size_t)row * p.ldc + f] = __float2bfloat16(v + bias);
    };
    if (ks == 1) {
      if (ok) {
#pragma unroll
        for (int j = 0; j < 64; ++j) store(j, acc[j]);
      }
    } else {
      const int ng = ncols / GW, GL = (ng + ks - 1) / ks;
      const uint32_t recv = smem_u32(smem);            // slot [source CTA][group][column quad][feature], over the operand ring
      if (threadIdx.x == 64) {
        for (int r = 0; r < ks; ++r) mbar_arrive_remote(mapa_shared(smem_u32(ring_free), r));
      }
      // an aborted CTA still arrives and still waits, so that its peers are not left waiting for it
      const bool free_all = __all_sync(0xffffffffu, mbar_wait_cluster(ring_free, 0, abort_flag, p.status));
      if (ok && free_all) {
#pragma unroll
        for (int cq = 0; cq < 16; ++cq) {
          if (cq * 4 >= ncols) break;
          const int g = cq / 2, owner = (g * ks + ks - 1) / ng, gl = g - owner * ng / ks;       // owner * ng / ks <= g
          st_dsmem_f4(mapa_shared(recv + (uint32_t)(((kr * GL + gl) * 2 + (cq & 1)) * 128 + fl) * 16u, owner), acc[4 * cq], acc[4 * cq + 1],
                      acc[4 * cq + 2], acc[4 * cq + 3]);
        }
      }
      fence_acq_rel_cluster();
      bar_sync(1, 128);
      if (threadIdx.x == 64) {
        for (int r = 0; r < ks; ++r) mbar_arrive_remote(mapa_shared(smem_u32(part_ready), r));
      }
      const bool all = __all_sync(0xffffffffu, mbar_wait_cluster(part_ready, 0, abort_flag, p.status));
      if (all && ok && free_all && !*abort_flag) {
        const float4* got = reinterpret_cast<const float4*>(smem);
        const int g0 = kr * ng / ks, g1 = (kr + 1) * ng / ks;
        for (int cq = g0 * 2; cq < g1 * 2; ++cq) {
          float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
          for (int r = 0; r < ks; ++r) {               // rank order: the sum does not depend on timing
            const float4 x = got[((r * GL + (cq / 2 - g0)) * 2 + (cq & 1)) * 128 + fl];
            v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
          }
          store(cq * 4, v.x); store(cq * 4 + 1, v.y); store(cq * 4 + 2, v.z); store(cq * 4 + 3, v.w);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag) {
    // a wait ran out: the copies that are still on their way write to this CTA's memory (these waits are limited, too)
    *abort_flag = 0;
    for (int i = max(issued - STAGES, 0); i < issued; ++i) mbar_wait(&full[i % STAGES], (uint32_t)((i / STAGES) & 1), abort_flag, p.status);
    for (int i = max(issued - Cfg::SA_SLOTS, 0); i < issued; ++i)
      mbar_wait(&sa_full[i % Cfg::SA_SLOTS], (uint32_t)((i / Cfg::SA_SLOTS) & 1), abort_flag, p.status);
  }
  if (ks > 1) {
    // ... and a peer whose waits ran out later still writes and arrives here: nobody leaves before all are done
    __syncwarp();
    cluster_arrive();
    cluster_wait();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, Cfg::TMEM_COLS);
  }
}

// CTAs that share a feature tile (1, 2, 4 or 8; odd clusters pack badly), 0: the kernel above is the faster one.
// The kernel above walks all k blocks in one CTA per 128 features (5 us + 0.3 us a block while they fit on the chip at once), this one
// a part of them, for an exchange of 4 us that grows with the number of CTAs.  Clusters of four find room up to 8/5 CTAs per SM (beyond,
// some wait for a second turn), and more than 32 rows double the exchange.  Time over the kernel above's at N x K, 16 - 32 rows:
//   four CTAs    N <= 4096: K 1024 1.04 - 1.10, 2048 0.86 - 0.95, 4096 0.67 - 0.77, 7168 0.55 - 0.64; N 5120, 7168: K 3072 1.01 - 1.05,
//                4096 0.89 - 0.97, 5120 0.79 - 0.89, 25600 0.47; N 9216: K 5120 1.04 - 1.34
//   two          N 5120 - 9216: K 2048 0.94 - 1.04, 3072 0.84 - 0.98, 4096 0.77 - 0.95, 5120 0.72 - 0.90; N 12288 - 18432: K 4096
//                0.88 - 0.94 (16 rows), 0.85 - 0.97 (24), 0.91 - 1.11 (28 - 32), 5120 1.00 - 1.06 (28 - 32), 7168 0.78 - 0.96
//   one          N 24576, 36864 (more tiles than SMs): K 1024 - 7168 0.61 - 0.83
// and at 36 - 64 rows:
//   eight        N <= 1024: K 2048 1.06 - 1.09, 3072 0.90 - 0.93, 7168 0.60 - 0.62; N 2048: K 4096 1.01
//   four         N 2048 - 4096: K 2048 1.04 - 1.11, 3072 0.92 - 0.99, 7168 0.69 - 0.75; N 5120, 7168: K 5120 1.03 - 1.07, 7168
//                0.94 - 0.98, 8192 0.91, 25600 0.59; N 9216: K 7168 1.42
// The fp32 sums of a row's parts differ from the sum block by block in their roundings: error against 64 bits 6e-8 - 1.4e-7 where that
// has 8e-8 - 2.6e-7 (K 2048 - 25600).
static int fp8_rows_ks(const FbParams& p) {
  const int tiles = (p.N + 127) / 128, nkb = p.K / 128, sms = sm_count();
  const bool four = tiles * 4 <= sms, four_fit = tiles * 4 <= sms * 8 / 5;
  if (p.M > 32) {
    if (nkb >= 24 && four) return tiles * 16 <= sms ? 8 : 4;
    return nkb >= 56 && four_fit ? 4 : 0;
  }
  if (tiles > sms) return 1;
  if (four) return nkb >= 16 ? 4 : 0;
  if (tiles * 2 <= sms) return nkb >= 40 && four_fit ? 4 : nkb >= 24 ? 2 : 0;
  return nkb >= (p.M <= 24 ? 32 : 56) ? 2 : 0;
}

static cudaError_t launch_fp8_rows(const FbParams& p, int ks, const void* A, long long lda, const void* B, long long ldb, cudaStream_t stream) {
  const int tiles = (p.N + 127) / 128;
  CUtensorMap tmW, tmX;
  cudaError_t e = encode_tmap(&tmW, B, 1, (uint64_t)p.K, p.N, ldb, 128, 128, 3);
  if (e != cudaSuccess) return e;
  e = encode_tmap(&tmX, A, 1, (uint64_t)p.K, p.M, lda, 128, 32, 3);
  if (e != cudaSuccess) return e;
  static PerDeviceOnce configured;
  e = configured.smem_limit(gemm_fp8_rows_kernel, FrCfg::SMEM);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tiles * ks));
  cfg.blockDim = dim3(192);
  cfg.dynamicSmemBytes = FrCfg::SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (ks > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = ks;
    attr[n].val.clusterDim.y = 1;
    attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (pdl_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, gemm_fp8_rows_kernel, tmW, tmX, p, ks);
}

// ---------------------------------------------------------------------------------------------------------------------
// Activation quantiser: bf16 [T, K] -> e4m3 [T, K] with one fp32 scale per (row, 128-column group), scale = amax / 448,
// written k-block-major ([K / 128, ld_s]) so that the GEMM's promotion warps read them coalesced.  GATED: the rows are [gate | up]
// and silu(gate) * up, rounded to bf16, is what is quantised.
// Bound by memory where rows are many, by the launch where they are few.  Eight threads per group, 16 elements each; the warps of a CTA
// take the same four groups of eight neighbouring rows, so that the scales' 4-byte stores, ld_s apart within a warp, fill 32-byte sectors.
// us, one warp per group with 4 elements a thread / now: 4096 rows of 25600 155 / 85, 825 rows 38 / 24, 64 rows 9.2 / 9.2; with the
// gated activation (a kernel of its own before): 4096 rows 269 / 150, 825 rows 65 / 38, 64 rows 17.4 / 11.2, of 5120 13.3 / 9.2.
// Plain rows of fewer than 3 x 2^18 elements are the warp's per group: so little work is bound by the longer chain of 16 divisions per
// thread (back to back, 4 / 16 elements a thread: 1 row of 5120 1.93 / 2.26, 16 rows 2.04 / 2.46, 64 x 2048 2.09 / 2.58, 64 x 7168
// 2.39 / 2.68, 128 x 5120 2.60 / 2.85; 150 x 5120 2.80 / 2.79, 64 x 12288 2.93 / 2.80).
__global__ void __launch_bounds__(256)
quant_fp8_few_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, uint8_t* __restrict__ q, float* __restrict__ scales,
                     long long ld_s, int T, int K) {
  pdl_wait();
  pdl_trigger();
  const int groups = K / 128, lane = threadIdx.x & 31;
  const int g = (int)blockIdx.x * 8 + (int)(threadIdx.x >> 5);
  if (g >= T * groups) return;
  const int row = g / groups, kb = g % groups;
  const uint2 raw = *reinterpret_cast<const uint2*>(x + (size_t)row * ldx + kb * 128 + lane * 4);
  const float v[4] = {__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u), __uint_as_float(raw.y << 16), __uint_as_float(raw.y & 0xffff0000u)};
  const float m = warp_max(fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3]))));
  const float scale = fmaxf(m / 448.f, 1e-12f);
  const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(v[0] / scale, v[1] / scale), __NV_SATFINITE, __NV_E4M3);
  const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(v[2] / scale, v[3] / scale), __NV_SATFINITE, __NV_E4M3);
  *reinterpret_cast<uint32_t*>(q + (size_t)row * K + kb * 128 + lane * 4) = lo | hi << 16;
  if (lane == 0) scales[(size_t)kb * ld_s + row] = scale;
}

template <bool GATED>
__global__ void __launch_bounds__(256)
quant_fp8_block_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, uint8_t* __restrict__ q, float* __restrict__ scales,
                       long long ld_s, int T, int K, int on16) {
  pdl_wait();
  pdl_trigger();
  const int across = (K + 511) / 512, lane = threadIdx.x & 31;
  const int row = (int)(blockIdx.x / across) * 8 + (threadIdx.x >> 5), col = (int)(blockIdx.x % across) * 512 + lane * 16;
  const bool live = row < T && col < K;
  uint32_t w[8] = {}, u[GATED ? 8 : 1];
  auto load = [&](uint32_t* d, const __nv_bfloat16* src) {
    if (on16) {
#pragma unroll
      for (int j = 0; j < 2; ++j) *reinterpret_cast<uint4*>(d + 4 * j) = reinterpret_cast<const uint4*>(src)[j];
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) *reinterpret_cast<uint2*>(d + 2 * j) = reinterpret_cast<const uint2*>(src)[j];
    }
  };
  if (live) load(w, x + (size_t)row * ldx + col);
  if constexpr (GATED) {
    if (live) load(u, x + (size_t)row * ldx + K + col);
  }
  float v[16], m = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    v[2 * j] = __uint_as_float(w[j] << 16);
    v[2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u);
    if constexpr (GATED) {
      if (live) {
        v[2 * j] = __bfloat162float(__float2bfloat16(silu(v[2 * j]) * __uint_as_float(u[j] << 16)));
        v[2 * j + 1] = __bfloat162float(__float2bfloat16(silu(v[2 * j + 1]) * __uint_as_float(u[j] & 0xffff0000u)));
      }
    }
    m = fmaxf(fmaxf(m, fabsf(v[2 * j])), fabsf(v[2 * j + 1]));
  }
#pragma unroll
  for (int d = 1; d < 8; d *= 2) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
  const float scale = fmaxf(m / 448.f, 1e-12f);
  if (!live) return;
  uint32_t out[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(v[4 * j] / scale, v[4 * j + 1] / scale), __NV_SATFINITE, __NV_E4M3);
    const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(v[4 * j + 2] / scale, v[4 * j + 3] / scale), __NV_SATFINITE, __NV_E4M3);
    out[j] = lo | hi << 16;
  }
  *reinterpret_cast<uint4*>(q + (size_t)row * K + col) = make_uint4(out[0], out[1], out[2], out[3]);
  if (lane % 8 == 0) scales[(size_t)(col / 128) * ld_s + row] = scale;
}

template <bool GATED>
static cudaError_t launch_quant_fp8(const void* x, long long ldx, void* q, float* scales, long long ld_s, int T, int K, cudaStream_t stream) {
  const __nv_bfloat16* rows = reinterpret_cast<const __nv_bfloat16*>(x);
  uint8_t* codes = reinterpret_cast<uint8_t*>(q);
  if (!GATED && (long long)T * K < 3 << 18)
    return launch_pdl(quant_fp8_few_kernel, dim3((unsigned)((T * (K / 128) + 7) / 8)), dim3(256), 0, stream, rows, ldx, codes, scales, ld_s, T, K);
  const int on16 = ldx % 8 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  return launch_pdl(quant_fp8_block_kernel<GATED>, dim3((unsigned)((long long)((T + 7) / 8) * ((K + 511) / 512))), dim3(256), 0, stream, rows, ldx,
                    codes, scales, ld_s, T, K, on16);
}

}  // namespace blz

// A e4m3 [M, K] (lda bytes), B e4m3 [N, K] (ldb bytes), sa fp32 [K / 128, ld_sa], sb fp32 [ceil(N / 128), K / 128]; C bf16 or
// fp32 [M, N] with ldc in elements.  K must be a multiple of 128.
BLZ_API int blz_gemm_fp8_block(const void* A, long long lda, const void* B, long long ldb, void* C, long long ldc, int M, int N,
                               int K, const float* sa, long long ld_sa, const float* sb, const void* bias, int out_f32,
                               cudaStream_t stream) {
  using namespace blz;
  if (M <= 0 || N <= 0 || K <= 0 || K % 128 || !sa || !sb || ld_sa < M) return (int)cudaErrorInvalidValue;
  // The pairs' kernel is the faster one at any size; it fetches the token scales by a tensor map, which start and step on 16 bytes
  // (blz_quant_fp8_block's do), and needs a context with room for two neighbouring CTAs.
  const bool on16 = ld_sa % 4 == 0 && (reinterpret_cast<uintptr_t>(sa) & 15) == 0;
  if (on16 && pair_cluster_room(2) > 0)
    return (int)gemm_fp8_pair(A, lda, B, ldb, C, ldc, M, N, K, sa, ld_sa, sb, bias, out_f32, 0, 0, stream);
  FbParams p;
  p.M = M; p.N = N; p.K = K; p.C = C; p.ldc = ldc; p.out_f32 = out_f32;
  p.sa = sa; p.ld_sa = ld_sa; p.sb = sb; p.bias = reinterpret_cast<const __nv_bfloat16*>(bias);
  p.status = status_word();
  if (M <= 64 && on16) {                     // the scales' rows are copied by 16 bytes
    const int ks = fp8_rows_ks(p);
    if (ks > 0) return (int)launch_fp8_rows(p, ks, A, lda, B, ldb, stream);
  }
  CUtensorMap tmA, tmB;
  cudaError_t e = encode_tmap(&tmA, A, 1, (uint64_t)K, M, lda, 128, 128, 3);
  if (e != cudaSuccess) return (int)e;
  e = encode_tmap(&tmB, B, 1, (uint64_t)K, N, ldb, 128, 128, 3);
  if (e != cudaSuccess) return (int)e;
  auto kern = gemm_fp8_block_kernel;
  static PerDeviceOnce configured;
  e = configured.smem_limit(kern, FbCfg::SMEM);
  if (e != cudaSuccess) return (int)e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(((M + 127) / 128) * ((N + 127) / 128));
  cfg.blockDim = dim3(320);
  cfg.dynamicSmemBytes = FbCfg::SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  int n = 0;
  if (pdl_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return (int)cudaLaunchKernelEx(&cfg, kern, tmA, tmB, p);
}

// x bf16 [T, K] (ldx elements) -> q e4m3 [T, K] contiguous, scales fp32 [K / 128, ld_s].  K % 128 == 0, ldx % 4 == 0.
BLZ_API int blz_quant_fp8_block(const void* x, long long ldx, void* q, float* scales, long long ld_s, int T, int K,
                                cudaStream_t stream) {
  using namespace blz;
  if (T <= 0) return 0;
  if (K <= 0 || K % 128 || (ldx & 3) || ld_s < T) return (int)cudaErrorInvalidValue;
  return (int)launch_quant_fp8<false>(x, ldx, q, scales, ld_s, T, K, stream);
}

// The same of silu(gate) * up, rounded to bf16: gu bf16 [T, 2K] = [gate | up].
BLZ_API int blz_swiglu_fp8_block(const void* gu, void* q, float* scales, long long ld_s, int T, int K, cudaStream_t stream) {
  using namespace blz;
  if (T <= 0) return 0;
  if (K <= 0 || K % 128 || ld_s < T) return (int)cudaErrorInvalidValue;
  return (int)launch_quant_fp8<true>(gu, 2LL * K, q, scales, ld_s, T, K, stream);
}
