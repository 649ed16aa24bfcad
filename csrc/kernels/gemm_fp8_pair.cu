// FP8 GEMM with 128x128 fp32 weight block scales and 1x128 fp32 activation scales on CTA pairs (the product of gemm_fp8_block.cu):
//     C[m, n] = sum_kb  sa[kb, m] * sb[n / 128, kb] * ( A8[m, kb*128 : kb*128+128] . B8[n, kb*128 : kb*128+128] )  (+ bias[n])
// A pair (tcgen05 cta_group::2) computes 256 features (MMA lanes, 128 in each CTA) x 64 or 128 tokens (columns).  Every block of 128 along
// K is multiplied into tensor-memory columns of its own, and the epilogue warps promote it: a thread owns one feature and 32 tokens, multiplies
// the partial by (token scale x block scale) and adds it to fp32 registers, two values at a time.  Two blocks share a stage, a buffer (two
// in turn) and their barriers: waits and commits per block cost as much as its products.
//
// Persistent, one pair per two SMs.  The token scales come by a tensor map into a ring of 8 slots in each CTA, with barriers of their own,
// since they outlive the operands' stage: `sa_full`, and `sa_empty`, on which every epilogue warp of the CTA arrives when it has read a slot.
// (A buffer that is handed back says so too, but only of tensor memory, and to the MMA warp of the first CTA.)  A slot is filled STAGES
// steps ahead of its products, which wait for the reading of a step NBUF before theirs, so with 8 slots that wait holds nothing up.
//
// Against one CTA per 128 x 128 tile, and one or a cluster of CTAs per 128 features up to 64 rows (us, inputs from memory): 64 rows x 10240 x
// 5120 24.8 -> 17.2, x 5120 x 8192 23.9 -> 16.6, x 51200 x 5120 76 -> 58, x 5120 x 25600 47 -> 37; 128 rows of those 27 -> 19.5, 32 ->
// 19.6, 78 -> 61, 88 -> 43; 1000 rows 89 -> 71, 80 -> 65, 357 -> 298, 252 -> 190; 4096 rows 292 -> 244, 223 -> 188, 1345 -> 1330,
// 775 -> 629.  (With one block per stage 1000 rows x 51200 x 5120 took 380.  The forms of 128 tokens, 18 warps, have 96 registers a thread
// and spill 20 and, split, 44 bytes; loads of the next partials ahead of the sums spill more.)  A slot that is released with the next
// step's buffer instead of a barrier of its own holds the producer up: 64 rows x 10240 x 5120 15.3 -> 16.3, 16 x 5120 x 25600 30.7 -> 35.6.
//
// Few tiles: K is split over the pairs of a cluster, which exchange their sums through distributed shared memory as in gemm_pair.cu.
// Every wait is bounded; no load is multicast.
//
// Reference counterpart: as gemm_fp8_block.cu.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <type_traits>

#include "blaze/host.h"
#include "blaze/sm100.cuh"

namespace blz {

struct FpParams {
  int M, N, K;
  void* C;                    // bf16 or fp32 [M, ldc]
  long long ldc;
  int out_f32;
  int paired;                 // features may be stored two at a time
  const float* sb;            // [ceil(N / 128), K / 128]
  const __nv_bfloat16* bias;  // [N] or null
  int ks;                     // pairs that share a tile's K
  int* status;
};

template <int CN>
struct FpCfg {
  static constexpr int A_BYTES = 128 * 128, B_BYTES = CN * 64;     // of one block of K; a stage holds two
  static constexpr int STAGE_BYTES = 2 * (A_BYTES + B_BYTES);
  static constexpr int STAGES = (200 * 1024) / STAGE_BYTES;
  static constexpr int NBUF = 2, SLOTS = 8;                 // buffers and scales of two blocks each
  static constexpr int EPI = CN / 8;                        // epilogue warps: one per lane quadrant and 32 columns
  static constexpr int THREADS = 64 + EPI * 32;
  static constexpr int SMEM = STAGES * STAGE_BYTES + SLOTS * CN * 8 + 1024 + 512;
  static_assert((2 * STAGES + 2 * NBUF + 2 * SLOTS + 3) * 8 + 8 <= 512 && SMEM <= 227 * 1024, "shared memory");
};

template <int CN, bool SPLIT>
__global__ void __launch_bounds__(FpCfg<CN>::THREADS, 1) gemm_fp8_pair_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX,
                                                                              const __grid_constant__ CUtensorMap tmS, const FpParams p) {
  using Cfg = FpCfg<CN>;
  constexpr int STAGES = Cfg::STAGES, NBUF = Cfg::NBUF, SLOTS = Cfg::SLOTS;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);      // the same offset in every CTA of the cluster
  uint8_t* sA = base;
  uint8_t* sB = sA + STAGES * 2 * Cfg::A_BYTES;
  float* sSA = reinterpret_cast<float*>(sB + STAGES * 2 * Cfg::B_BYTES);                // [SLOTS][2][CN]
  uint64_t* full = reinterpret_cast<uint64_t*>(sSA + SLOTS * 2 * CN);
  uint64_t* empty = full + STAGES;
  uint64_t* part_full = empty + STAGES;     // [NBUF] a block's products are complete
  uint64_t* part_empty = part_full + NBUF;  // [NBUF] both CTAs' epilogue warps have read them
  uint64_t* sa_full = part_empty + NBUF;    // [SLOTS]
  uint64_t* sa_empty = sa_full + SLOTS;     // [SLOTS] this CTA's epilogue warps have read a slot
  uint64_t* drain = sa_empty + SLOTS;
  uint64_t* ring_free = drain + 1;          // every CTA of the split is done with its operands (its ring may be written)
  uint64_t* part_ready = ring_free + 1;     // and has handed out its sums
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(part_ready + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t crank = cluster_ctarank(), rank = crank & 1, lead = crank & ~1u;
  const int ks = SPLIT ? p.ks : 1, kp = SPLIT ? (int)(crank >> 1) : 0;
  const int pair = blockIdx.x / (2 * ks), pairs = gridDim.x / (2 * ks);
  const int tiles_f = (p.N + 255) / 256, tiles_t = (p.M + CN - 1) / CN, tiles = tiles_f * tiles_t;
  const int nkb = p.K / 128, steps = (nkb + 1) / 2, kb0 = kp * steps / ks, kb1 = (kp + 1) * steps / ks;      // in steps of two blocks

  if (threadIdx.x == 0) {
    for (int i = 0; i < STAGES; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    for (int i = 0; i < NBUF; ++i) { mbar_init(&part_full[i], 1); mbar_init(&part_empty[i], 2 * Cfg::EPI); }
    for (int i = 0; i < SLOTS; ++i) { mbar_init(&sa_full[i], 1); mbar_init(&sa_empty[i], Cfg::EPI); }
    mbar_init(drain, 1);
    mbar_init(ring_free, ks);
    mbar_init(part_ready, ks);
    *abort_flag = 0;
    mbar_fence_init();
    prefetch_tmap(&tmW);
    prefetch_tmap(&tmX);
    prefetch_tmap(&tmS);
  }
  __syncwarp();
  if (warp == 1) tmem_alloc_pair(tmem_slot, NBUF * 2 * CN);
  tc_fence_before();
  __syncthreads();
  cluster_arrive();                         // the peers' barriers are initialised before anything signals them
  cluster_wait();
  tc_fence_after();
  pdl_trigger();        // after the allocation (sm100.cuh)
  const uint32_t tmem = *tmem_slot;
  pdl_wait();

  // tile u -> (feature tile, token tile), in bands of eight token tiles (see gemm_pair.cu)
  auto tile_at = [&](int u, int& ft, int& t0) {
    const int per_band = 8 * tiles_f, band = u / per_band, in = u - band * per_band, width = min(8, tiles_t - band * 8);
    ft = in / width;
    t0 = (band * 8 + in - ft * width) * CN;
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ producer: this CTA's half of the operands, the tile's scales
    if (lane == 0) {
      int s = 0; uint32_t ph = 0;
      int gb = 0;                           // blocks so far
      uint32_t used = 0, last = 0;          // stages filled so far, and the parity of their latest fill
      bool ok = true;
      for (int u = pair; u < tiles && ok; u += pairs) {
        int ft, t0;
        tile_at(u, ft, t0);
        for (int kb = kb0; kb < kb1; ++kb, ++gb) {
          if (!mbar_wait(&empty[s], ph ^ 1, abort_flag, p.status)) { ok = false; break; }
          if (gb >= SLOTS && !mbar_wait(&sa_empty[gb % SLOTS], (gb / SLOTS - 1) & 1, abort_flag, p.status)) { ok = false; break; }
          const uint32_t bar = mapa_shared(smem_u32(&full[s]), lead);
          if (rank == 0) mbar_expect_tx(&full[s], 2u * Cfg::STAGE_BYTES);
          // (an odd number of blocks: the last one's neighbour lies beyond K and is filled with zeros)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            tma_load_2d_pair(sA + (s * 2 + h) * Cfg::A_BYTES, &tmW, (kb * 2 + h) * 128, ft * 256 + (int)rank * 128, bar);
            tma_load_2d_pair(sB + (s * 2 + h) * Cfg::B_BYTES, &tmX, (kb * 2 + h) * 128, t0 + (int)rank * (CN / 2), bar);
          }
          uint64_t* sbar = &sa_full[gb % SLOTS];
          mbar_expect_tx(sbar, CN * 8);
          tma_load_2d_pair(sSA + (gb % SLOTS) * 2 * CN, &tmS, t0, kb * 2, mapa_shared(smem_u32(sbar), crank));
          used |= 1u << s;
          last = (last & ~(1u << s)) | (ph << s);
          if (++s == STAGES) { s = 0; ph ^= 1; }
        }
      }
      if (!ok) {                            // no copy is in flight when the pair leaves
        for (int i = max(gb - SLOTS, 0); i < gb; ++i) mbar_drain(&sa_full[i % SLOTS], (i / SLOTS) & 1);
        if (rank == 0)
          for (int i = 0; i < STAGES; ++i)
            if (used >> i & 1) mbar_drain(&full[i], last >> i & 1);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer of the pair
    if (rank == 0) {
      int s = 0; uint32_t ph = 0;
      int gb = 0;
      bool ok = true;
      const bool leader = elect_one();
      const uint32_t a_lo0 = (uint32_t)desc_sw128(smem_u32(sA)), b_lo0 = (uint32_t)desc_sw128(smem_u32(sB));
      constexpr uint32_t OP_HI = (1024u >> 4) | 1u << 14 | (uint32_t)kSwz128 << 29;
      auto desc = [](uint32_t lo) { return (uint64_t)OP_HI << 32 | lo; };
      for (int u = pair; u < tiles && ok; u += pairs) {
        for (int kb = kb0; kb < kb1; ++kb, ++gb) {
          const int b = gb % NBUF;
          if (gb >= NBUF && !mbar_wait_cluster(&part_empty[b], (gb / NBUF - 1) & 1, abort_flag, p.status)) { ok = false; break; }
          if (!mbar_wait(&full[s], ph, abort_flag, p.status)) { ok = false; break; }
          tc_fence_after();
          const uint32_t a_lo = a_lo0 + s * (2 * Cfg::A_BYTES >> 4), b_lo = b_lo0 + s * (2 * Cfg::B_BYTES >> 4);
          if (leader) {
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
              for (int j = 0; j < 4; ++j)
                mma_f8_pair(tmem + (b * 2 + h) * CN, desc(a_lo + h * (Cfg::A_BYTES >> 4) + j * 2), desc(b_lo + h * (Cfg::B_BYTES >> 4) + j * 2),
                            make_idesc(0, 0, 256, CN), j > 0 ? 1u : 0u);
            mma_commit_pair(&empty[s], lead);
            mma_commit_pair(&part_full[b], lead);
          }
          __syncwarp();
          if (++s == STAGES) { s = 0; ph ^= 1; }
        }
      }
      if (!ok && leader) {                  // the MMAs in flight end before their operands' memory goes
        mma_commit_pair(drain, lead);
        mbar_drain(drain, 0);
      }
    }
  } else {
    // ------------------------------------------------------------------ promotion: lane = feature, half of the columns per warp
    const int q = warp & 3, part = (warp - 2) >> 2, c0 = part * 32, etid = threadIdx.x - 64;
    const bool odd = lane & 1;
    const uint32_t pick = odd ? 0x3276u : 0x5410u;
    const uint32_t quad = (uint32_t)(q * 32) << 16;
    int gb = 0;
    bool ok = true;
    for (int u = pair; u < tiles && ok; u += pairs) {
      int ft, t0;
      tile_at(u, ft, t0);
      const int feat = ft * 256 + (int)rank * 128 + q * 32 + lane;
      const bool feat_ok = feat < p.N;
      const float* sb = p.sb + (size_t)min(ft * 2 + (int)rank, (p.N + 127) / 128 - 1) * nkb;
      float acc[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) acc[j] = 0.f;
#pragma unroll 1
      for (int kb = kb0; kb < kb1; ++kb, ++gb) {
        const int b = gb % NBUF, slot = gb % SLOTS;
        const float w[2] = {__ldg(sb + kb * 2), kb * 2 + 1 < nkb ? __ldg(sb + kb * 2 + 1) : 0.f};
        // tcgen05.ld is warp-collective: the outcome of the waits is made warp-uniform before any lane loads
        ok = __all_sync(0xffffffffu, mbar_wait(&sa_full[slot], (gb / SLOTS) & 1, abort_flag, p.status) &&
                                         mbar_wait(&part_full[b], (gb / NBUF) & 1, abort_flag, p.status));
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t r[32];
          tmem_ld32(tmem + (b * 2 + h) * CN + c0 + quad, r);
          tmem_ld_wait();
          if (h == 1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_remote_tmem(mapa_shared(smem_u32(&part_empty[b]), lead));
          }
          const float4* sa = reinterpret_cast<const float4*>(sSA + (slot * 2 + h) * CN + c0);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float4 s4 = sa[j];
            fma_scaled_pair(acc[4 * j], acc[4 * j + 1], r[4 * j], r[4 * j + 1], s4.x, s4.y, w[h]);
            fma_scaled_pair(acc[4 * j + 2], acc[4 * j + 3], r[4 * j + 2], r[4 * j + 3], s4.z, s4.w, w[h]);
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&sa_empty[slot]);
      }
      const float bias = p.bias && feat_ok ? bf2f(p.bias[feat]) : 0.f;
      // finished sums of the columns [c, c + NC) of the tile
      auto finish = [&](const float* v, int c, auto count) {
        constexpr int NC = decltype(count)::value;
        if (p.out_f32 || !p.paired) {
          const int left = feat_ok ? p.M - t0 - c : 0;
#pragma unroll
          for (int j = 0; j < NC; ++j) {
            if (j >= left) continue;
            const size_t at = (size_t)(t0 + c + j) * p.ldc + feat;
            if (p.out_f32) reinterpret_cast<float*>(p.C)[at] = v[j] + bias;
            else reinterpret_cast<__nv_bfloat16*>(p.C)[at] = __float2bfloat16(v[j] + bias);
          }
          return;
        }
        const int first = t0 + c + (odd ? 1 : 0), left = feat_ok ? p.M - first : 0;
        __nv_bfloat16* C = reinterpret_cast<__nv_bfloat16*>(p.C) + (size_t)first * p.ldc + (feat & ~1);
        const size_t step = (size_t)p.ldc * 2;
#pragma unroll
        for (int j = 0; j < NC; j += 2) {
          const uint32_t own = pack_bf16x2(v[j] + bias, v[j + 1] + bias);
          const uint32_t two = __byte_perm(own, __shfl_xor_sync(0xffffffffu, own, 1), pick);
          if (j < left) *reinterpret_cast<uint32_t*>(C) = two;
          C += step;
        }
      };
      if constexpr (!SPLIT) {
        if (ok) finish(acc, c0, std::integral_constant<int, 32>());
      } else {
        // the exchange of gemm_pair.cu, from registers: groups of 16 columns, pair i owns [i * ng / ks, (i + 1) * ng / ks)
        const int ng = CN / 16, most = (ng + ks - 1) / ks, f = q * 32 + lane;
        bar_sync(2, Cfg::EPI * 32);          // all warps of this CTA have read its last buffers
        if (etid == 0)
          for (int i = 0; i < ks; ++i) mbar_arrive_remote(mapa_shared(smem_u32(ring_free), 2 * i + rank));
        ok = __all_sync(0xffffffffu, mbar_wait_cluster(ring_free, 0, abort_flag, p.status)) && ok;
        if (ok) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int g = c0 / 16 + h, owner = (g * ks + ks - 1) / ng, gl = g - owner * ng / ks;
            const uint32_t dst = mapa_shared(smem_u32(base) + (uint32_t)(((kp * most + gl) * 4 * 128 + f) * 16), 2 * owner + rank);
#pragma unroll
            for (int k = 0; k < 4; ++k)
              st_dsmem_f4(dst + k * 2048, acc[h * 16 + k * 4], acc[h * 16 + k * 4 + 1], acc[h * 16 + k * 4 + 2], acc[h * 16 + k * 4 + 3]);
          }
        }
        fence_acq_rel_cluster();
        bar_sync(2, Cfg::EPI * 32);
        if (etid == 0)
          for (int i = 0; i < ks; ++i) mbar_arrive_remote(mapa_shared(smem_u32(part_ready), 2 * i + rank));
        ok = __all_sync(0xffffffffu, mbar_wait_cluster(part_ready, 0, abort_flag, p.status)) && ok;
        if (!ok || *abort_flag) break;
        const int g0 = kp * ng / ks, g1 = (kp + 1) * ng / ks;
        for (int g = g0 + part; g < g1; g += CN / 32) {
          float v[16];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int i = 0; i < ks; ++i) {
              const float4 x = reinterpret_cast<const float4*>(base)[((i * most + g - g0) * 4 + k) * 128 + f];
              a.x += x.x; a.y += x.y; a.z += x.z; a.w += x.w;
            }
            v[4 * k] = a.x; v[4 * k + 1] = a.y; v[4 * k + 2] = a.z; v[4 * k + 3] = a.w;
          }
          finish(v, g * 16, std::integral_constant<int, 16>());
        }
      }
    }
  }
  tc_fence_before();
  __syncwarp();
  cluster_arrive();                         // no CTA leaves while another still reads its memory or signals its barriers
  cluster_wait();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem, NBUF * 2 * CN);
  }
}

template <int CN, bool SPLIT>
static cudaError_t launch_fp8_pair(const CUtensorMap& tmW, const CUtensorMap& tmX, const CUtensorMap& tmS, const FpParams& p, cudaStream_t stream) {
  using Cfg = FpCfg<CN>;
  auto kern = gemm_fp8_pair_kernel<CN, SPLIT>;
  static PerDeviceOnce configured;
  cudaError_t e = configured.smem_limit(kern, Cfg::SMEM);
  if (e != cudaSuccess) return e;
  const int tiles = ((p.N + 255) / 256) * ((p.M + CN - 1) / CN), most = sm_count() / 2;
  const int pairs = SPLIT ? tiles * p.ks : tiles < most ? tiles : most;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(pairs * 2));
  cfg.blockDim = dim3(Cfg::THREADS);
  cfg.dynamicSmemBytes = Cfg::SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)(2 * p.ks);
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;      // the set-up beside the end of the kernel before (see gemm_pair.cu)
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_pairs() ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kern, tmW, tmX, tmS, p);
}

int pair_cluster_room(int ctas);   // gemm_pair.cu

// Tokens per tile and pairs per tile's K: the least rounds x time of a round, in nanoseconds per step of two blocks (51200 x 5120, 1000
// rows), a microsecond per tile, and some six or nine for the exchange of a split, where all clusters run at once.
static void fp8_pair_shape(int M, int N, int K, int* cn, int* ks) {
  const int tiles_f = (N + 255) / 256, most = sm_count() / 2, steps = (K / 128 + 1) / 2;
  long best = 1L << 60;
  int best_cn = 64, best_ks = 1;
  for (int c = 64; c <= 128; c += 64) {
    if (*cn && c != *cn) continue;
    const long tiles = (long)tiles_f * ((M + c - 1) / c), step = c == 64 ? 465 : 678;
    for (int k = 1; k <= 4 && k <= steps; ++k) {
      if (*ks && k != *ks) continue;
      if (k > 1 && !*ks && (tiles * k > most || tiles > pair_cluster_room(2 * k))) continue;
      const long cost = k == 1 ? (tiles + most - 1) / most * (steps * step + 1000) : (steps + k - 1) / k * step + (c == 64 ? 6500 : 10000);
      if (cost < best) { best = cost; best_cn = c; best_ks = k; }
    }
  }
  *cn = best_cn;
  *ks = best_ks;
}

cudaError_t gemm_fp8_pair(const void* A, long long lda, const void* B, long long ldb, void* C, long long ldc, int M, int N, int K,
                          const float* sa, long long ld_sa, const float* sb, const void* bias, int out_f32, int cn, int ks, cudaStream_t stream) {
  FpParams p = {};
  p.M = M; p.N = N; p.K = K; p.C = C; p.ldc = ldc; p.out_f32 = out_f32;
  p.paired = N % 2 == 0 && ldc % 2 == 0 && (reinterpret_cast<uintptr_t>(C) & 3) == 0;
  p.sb = sb; p.bias = reinterpret_cast<const __nv_bfloat16*>(bias);
  p.status = status_word();
  fp8_pair_shape(M, N, K, &cn, &ks);
  p.ks = ks;
  CUtensorMap tmW, tmX, tmS;
  cudaError_t e = encode_tmap(&tmW, B, 1, (uint64_t)K, N, ldb, 128, 128, 3);
  if (e == cudaSuccess) e = encode_tmap(&tmX, A, 1, (uint64_t)K, M, lda, 128, cn / 2, 3);
  if (e == cudaSuccess) e = encode_tmap(&tmS, sa, 4, (uint64_t)M, K / 128, ld_sa * 4, cn, 2, 0);
  if (e != cudaSuccess) return e;
  if (cn == 64) return ks > 1 ? launch_fp8_pair<64, true>(tmW, tmX, tmS, p, stream) : launch_fp8_pair<64, false>(tmW, tmX, tmS, p, stream);
  return ks > 1 ? launch_fp8_pair<128, true>(tmW, tmX, tmS, p, stream) : launch_fp8_pair<128, false>(tmW, tmX, tmS, p, stream);
}

}  // namespace blz

// As blz_gemm_fp8_block, where the token scales start and step on 16 bytes (ld_sa % 4 == 0).  cn: tokens per tile (64 or 128), ks: pairs
// that share a tile's K (1 - 4, at most one per two blocks); 0 to choose.
BLZ_API int blz_gemm_fp8_pair(const void* A, long long lda, const void* B, long long ldb, void* C, long long ldc, int M, int N, int K,
                              const float* sa, long long ld_sa, const float* sb, const void* bias, int out_f32, int cn, int ks,
                              cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0 || K % 128 || !sa || !sb || ld_sa < M || (cn != 0 && cn != 64 && cn != 128) || ks < 0 || ks > 4 || ks > (K + 255) / 256)
    return (int)cudaErrorInvalidValue;
  return (int)blz::gemm_fp8_pair(A, lda, B, ldb, C, ldc, M, N, K, sa, ld_sa, sb, bias, out_f32, cn, ks, stream);
}
