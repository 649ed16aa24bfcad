// Bandwidth-bound fused ops around the GEMMs:
//   embedding gather; residual-add + RMSNorm (+ NVFP4 / MXFP8 row quantisation for the next GEMM);
//   SwiGLU (+ quantisation); per-head q/k RMSNorm + NeoX rotary + gate split + FP8 paged-KV write in the
//   tcgen05 attention layout; sigmoid gate; argmax with lowest-index ties; row gather.
//
// Same math as the reference's kernels/src/cuda/ops_basic.cu (rmsnorm_kernel :42, attn_prep_kernel :102,
// mul_sigmoid :161, silu_mul :166, argmax_kernel :249, gather_rows :346), kernels/src/cuda/nvfp4_gemm.cu
// quant_rows_kernel :33, kernels/src/cuda/nvfp4_kv.cu kv_store_dense_kernel :188 and embed.cu:6 — fused so
// that each activation makes one trip through HBM between GEMMs.
#include "blaze/glu.cuh"
#include "blaze/host.h"
#include "blaze/sm100.cuh"

namespace blz {

// ---------------------------------------------------------------------------------------------- helpers
__device__ __forceinline__ float block_reduce(float v, float* sh, bool is_max) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = is_max ? warp_max(v) : warp_sum(v);
  __syncthreads();
  if (lane == 0) sh[warp] = v;
  __syncthreads();
  float r = is_max ? -INFINITY : 0.f;
  for (int i = 0; i < nw; ++i) r = is_max ? fmaxf(r, sh[i]) : r + sh[i];
  return r;
}

__device__ __forceinline__ uint8_t f2e4m3(float x) {
  return (uint8_t)__nv_cvt_float_to_fp8(x, __NV_SATFINITE, __NV_E4M3);
}
__device__ __forceinline__ float e4m32f(uint8_t b) {
  __half_raw h = __nv_cvt_fp8_to_halfraw((__nv_fp8_storage_t)b, __NV_E4M3);
  return __half2float(*reinterpret_cast<__half*>(&h));
}
// round to E2M1 code (sign bit 3); nearest, ties to the even code, saturating at 6
__device__ __forceinline__ uint32_t f2e2m1(float x) {
  const float a = fminf(fabsf(x), 6.0f);
  uint32_t c = (a > 0.25f) + (a >= 0.75f) + (a > 1.25f) + (a >= 1.75f) + (a > 2.5f) + (a >= 3.5f) + (a > 5.0f);
  return c | ((__float_as_uint(x) >> 31) << 3);
}
// byte offset of scale (row, col) in the 128x4-tiled scale array with `col_tiles` tiles per row tile
__device__ __forceinline__ size_t sf_offset(int row, int col, int col_tiles) {
  return ((size_t)(row >> 7) * col_tiles + (col >> 2)) * 512 + (row & 31) * 16 + ((row >> 5) & 3) * 4 + (col & 3);
}

// ---------------------------------------------------------------------------------------------- embedding
__global__ void embed_kernel(const __nv_bfloat16* __restrict__ table, const int* __restrict__ tokens,
                             __nv_bfloat16* __restrict__ out, int H, int vocab) {
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x;
  int tok = tokens[t];
  tok = tok < 0 ? 0 : (tok >= vocab ? vocab - 1 : tok);
  if (H % 8) {
    for (int i = threadIdx.x; i < H; i += blockDim.x) out[(size_t)t * H + i] = table[(size_t)tok * H + i];
    return;
  }
  const uint4* src = reinterpret_cast<const uint4*>(table + (size_t)tok * H);
  uint4* dst = reinterpret_cast<uint4*>(out + (size_t)t * H);
  for (int i = threadIdx.x; i < H / 8; i += blockDim.x) dst[i] = src[i];
}

// ---------------------------------------------------------------------------------------------- RMSNorm (+quant)
// QUANT: 0 none (bf16 out), 1 NVFP4 (packed + tiled e4m3 scales + per-row fp32 scale), 2 MXFP8 (e4m3 + tiled e8m0)
template <int QUANT>
__global__ void rmsnorm_kernel(__nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ residual,
                               const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ out,
                               uint8_t* __restrict__ q_out, uint8_t* __restrict__ sf_out, float* __restrict__ row_scale,
                               int H, float eps, int zero_centered, int sf_col_tiles, int zero_src) {
  extern __shared__ __align__(16) uint8_t dyn[];
  __nv_bfloat16* row = reinterpret_cast<__nv_bfloat16*>(dyn);     // the (x + residual) row, then the normed row
  __shared__ float red[32];
  const int t = blockIdx.x;
  __nv_bfloat16* xr = x + (size_t)t * H;
  __nv_bfloat16* rr = residual ? residual + (size_t)t * H : nullptr;
  float ss = 0.f;
  for (int i = threadIdx.x * 8; i < H; i += blockDim.x * 8) {
    uint4 u = *reinterpret_cast<const uint4*>(xr + i);
    if (zero_src) *reinterpret_cast<uint4*>(xr + i) = make_uint4(0, 0, 0, 0);   // hand the accumulation buffer back zeroed
    __nv_bfloat16* e = reinterpret_cast<__nv_bfloat16*>(&u);
    if (rr) {
      uint4 ur = *reinterpret_cast<const uint4*>(rr + i);
      const __nv_bfloat16* er = reinterpret_cast<const __nv_bfloat16*>(&ur);
#pragma unroll
      for (int j = 0; j < 8; ++j) e[j] = __float2bfloat16(bf2f(e[j]) + bf2f(er[j]));
      *reinterpret_cast<uint4*>(rr + i) = u;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) { float f = bf2f(e[j]); ss += f * f; }
    *reinterpret_cast<uint4*>(row + i) = u;
  }
  ss = block_reduce(ss, red, false);
  const float rstd = rsqrtf(ss / H + eps);
  float amax = 0.f;
  for (int i = threadIdx.x * 8; i < H; i += blockDim.x * 8) {
    uint4 u = *reinterpret_cast<uint4*>(row + i);
    uint4 uw = *reinterpret_cast<const uint4*>(w + i);
    __nv_bfloat16* e = reinterpret_cast<__nv_bfloat16*>(&u);
    const __nv_bfloat16* ew = reinterpret_cast<const __nv_bfloat16*>(&uw);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float wf = bf2f(ew[j]) + (zero_centered ? 1.f : 0.f);
      e[j] = __float2bfloat16(bf2f(e[j]) * rstd * wf);
      amax = fmaxf(amax, fabsf(bf2f(e[j])));
    }
    if (QUANT == 0) *reinterpret_cast<uint4*>(out + (size_t)t * H + i) = u;
    else *reinterpret_cast<uint4*>(row + i) = u;
  }
  if (QUANT == 0) return;
  if (QUANT == 1) {
    amax = block_reduce(amax, red, true);
    const float g = fmaxf(amax / (6.f * 448.f), 1e-30f);
    if (threadIdx.x == 0) row_scale[t] = g;
    __syncthreads();
    for (int b = threadIdx.x; b < H / 16; b += blockDim.x) {
      float v[16];
      float bm = 0.f;
#pragma unroll
      for (int j = 0; j < 16; ++j) { v[j] = bf2f(row[b * 16 + j]); bm = fmaxf(bm, fabsf(v[j])); }
      const uint8_t sf = f2e4m3(bm / 6.f / g);
      const float denom = e4m32f(sf) * g;
      const float inv = denom > 0.f ? 1.f / denom : 0.f;
      uint32_t lo = 0, hi = 0;
#pragma unroll
      for (int j = 0; j < 8; ++j) lo |= f2e2m1(denom > 0.f ? v[j] / denom : 0.f) << (4 * j);
#pragma unroll
      for (int j = 0; j < 8; ++j) hi |= f2e2m1(denom > 0.f ? v[8 + j] / denom : 0.f) << (4 * j);
      (void)inv;
      *reinterpret_cast<uint2*>(q_out + (size_t)t * (H / 2) + b * 8) = make_uint2(lo, hi);
      sf_out[sf_offset(t, b, sf_col_tiles)] = sf;
    }
  } else {
    __syncthreads();
    for (int b = threadIdx.x; b < H / 32; b += blockDim.x) {
      float v[32];
      float bm = 0.f;
#pragma unroll
      for (int j = 0; j < 32; ++j) { v[j] = bf2f(row[b * 32 + j]); bm = fmaxf(bm, fabsf(v[j])); }
      bm = fmaxf(bm, 1.17549435e-38f);
      int ex = (int)ceilf(log2f(bm / 448.f));
      ex = max(-127, min(127, ex));
      const float inv = exp2f((float)-ex);
      uint32_t pk[8];
#pragma unroll
      for (int j = 0; j < 8; ++j)
        pk[j] = f2e4m3(v[4 * j] * inv) | (f2e4m3(v[4 * j + 1] * inv) << 8) | (f2e4m3(v[4 * j + 2] * inv) << 16) |
                (f2e4m3(v[4 * j + 3] * inv) << 24);
      uint4* dst = reinterpret_cast<uint4*>(q_out + (size_t)t * H + b * 32);
      dst[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
      dst[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
      sf_out[sf_offset(t, b, sf_col_tiles)] = (uint8_t)(ex + 127);
    }
  }
}

// ---------------------------------------------------------------------------------------------- SwiGLU (+quant)
// gu [T, 2I] = [gate | up];  MODE 0: out bf16 [T, I];  MODE 1: NVFP4;  MODE 2: MXFP8.  Optional plain-row input
// (gate_up == nullptr is invalid).  `src_is_act`: quantise `gu` itself ([T, I], no SwiGLU) — used for attention output.
// `il` (here and in the kernels below): gate and up values in groups of 16 | 16, what a product of interleaved weights stores.
__device__ __forceinline__ int gate_at(int i, int il) { return il ? 2 * i - (i & 15) : i; }
template <int MODE>
__global__ void swiglu_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ out,
                              uint8_t* __restrict__ q_out, uint8_t* __restrict__ sf_out, float* __restrict__ row_scale,
                              int I, int src_is_act, int il, int sf_col_tiles, const int* __restrict__ row_list) {
  extern __shared__ __align__(16) uint8_t dyn[];
  __nv_bfloat16* row = reinterpret_cast<__nv_bfloat16*>(dyn);
  __shared__ float red[32];
  // row_list (optional): the rows to process, one per CTA, -1 = none (routed expert rows in their padded row space)
  const int t = row_list ? row_list[blockIdx.x] : (int)blockIdx.x;
  if (t < 0) return;
  const __nv_bfloat16* g = gu + (size_t)t * (src_is_act ? I : 2 * I);
  const __nv_bfloat16* u = g + (il ? 16 : I);
  float amax = 0.f;
  for (int i = threadIdx.x * 8; i < I; i += blockDim.x * 8) {
    uint4 ug = *reinterpret_cast<const uint4*>(g + gate_at(i, il));
    __nv_bfloat16* eg = reinterpret_cast<__nv_bfloat16*>(&ug);
    if (!src_is_act) {
      uint4 uu = *reinterpret_cast<const uint4*>(u + gate_at(i, il));
      const __nv_bfloat16* eu = reinterpret_cast<const __nv_bfloat16*>(&uu);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float a = bf2f(eg[j]);
        eg[j] = __float2bfloat16(a / (1.f + __expf(-a)) * bf2f(eu[j]));
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(bf2f(eg[j])));
    if (MODE == 0) *reinterpret_cast<uint4*>(out + (size_t)t * I + i) = ug;
    else *reinterpret_cast<uint4*>(row + i) = ug;
  }
  if (MODE == 0) return;
  if (MODE == 1) {
    amax = block_reduce(amax, red, true);
    const float gs = fmaxf(amax / (6.f * 448.f), 1e-30f);
    if (threadIdx.x == 0) row_scale[t] = gs;
    __syncthreads();
    for (int b = threadIdx.x; b < I / 16; b += blockDim.x) {
      float v[16];
      float bm = 0.f;
#pragma unroll
      for (int j = 0; j < 16; ++j) { v[j] = bf2f(row[b * 16 + j]); bm = fmaxf(bm, fabsf(v[j])); }
      const uint8_t sf = f2e4m3(bm / 6.f / gs);
      const float denom = e4m32f(sf) * gs;
      uint32_t lo = 0, hi = 0;
#pragma unroll
      for (int j = 0; j < 8; ++j) lo |= f2e2m1(denom > 0.f ? v[j] / denom : 0.f) << (4 * j);
#pragma unroll
      for (int j = 0; j < 8; ++j) hi |= f2e2m1(denom > 0.f ? v[8 + j] / denom : 0.f) << (4 * j);
      *reinterpret_cast<uint2*>(q_out + (size_t)t * (I / 2) + b * 8) = make_uint2(lo, hi);
      sf_out[sf_offset(t, b, sf_col_tiles)] = sf;
    }
  } else {
    __syncthreads();
    for (int b = threadIdx.x; b < I / 32; b += blockDim.x) {
      float v[32];
      float bm = 0.f;
#pragma unroll
      for (int j = 0; j < 32; ++j) { v[j] = bf2f(row[b * 32 + j]); bm = fmaxf(bm, fabsf(v[j])); }
      bm = fmaxf(bm, 1.17549435e-38f);
      int ex = (int)ceilf(log2f(bm / 448.f));
      ex = max(-127, min(127, ex));
      const float inv = exp2f((float)-ex);
      uint32_t pk[8];
#pragma unroll
      for (int j = 0; j < 8; ++j)
        pk[j] = f2e4m3(v[4 * j] * inv) | (f2e4m3(v[4 * j + 1] * inv) << 8) | (f2e4m3(v[4 * j + 2] * inv) << 16) |
                (f2e4m3(v[4 * j + 3] * inv) << 24);
      uint4* dst = reinterpret_cast<uint4*>(q_out + (size_t)t * I + b * 32);
      dst[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
      dst[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
      sf_out[sf_offset(t, b, sf_col_tiles)] = (uint8_t)(ex + 127);
    }
  }
}

// ---------------------------------------------------------------------------------------------- register-resident rows
// Fast path of the two row kernels above for widths up to 6 chunks of 8 elements per thread: the row never touches
// shared memory, every load of a thread is issued before the first use, and the quantiser works on the registers
// (a 16-element NVFP4 block is two neighbouring threads, a 32-element MXFP8 block four).
__device__ __forceinline__ uint32_t pack_e2m1x8(const float (&v)[8], float inv) {
  uint32_t r;
  asm("{\n"
      ".reg .b8 b0, b1, b2, b3;\n"
      "cvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\n"
      "cvt.rn.satfinite.e2m1x2.f32 b1, %4, %3;\n"
      "cvt.rn.satfinite.e2m1x2.f32 b2, %6, %5;\n"
      "cvt.rn.satfinite.e2m1x2.f32 b3, %8, %7;\n"
      "mov.b32 %0, {b0, b1, b2, b3};\n"
      "}"
      : "=r"(r)
      : "f"(v[0] * inv), "f"(v[1] * inv), "f"(v[2] * inv), "f"(v[3] * inv), "f"(v[4] * inv), "f"(v[5] * inv), "f"(v[6] * inv),
        "f"(v[7] * inv));
  return r;
}
__device__ __forceinline__ uint32_t pack_e4m3x4_f(float a, float b, float c, float d) {
  const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
  const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(c, d), __NV_SATFINITE, __NV_E4M3);
  return lo | (hi << 16);
}

// Quantise this thread's 8 elements [e0, e0+8) of row t, neighbouring lanes holding neighbouring elements (a warp starts at a
// multiple of 256).  Every lane of the warp must call it (shuffles); `valid` gates the stores.
template <int QUANT>
__device__ __forceinline__ void quant_store8(const uint4& packed, bool valid, int t, int e0, int W, float g, uint8_t* q_out,
                                             uint8_t* sf_out, int ct) {
  const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(&packed);
  float v[8];
  float bm = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) { v[j] = valid ? bf2f(e[j]) : 0.f; bm = fmaxf(bm, fabsf(v[j])); }
  bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, 1));
  if (QUANT == 1) {
    const uint8_t sf = f2e4m3(bm / 6.f / g);           // (ties between two scales are common: the same roundings as ever)
    const float denom = e4m32f(sf) * g;
    const float inv = denom > 0.f ? 1.f / denom : 0.f;
    const uint32_t codes = pack_e2m1x8(v, inv);
    if (valid) *reinterpret_cast<uint32_t*>(q_out + (size_t)t * (W / 2) + e0 / 2) = codes;
    if (valid && (e0 & 15) == 0) {
      sf_out[sf_offset(t, e0 >> 4, ct)] = sf;
    }
  } else {
    bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, 2));
    bm = fmaxf(bm, 1.17549435e-38f);
    int ex = (int)ceilf(log2f(bm / 448.f));
    ex = max(-127, min(127, ex));
    const float inv = exp2f((float)-ex);
    if (valid) {
      *reinterpret_cast<uint2*>(q_out + (size_t)t * W + e0) =
          make_uint2(pack_e4m3x4_f(v[0] * inv, v[1] * inv, v[2] * inv, v[3] * inv),
                     pack_e4m3x4_f(v[4] * inv, v[5] * inv, v[6] * inv, v[7] * inv));
    }
    if (valid && (e0 & 31) == 0) {
      sf_out[sf_offset(t, e0 >> 5, ct)] = (uint8_t)(ex + 127);
    }
  }
}

// ---- Rows of many tokens: 16 neighbouring elements per thread, so that an NVFP4 block is one thread's (an MXFP8 block two threads').  The
// quantisers are bound by their instructions, and most of those are per block: two divisions for the scale, one for its reciprocal.
// Magnitudes are compared two at a time on the 16-bit values, and the largest of a block serves the row's maximum too.
__device__ __forceinline__ float lo_f(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float hi_f(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
// largest magnitude of 16 bf16 values (those that are not numbers do not count, as with fmaxf)
__device__ __forceinline__ float amax16(const uint32_t (&w)[8]) {
  __nv_bfloat162 m = __habs2(*reinterpret_cast<const __nv_bfloat162*>(&w[0]));
#pragma unroll
  for (int j = 1; j < 8; ++j) m = __hmax2(m, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&w[j])));
  return fmaxf(fmaxf(0.f, __low2float(m)), __high2float(m));
}
__device__ __forceinline__ void load16(uint32_t (&w)[8], const __nv_bfloat16* src, bool valid) {
  const uint4 z = make_uint4(0, 0, 0, 0);
  const uint4 a = valid ? reinterpret_cast<const uint4*>(src)[0] : z, b = valid ? reinterpret_cast<const uint4*>(src)[1] : z;
  w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w;
  w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
}
// Quantise 16 elements [e0, e0 + 16) of row t, of which `bm` is the largest magnitude; every lane of the warp calls it, a warp starts at a
// multiple of 512.  Four scales of neighbours make one store.
template <int QUANT>
__device__ __forceinline__ void quant_store16(const uint32_t (&w)[8], float bm, bool valid, int t, int e0, int W, float g, uint8_t* q_out,
                                              uint8_t* sf_out, int ct) {
  const int lane = threadIdx.x & 31;
  if (QUANT == 1) {
    const uint8_t sf = f2e4m3(bm / 6.f / g);           // the same roundings as quant_store8
    const float denom = e4m32f(sf) * g;
    const float inv = denom > 0.f ? 1.f / denom : 0.f;
    uint32_t codes[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float v[8];
#pragma unroll
      for (int j = 0; j < 4; ++j) { v[2 * j] = lo_f(w[4 * h + j]); v[2 * j + 1] = hi_f(w[4 * h + j]); }
      codes[h] = pack_e2m1x8(v, inv);
    }
    if (valid) *reinterpret_cast<uint2*>(q_out + (size_t)t * (W / 2) + e0 / 2) = make_uint2(codes[0], codes[1]);
    uint32_t four = valid ? (uint32_t)sf << (8 * (lane & 3)) : 0u;
    four |= __shfl_xor_sync(0xffffffffu, four, 1);
    four |= __shfl_xor_sync(0xffffffffu, four, 2);
    if (valid && (lane & 3) == 0) *reinterpret_cast<uint32_t*>(sf_out + sf_offset(t, e0 >> 4, ct)) = four;
  } else {
    bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, 1));
    bm = fmaxf(bm, 1.17549435e-38f);
    int ex = (int)ceilf(log2f(bm / 448.f));
    ex = max(-127, min(127, ex));
    const float inv = exp2f((float)-ex);
    uint32_t q[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) q[j] = pack_e4m3x4_f(lo_f(w[2 * j]) * inv, hi_f(w[2 * j]) * inv, lo_f(w[2 * j + 1]) * inv, hi_f(w[2 * j + 1]) * inv);
    if (valid) *reinterpret_cast<uint4*>(q_out + (size_t)t * W + e0) = make_uint4(q[0], q[1], q[2], q[3]);
    uint32_t four = valid ? (uint32_t)(ex + 127) << (8 * ((lane >> 1) & 3)) : 0u;
    four |= __shfl_xor_sync(0xffffffffu, four, 2);
    four |= __shfl_xor_sync(0xffffffffu, four, 4);
    if (valid && (lane & 7) == 0) *reinterpret_cast<uint32_t*>(sf_out + sf_offset(t, e0 >> 5, ct)) = four;
  }
}

// The squares are added up in the order of rmsnorm_reg_kernel with `sum_threads` threads of 8 elements per pass: another order moves the
// root's last bit, and with it whole 4-bit codes, some in a few rows of thousands.  Where those threads take one pass, a thread here has the
// elements of two neighbours of theirs, and 16 lanes add up what a warp would; else the rows go by way of shared memory
// (8192 rows of 4096 in NVFP4 from cold caches: 53 us with 8 elements per thread, 51 so; within a step 45, where handing the first pass's sums
// on to the threads of the second instead of the rows took 44).
template <int QUANT, int CH>
__global__ void __launch_bounds__(256) rmsnorm_row16_kernel(__nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ residual,
                                                              const __nv_bfloat16* __restrict__ w, uint8_t* __restrict__ q_out,
                                                              uint8_t* __restrict__ sf_out, float* __restrict__ row_scale, int H,
                                                              float eps, int zero_centered, int sf_col_tiles, int zero_src, int sum_threads) {
  pdl_trigger();
  pdl_wait();
  extern __shared__ __align__(16) uint4 row16[];
  __shared__ float red[32];
  const int t = blockIdx.x;
  __nv_bfloat16* xr = x + (size_t)t * H;
  __nv_bfloat16* rr = residual ? residual + (size_t)t * H : nullptr;
  uint32_t u[CH][8];
  const bool one_pass = CH == 1 && H / 8 <= sum_threads;
  {
    uint32_t r[CH][8];
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      const int i = (c * blockDim.x + threadIdx.x) * 16;
      load16(u[c], xr + i, i < H);
      if (rr) load16(r[c], rr + i, i < H);
    }
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      const int i = (c * blockDim.x + threadIdx.x) * 16;
      if (i < H && zero_src) {
        reinterpret_cast<uint4*>(xr + i)[0] = make_uint4(0, 0, 0, 0);
        reinterpret_cast<uint4*>(xr + i)[1] = make_uint4(0, 0, 0, 0);
      }
      if (rr) {
#pragma unroll
        for (int j = 0; j < 8; ++j) u[c][j] = pack_bf16x2(lo_f(u[c][j]) + lo_f(r[c][j]), hi_f(u[c][j]) + hi_f(r[c][j]));
        if (i < H) {
          reinterpret_cast<uint4*>(rr + i)[0] = make_uint4(u[c][0], u[c][1], u[c][2], u[c][3]);
          reinterpret_cast<uint4*>(rr + i)[1] = make_uint4(u[c][4], u[c][5], u[c][6], u[c][7]);
        }
      }
      if (!one_pass && i < H) {
        row16[i / 8] = make_uint4(u[c][0], u[c][1], u[c][2], u[c][3]);
        row16[i / 8 + 1] = make_uint4(u[c][4], u[c][5], u[c][6], u[c][7]);
      }
    }
  }
  float ss = 0.f;
  if (one_pass) {
    float p[2] = {0.f, 0.f};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      p[j / 4] = fmaf(lo_f(u[0][j]), lo_f(u[0][j]), p[j / 4]);
      p[j / 4] = fmaf(hi_f(u[0][j]), hi_f(u[0][j]), p[j / 4]);
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
      p[0] += __shfl_xor_sync(0xffffffffu, p[0], o);
      p[1] += __shfl_xor_sync(0xffffffffu, p[1], o);
    }
    if ((threadIdx.x & 15) == 0) red[threadIdx.x >> 4] = p[0] + p[1];
    __syncthreads();
    for (int i = 0; i < (int)blockDim.x >> 4; ++i) ss += red[i];
  } else {
    __syncthreads();
    for (int sw = threadIdx.x >> 5; sw < sum_threads >> 5; sw += blockDim.x >> 5) {
      float part = 0.f;
      for (int g = sw * 32 + (threadIdx.x & 31); g < H / 8; g += sum_threads) {
        const uint4 v = row16[g];
        const uint32_t e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) { part = fmaf(lo_f(e[j]), lo_f(e[j]), part); part = fmaf(hi_f(e[j]), hi_f(e[j]), part); }
      }
      part = warp_sum(part);
      if ((threadIdx.x & 31) == 0) red[sw] = part;
    }
    __syncthreads();
    for (int i = 0; i < sum_threads >> 5; ++i) ss += red[i];
  }
  const float rstd = rsqrtf(ss / H + eps);
  float bm[CH], amax = 0.f;
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int i = (c * blockDim.x + threadIdx.x) * 16;
    uint32_t uw[8];
    load16(uw, w + i, i < H);
    const float one = zero_centered ? 1.f : 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j)
      u[c][j] = pack_bf16x2(lo_f(u[c][j]) * rstd * (lo_f(uw[j]) + one), hi_f(u[c][j]) * rstd * (hi_f(uw[j]) + one));
    bm[c] = amax16(u[c]);
    amax = fmaxf(amax, bm[c]);
  }
  float g = 1.f;
  if (QUANT == 1) {
    amax = block_reduce(amax, red, true);
    g = fmaxf(amax / (6.f * 448.f), 1e-30f);
    if (threadIdx.x == 0) row_scale[t] = g;
  }
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int i = (c * blockDim.x + threadIdx.x) * 16;
    quant_store16<QUANT>(u[c], bm[c], i < H, t, i, H, g, q_out, sf_out, sf_col_tiles);
  }
}

// ACT: the source rows are activations already (no up half).
template <int MODE, int CH, bool ACT>
__global__ void __launch_bounds__(256) swiglu_row16_kernel(const __nv_bfloat16* __restrict__ gu, uint8_t* __restrict__ q_out,
                                                             uint8_t* __restrict__ sf_out, float* __restrict__ row_scale, int I, int il,
                                                             int sf_col_tiles, const int* __restrict__ row_list) {
  pdl_trigger();
  pdl_wait();
  __shared__ float red[32];
  const int t = row_list ? row_list[blockIdx.x] : (int)blockIdx.x;
  if (t < 0) return;
  const __nv_bfloat16* src = gu + (size_t)t * (ACT ? I : 2 * I);
  uint32_t a[CH][8], b[ACT ? 1 : CH][8];
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int i = (c * blockDim.x + threadIdx.x) * 16;
    load16(a[c], src + gate_at(i, il), i < I);
    if constexpr (!ACT) load16(b[c], src + (il ? 16 : I) + gate_at(i, il), i < I);
  }
  float bm[CH], amax = 0.f;
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    if constexpr (!ACT) {
#pragma unroll
      for (int j = 0; j < 8; ++j) a[c][j] = pack_bf16x2(silu(lo_f(a[c][j])) * lo_f(b[c][j]), silu(hi_f(a[c][j])) * hi_f(b[c][j]));
    }
    bm[c] = amax16(a[c]);
    amax = fmaxf(amax, bm[c]);
  }
  float gs = 1.f;
  if (MODE == 1) {
    amax = block_reduce(amax, red, true);
    gs = fmaxf(amax / (6.f * 448.f), 1e-30f);
    if (threadIdx.x == 0) row_scale[t] = gs;
  }
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int i = (c * blockDim.x + threadIdx.x) * 16;
    quant_store16<MODE>(a[c], bm[c], i < I, t, i, I, gs, q_out, sf_out, sf_col_tiles);
  }
}

// Rows of at most 1024 activations, several per CTA (see swiglu_rows_kernel): a warp, or two, per row.
template <int MODE>
__global__ void __launch_bounds__(256) quant_rows16_kernel(const __nv_bfloat16* __restrict__ act, uint8_t* __restrict__ q_out,
                                                             uint8_t* __restrict__ sf_out, float* __restrict__ row_scale, int I,
                                                             int sf_col_tiles, const int* __restrict__ row_list, int n_rows, int tpr) {
  pdl_trigger();
  pdl_wait();
  __shared__ float red[8];
  const int sub = threadIdx.x / tpr, in_row = threadIdx.x - sub * tpr;
  const int r = blockIdx.x * (blockDim.x / tpr) + sub;
  int t = -1;
  if (r < n_rows) t = row_list ? row_list[r] : r;
  const bool live = t >= 0;
  const int i = in_row * 16;
  const bool valid = live && i < I;
  uint32_t a[8];
  load16(a, act + (size_t)(live ? t : 0) * I + i, valid);
  const float bm = amax16(a);
  float gs = 1.f;
  if (MODE == 1) {
    float m = warp_max(bm);
    if (tpr > 32) {
      if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
      __syncthreads();
      m = 0.f;
      for (int k = 0; k < (tpr >> 5); ++k) m = fmaxf(m, red[((sub * tpr) >> 5) + k]);
    }
    gs = fmaxf(m / (6.f * 448.f), 1e-30f);
    if (live && in_row == 0) row_scale[t] = gs;
  }
  quant_store16<MODE>(a, bm, valid, live ? t : 0, i, I, gs, q_out, sf_out, sf_col_tiles);
}

template <int QUANT, int CH>
__global__ void __launch_bounds__(512) rmsnorm_reg_kernel(__nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ residual,
                                                            const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ out,
                                                            uint8_t* __restrict__ q_out, uint8_t* __restrict__ sf_out,
                                                            float* __restrict__ row_scale, int H, float eps, int zero_centered,
                                                            int sf_col_tiles, int zero_src) {
  pdl_trigger();
  pdl_wait();
  __shared__ float red[32];
  const int t = blockIdx.x;
  __nv_bfloat16* xr = x + (size_t)t * H;
  __nv_bfloat16* rr = residual ? residual + (size_t)t * H : nullptr;
  uint4 u[CH], ur[CH];
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int i = (c * blockDim.x + threadIdx.x) * 8;
    u[c] = ur[c] = make_uint4(0, 0, 0, 0);
    if (i < H) {
      u[c] = *reinterpret_cast<const uint4*>(xr + i);
      if (rr) ur[c] = *reinterpret_cast<const uint4*>(rr + i);
    }
  }
  float ss = 0.f;
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int i = (c * blockDim.x + threadIdx.x) * 8;
    __nv_bfloat16* e = reinterpret_cast<__nv_bfloat16*>(&u[c]);
    if (i < H) {
      if (zero_src) *reinterpret_cast<uint4*>(xr + i) = make_uint4(0, 0, 0, 0);
      if (rr) {
        const __nv_bfloat16* er = reinterpret_cast<const __nv_bfloat16*>(&ur[c]);
#pragma unroll
        for (int j = 0; j < 8; ++j) e[j] = __float2bfloat16(bf2f(e[j]) + bf2f(er[j]));
        *reinterpret_cast<uint4*>(rr + i) = u[c];
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) { const float f = bf2f(e[j]); ss += f * f; }
  }
  ss = block_reduce(ss, red, false);
  const float rstd = rsqrtf(ss / H + eps);
  float amax = 0.f;
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int i = (c * blockDim.x + threadIdx.x) * 8;
    __nv_bfloat16* e = reinterpret_cast<__nv_bfloat16*>(&u[c]);
    const uint4 uw = i < H ? *reinterpret_cast<const uint4*>(w + i) : make_uint4(0, 0, 0, 0);   // the weight row stays in L1/L2
    const __nv_bfloat16* ew = reinterpret_cast<const __nv_bfloat16*>(&uw);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float wf = bf2f(ew[j]) + (zero_centered ? 1.f : 0.f);
      e[j] = __float2bfloat16(bf2f(e[j]) * rstd * wf);
      if (QUANT) amax = fmaxf(amax, fabsf(bf2f(e[j])));
    }
    if (QUANT == 0 && i < H) *reinterpret_cast<uint4*>(out + (size_t)t * H + i) = u[c];
  }
  if (QUANT == 0) return;
  float g = 1.f;
  if (QUANT == 1) {
    amax = block_reduce(amax, red, true);
    g = fmaxf(amax / (6.f * 448.f), 1e-30f);
    if (threadIdx.x == 0) row_scale[t] = g;
  }
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int i = (c * blockDim.x + threadIdx.x) * 8;
    quant_store8<QUANT>(u[c], i < H, t, i, H, g, q_out, sf_out, sf_col_tiles);
  }
}

// Gated rows; ACT (bf16 out only): the source rows are activations already.
template <int MODE, int CH, bool ACT>
__global__ void __launch_bounds__(512) swiglu_reg_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ out,
                                                           uint8_t* __restrict__ q_out, uint8_t* __restrict__ sf_out,
                                                           float* __restrict__ row_scale, int I, int il, int sf_col_tiles,
                                                           const int* __restrict__ row_list) {
  pdl_trigger();
  pdl_wait();
  __shared__ float red[32];
  // row_list (optional): the rows to process, one per CTA, -1 = none (routed expert rows in their padded row space)
  const int t = row_list ? row_list[blockIdx.x] : (int)blockIdx.x;
  if (t < 0) return;
  const __nv_bfloat16* g = gu + (size_t)t * (ACT ? I : 2 * I);
  const __nv_bfloat16* up = g + (il ? 16 : I);
  uint4 a[CH], b[ACT ? 1 : CH];
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int i = (c * blockDim.x + threadIdx.x) * 8;
    a[c] = make_uint4(0, 0, 0, 0);
    if constexpr (!ACT) b[c] = a[c];
    if (i < I) {
      a[c] = *reinterpret_cast<const uint4*>(g + gate_at(i, il));
      if constexpr (!ACT) b[c] = *reinterpret_cast<const uint4*>(up + gate_at(i, il));
    }
  }
  float amax = 0.f;
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int i = (c * blockDim.x + threadIdx.x) * 8;
    __nv_bfloat16* eg = reinterpret_cast<__nv_bfloat16*>(&a[c]);
    const __nv_bfloat16* eu = reinterpret_cast<const __nv_bfloat16*>(&b[ACT ? 0 : c]);
    if constexpr (!ACT) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float x = bf2f(eg[j]);
        eg[j] = __float2bfloat16(silu(x) * bf2f(eu[j]));
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(bf2f(eg[j])));
    if (MODE == 0 && i < I) *reinterpret_cast<uint4*>(out + (size_t)t * I + i) = a[c];
  }
  if (MODE == 0) return;
  float gs = 1.f;
  if (MODE == 1) {
    amax = block_reduce(amax, red, true);
    gs = fmaxf(amax / (6.f * 448.f), 1e-30f);
    if (threadIdx.x == 0) row_scale[t] = gs;
  }
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int i = (c * blockDim.x + threadIdx.x) * 8;
    quant_store8<MODE>(a[c], i < I, t, i, I, gs, q_out, sf_out, sf_col_tiles);
  }
}

// Rows of at most 1024 activations (expert intermediates): several rows per CTA, `tpr` threads each (a multiple of 32, so
// a warp never spans two rows), instead of one mostly idle 256-thread CTA per row.  Entry r of the launch handles row
// row_list[r] (or r); -1 and entries beyond n_rows are skipped.
template <int MODE>
__global__ void __launch_bounds__(256) swiglu_rows_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ out,
                                                            uint8_t* __restrict__ q_out, uint8_t* __restrict__ sf_out,
                                                            float* __restrict__ row_scale, int I, int src_is_act, int il, int sf_col_tiles,
                                                            const int* __restrict__ row_list, int n_rows, int tpr) {
  pdl_trigger();
  pdl_wait();
  __shared__ float red[8];
  const int sub = threadIdx.x / tpr, in_row = threadIdx.x - sub * tpr;
  const int r = blockIdx.x * (blockDim.x / tpr) + sub;
  int t = -1;
  if (r < n_rows) t = row_list ? row_list[r] : r;
  const bool live = t >= 0;
  const int i = in_row * 8;
  const bool valid = live && i < I;
  uint4 a = make_uint4(0, 0, 0, 0), b = a;
  if (valid) {
    const __nv_bfloat16* g = gu + (size_t)t * (src_is_act ? I : 2 * I);
    a = *reinterpret_cast<const uint4*>(g + gate_at(i, il));
    if (!src_is_act) b = *reinterpret_cast<const uint4*>(g + (il ? 16 : I) + gate_at(i, il));
  }
  __nv_bfloat16* eg = reinterpret_cast<__nv_bfloat16*>(&a);
  const __nv_bfloat16* eu = reinterpret_cast<const __nv_bfloat16*>(&b);
  float amax = 0.f;
  if (!src_is_act) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float x = bf2f(eg[j]);
      eg[j] = __float2bfloat16(silu(x) * bf2f(eu[j]));
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(bf2f(eg[j])));
  if (MODE == 0) {
    if (valid) *reinterpret_cast<uint4*>(out + (size_t)t * I + i) = a;
    return;
  }
  float gs = 1.f;
  if (MODE == 1) {
    // the row's largest magnitude: over the warp, then over the row's warps
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
    __syncthreads();
    float m = 0.f;
    for (int k = 0; k < (tpr >> 5); ++k) m = fmaxf(m, red[((sub * tpr) >> 5) + k]);
    gs = fmaxf(m / (6.f * 448.f), 1e-30f);
    if (live && in_row == 0) row_scale[t] = gs;
  }
  quant_store8<MODE>(a, valid, live ? t : 0, i, I, gs, q_out, sf_out, sf_col_tiles);
}

// ---------------------------------------------------------------------------------------------- attention prep
// One CTA per token; its warps walk the token's heads.  Heads 0..Hq-1 are query heads, then Hkv key heads, then Hkv
// value heads.  qkv row layout: [q heads (x2 when gated: q | gate per head)] [k heads] [v heads].  The rotary
// sine/cosine pairs of the token are computed once into shared memory and reused by every q and k head.
template <int D>
__global__ void __launch_bounds__(512) attn_prep_kernel(const __nv_bfloat16* __restrict__ qkv, __nv_bfloat16* __restrict__ q_out,
                                 __nv_bfloat16* __restrict__ gate_out, uint8_t* __restrict__ kv_pool,
                                 const int* __restrict__ positions, const int* __restrict__ slot_mapping,
                                 const float* __restrict__ inv_freq, const __nv_bfloat16* __restrict__ q_norm_w,
                                 const __nv_bfloat16* __restrict__ k_norm_w, int T, int Hq, int Hkv, int rot_dim,
                                 float eps, float rope_scale, int gated, int zero_centered, float k_scale_inv,
                                 float v_scale_inv, long long page_stride, long long head_stride, int rotate,
                                 long long pos_stride, int mrope0, int mrope1) {
  pdl_trigger();
  pdl_wait();
  constexpr int VPL = D / 32;
  __shared__ float2 cs[D / 2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int t = blockIdx.x;
  const int heads = Hq + 2 * Hkv;
  const int half = rot_dim / 2;
  {
    // M-RoPE (pos_stride > 0): positions is [3, T]; frequency i follows the temporal stream below mrope0, the height stream
    // below mrope1, the width stream above (reference: attn_prep_kernel<MROPE>, kernels/src/cuda/ops_basic.cu:102)
    const float p0 = (float)positions[t];
    const float p1 = pos_stride > 0 ? (float)positions[pos_stride + t] : p0;
    const float p2 = pos_stride > 0 ? (float)positions[2 * pos_stride + t] : p0;
    for (int i = threadIdx.x; i < half; i += blockDim.x) {
      const float pos = pos_stride > 0 ? (i < mrope0 ? p0 : (i < mrope1 ? p1 : p2)) : p0;
      float s, c;
      sincosf(pos * inv_freq[i], &s, &c);
      cs[i] = make_float2(c * rope_scale, s * rope_scale);
    }
  }
  __syncthreads();
  const int qw = Hq * D * (gated ? 2 : 1);
  const size_t row_w = (size_t)qw + 2 * (size_t)Hkv * D;
  const __nv_bfloat16* row = qkv + t * row_w;
  const int lanes_half = half / VPL;          // partner lane distance (power of two)
  const int slot = slot_mapping[t];
  float nwq[VPL], nwk[VPL];
#pragma unroll
  for (int j = 0; j < VPL; ++j) {
    nwq[j] = q_norm_w ? bf2f(q_norm_w[lane * VPL + j]) + (zero_centered ? 1.f : 0.f) : 0.f;
    nwk[j] = k_norm_w ? bf2f(k_norm_w[lane * VPL + j]) + (zero_centered ? 1.f : 0.f) : 0.f;
  }
  for (int h = warp; h < heads; h += nwarps) {
    const __nv_bfloat16* src;
    int kind;  // 0 q, 1 k, 2 v
    if (h < Hq) { kind = 0; src = row + (size_t)h * D * (gated ? 2 : 1); }
    else if (h < Hq + Hkv) { kind = 1; src = row + qw + (size_t)(h - Hq) * D; }
    else { kind = 2; src = row + qw + (size_t)Hkv * D + (size_t)(h - Hq - Hkv) * D; }
    if (kind != 0 && slot < 0) continue;
    __align__(16) __nv_bfloat16 raw[VPL];
    if constexpr (VPL == 4) *reinterpret_cast<uint2*>(raw) = *reinterpret_cast<const uint2*>(src + lane * 4);
    else if constexpr (VPL == 8) *reinterpret_cast<uint4*>(raw) = *reinterpret_cast<const uint4*>(src + lane * 8);
    else *reinterpret_cast<uint32_t*>(raw) = *reinterpret_cast<const uint32_t*>(src + lane * 2);
    float v[VPL];
#pragma unroll
    for (int j = 0; j < VPL; ++j) v[j] = bf2f(raw[j]);
    if (kind == 0 && gated) {
      __nv_bfloat16* gdst = gate_out + ((size_t)t * Hq + h) * D + lane * VPL;
      if constexpr (VPL == 4) *reinterpret_cast<uint2*>(gdst) = *reinterpret_cast<const uint2*>(src + D + lane * 4);
      else if constexpr (VPL == 8) *reinterpret_cast<uint4*>(gdst) = *reinterpret_cast<const uint4*>(src + D + lane * 8);
      else *reinterpret_cast<uint32_t*>(gdst) = *reinterpret_cast<const uint32_t*>(src + D + lane * 2);
    }
    if (kind < 2) {
      if (kind == 0 ? q_norm_w != nullptr : k_norm_w != nullptr) {
        float ss = 0.f;
#pragma unroll
        for (int j = 0; j < VPL; ++j) ss += v[j] * v[j];
        ss = warp_sum(ss);
        const float rstd = rsqrtf(ss / D + eps);
#pragma unroll
        for (int j = 0; j < VPL; ++j) v[j] = bf2f(__float2bfloat16(v[j] * rstd * (kind == 0 ? nwq[j] : nwk[j])));
      }
      // NeoX rotary over the first rot_dim dims: pairs (i, i + half)
#pragma unroll
      for (int j = 0; j < VPL; ++j) {
        const int i = lane * VPL + j;
        const float other = __shfl_xor_sync(0xffffffffu, v[j], lanes_half);
        if (i < rot_dim) {
          const float2 c = cs[i < half ? i : i - half];
          v[j] = i < half ? v[j] * c.x - other * c.y : v[j] * c.x + other * c.y;
        }
      }
      // Optional randomised Hadamard rotation of q and k (the same orthogonal map on both keeps q.k; it spreads
      // outliers over the head before the key is rounded to e4m3): sign flip by a fixed hash of the element index,
      // then a Walsh-Hadamard transform over the D elements the warp holds, scaled by 1/sqrt(D).
      if (rotate) {
#pragma unroll
        for (int j = 0; j < VPL; ++j)
          if (((uint32_t)(lane * VPL + j) * 2654435761u >> 15) & 1u) v[j] = -v[j];
#pragma unroll
        for (int st = 1; st < VPL; st <<= 1) {
#pragma unroll
          for (int j = 0; j < VPL; ++j)
            if (!(j & st)) { const float a = v[j], b = v[j | st]; v[j] = a + b; v[j | st] = a - b; }
        }
#pragma unroll
        for (int m = 1; m < 32; m <<= 1) {
#pragma unroll
          for (int j = 0; j < VPL; ++j) {
            const float other = __shfl_xor_sync(0xffffffffu, v[j], m);
            v[j] = (lane & m) ? other - v[j] : v[j] + other;
          }
        }
        const float sc = rsqrtf((float)D);
#pragma unroll
        for (int j = 0; j < VPL; ++j) v[j] *= sc;
      }
    }
    if (kind == 0) {
      __align__(16) __nv_bfloat16 o[VPL];
#pragma unroll
      for (int j = 0; j < VPL; ++j) o[j] = __float2bfloat16(v[j]);
      __nv_bfloat16* dst = q_out + ((size_t)t * Hq + h) * D + lane * VPL;
      if constexpr (VPL == 4) *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(o);
      else if constexpr (VPL == 8) *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(o);
      else *reinterpret_cast<uint32_t*>(dst) = *reinterpret_cast<const uint32_t*>(o);
      continue;
    }
    const int page = slot >> 4, tp = slot & 15;
    const int kh = kind == 1 ? h - Hq : h - Hq - Hkv;
    uint8_t* blk = kv_pool + (size_t)page * page_stride + (size_t)kh * head_stride;
    if (kind == 1) {
      // the lane's VPL dims are consecutive bytes of one 16-byte core-matrix row
      __align__(8) uint8_t b[VPL];
#pragma unroll
      for (int j = 0; j < VPL; ++j) b[j] = f2e4m3(bf2f(__float2bfloat16(v[j])) * k_scale_inv);
      const int i0 = lane * VPL;
      uint8_t* dst = blk + (tp >> 3) * 8 * D + (i0 >> 4) * 128 + (tp & 7) * 16 + (i0 & 15);
      if constexpr (VPL == 4) *reinterpret_cast<uint32_t*>(dst) = *reinterpret_cast<const uint32_t*>(b);
      else if constexpr (VPL == 8) *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(b);
      else *reinterpret_cast<uint16_t*>(dst) = *reinterpret_cast<const uint16_t*>(b);
    } else {
#pragma unroll
      for (int j = 0; j < VPL; ++j) {
        const int i = lane * VPL + j;
        blk[16 * D + i * 16 + tp] = f2e4m3(v[j] * v_scale_inv);
      }
    }
  }
}

// The same for head_dim 128 and 256 without the Hadamard rotation, 8 dims per lane: D / 8 lanes per head, so the rotary pairs and
// norm weights of a lane's dims stay in registers for all heads, and a warp does two heads of 128 at once.
// Values: one token's value is a byte in each of D 16-byte rows of its page (V is kept transposed), and a byte costs the memory
// system what a sector does.  With `v_blocks`, a page that 16 consecutive tokens fill is written as whole rows by a block of its own
// (one per 16 tokens behind the T token blocks, for the page that begins among them); the token blocks write the other values.
// Measured on a B200, 8192 tokens, 32 + 2 x 8 heads of 128 (184 MB, 28 us at copy bandwidth): 117 us by head and token
// (220 instructions per head and warp, byte stores of the values), now 63 us.
template <int D>
__global__ void __launch_bounds__(512) attn_prep_heads_kernel(const __nv_bfloat16* __restrict__ qkv, __nv_bfloat16* __restrict__ q_out,
                                 __nv_bfloat16* __restrict__ gate_out, uint8_t* __restrict__ kv_pool,
                                 const int* __restrict__ positions, const int* __restrict__ slot_mapping,
                                 const float* __restrict__ inv_freq, const __nv_bfloat16* __restrict__ q_norm_w,
                                 const __nv_bfloat16* __restrict__ k_norm_w, int T, int Hq, int Hkv, int rot_dim,
                                 float eps, float rope_scale, int gated, int zero_centered, float k_scale_inv,
                                 float v_scale_inv, long long page_stride, long long head_stride, int v_blocks,
                                 long long pos_stride, int mrope0, int mrope1) {
  pdl_trigger();
  pdl_wait();
  constexpr int LPH = D / 8, HPW = 32 / LPH;          // lanes per head, heads per warp
  constexpr int PART = D / 32;                        // dims of a partial sum of squares
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int qw = Hq * D * (gated ? 2 : 1);
  const size_t row_w = (size_t)qw + 2 * (size_t)Hkv * D;
  if ((int)blockIdx.x >= T) {
    // ---- values of the page that tokens fill from one of t0 .. t0 + 15 on (there is one such page at most)
    __shared__ int s_slot[31];
    const int t0 = ((int)blockIdx.x - T) * 16;
    if (threadIdx.x < 31) s_slot[threadIdx.x] = t0 + (int)threadIdx.x < T ? slot_mapping[t0 + threadIdx.x] : -1;
    __syncthreads();
    constexpr int VPL = D / 32;
    for (int i = 0; i < 16; ++i) {
      const int slot = s_slot[i];
      if (slot < 0 || (slot & 15) != 0 || !__all_sync(0xffffffffu, s_slot[i + (lane & 15)] == slot + (lane & 15))) continue;
      for (int h = warp; h < Hkv; h += nwarps) {
        const __nv_bfloat16* src = qkv + (size_t)(t0 + i) * row_w + qw + (size_t)(Hkv + h) * D + lane * VPL;
        uint8_t* dst = kv_pool + (size_t)(slot >> 4) * page_stride + (size_t)h * head_stride + 16 * D + lane * VPL * 16;
        uint32_t word[VPL][4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          __align__(16) __nv_bfloat16 raw[4][VPL];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if constexpr (VPL == 4) *reinterpret_cast<uint2*>(raw[j]) = *reinterpret_cast<const uint2*>(src + (size_t)(4 * k + j) * row_w);
            else *reinterpret_cast<uint4*>(raw[j]) = *reinterpret_cast<const uint4*>(src + (size_t)(4 * k + j) * row_w);
          }
#pragma unroll
          for (int d = 0; d < VPL; ++d)
            word[d][k] = pack_e4m3x4_f(bf2f(raw[0][d]) * v_scale_inv, bf2f(raw[1][d]) * v_scale_inv, bf2f(raw[2][d]) * v_scale_inv,
                                       bf2f(raw[3][d]) * v_scale_inv);
        }
#pragma unroll
        for (int d = 0; d < VPL; ++d) *reinterpret_cast<uint4*>(dst + d * 16) = make_uint4(word[d][0], word[d][1], word[d][2], word[d][3]);
      }
      return;
    }
    return;
  }
  __shared__ float2 cs[D / 2];
  const int t = blockIdx.x;
  const int half = rot_dim / 2;
  {
    // M-RoPE as above
    const float p0 = (float)positions[t];
    const float p1 = pos_stride > 0 ? (float)positions[pos_stride + t] : p0;
    const float p2 = pos_stride > 0 ? (float)positions[2 * pos_stride + t] : p0;
    for (int i = threadIdx.x; i < half; i += blockDim.x) {
      const float pos = pos_stride > 0 ? (i < mrope0 ? p0 : (i < mrope1 ? p1 : p2)) : p0;
      float s, c;
      sincosf(pos * inv_freq[i], &s, &c);
      cs[i] = make_float2(c * rope_scale, s * rope_scale);
    }
  }
  const int sub = lane / LPH, i0 = (lane % LPH) * 8;  // the lane's head of the warp's, and its first dim
  const int lanes_half = half / 8;                    // partner lane distance (power of two)
  const bool turned = i0 < rot_dim;
  const int slot = slot_mapping[t];
  bool paged = false;                                 // a block of its own writes this token's values (same in all warps)
  if (v_blocks && slot >= 0) {
    const int begin = t - (slot & 15), at = lane & 15;
    if (begin >= 0 && begin + 15 < T) paged = __all_sync(0xffffffffu, slot_mapping[begin + at] == (slot & ~15) + at);
  }
  const __nv_bfloat16* row = qkv + t * row_w;
  uint4 wq = make_uint4(0, 0, 0, 0), wk = wq;
  if (q_norm_w) wq = *reinterpret_cast<const uint4*>(q_norm_w + i0);
  if (k_norm_w) wk = *reinterpret_cast<const uint4*>(k_norm_w + i0);
  __syncthreads();
  // a lane's dims all lie in the first half of the pairs, in the second, or beyond: x cos - y sin, or y sin + x cos (the last product
  // is the one that is rounded by itself)
  const bool first = i0 < half;
  float2 rot[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    rot[j] = make_float2(1.f, 0.f);
    if (turned) {
      const float2 cj = cs[first ? i0 + j : i0 + j - half];
      rot[j] = first ? make_float2(cj.x, -cj.y) : make_float2(cj.y, cj.x);
    }
  }
  const int heads = Hq + (paged ? Hkv : 2 * Hkv);
  for (int h0 = warp * HPW; h0 < heads; h0 += nwarps * HPW) {
    const int h = h0 + sub;
    const bool is_q = h < Hq, is_v = h >= Hq + Hkv, live = h < heads && (is_q || slot >= 0);
    const __nv_bfloat16* src = row + (is_q ? (size_t)h * D * (gated ? 2 : 1) : (size_t)qw + (size_t)(h - Hq) * D) + i0;
    uint4 raw = make_uint4(0, 0, 0, 0);
    if (live) raw = *reinterpret_cast<const uint4*>(src);
    const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(&raw);
    // squares are summed as the kernel above does: 32 partial sums per head, added up by a butterfly from the farthest
    float v[8], sq[8 / PART];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      v[j] = bf2f(e[j]);
      sq[j / PART] = j % PART == 0 ? v[j] * v[j] : fmaf(v[j], v[j], sq[j / PART]);
    }
    if (live && is_q && gated)
      *reinterpret_cast<uint4*>(gate_out + ((size_t)t * Hq + h) * D + i0) = *reinterpret_cast<const uint4*>(src + D);
#pragma unroll
    for (int o = LPH / 2; o > 0; o >>= 1) {
#pragma unroll
      for (int j = 0; j < 8 / PART; ++j) sq[j] += __shfl_xor_sync(0xffffffffu, sq[j], o);
    }
    const float ss = PART == 8 ? sq[0] : sq[0] + sq[8 / PART - 1];
    if (!is_v && (is_q ? q_norm_w != nullptr : k_norm_w != nullptr)) {
      const float rstd = rsqrtf(ss / D + eps);
      const uint4 w8 = is_q ? wq : wk;
      const __nv_bfloat16* w = reinterpret_cast<const __nv_bfloat16*>(&w8);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = bf2f(__float2bfloat16(v[j] * rstd * (bf2f(w[j]) + (zero_centered ? 1.f : 0.f))));
    }
    float o[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float other = __shfl_xor_sync(0xffffffffu, v[j], lanes_half);
      const float turn = fmaf(first ? v[j] : other, rot[j].x, (first ? other : v[j]) * rot[j].y);
      o[j] = is_v || !turned ? v[j] : turn;
    }
    if (!live) continue;                                // (no shuffle follows in this iteration)
    if (is_q) {
      *reinterpret_cast<uint4*>(q_out + ((size_t)t * Hq + h) * D + i0) =
          make_uint4(pack_bf16x2(o[0], o[1]), pack_bf16x2(o[2], o[3]), pack_bf16x2(o[4], o[5]), pack_bf16x2(o[6], o[7]));
      continue;
    }
    uint8_t* blk = kv_pool + (size_t)(slot >> 4) * page_stride + (size_t)(is_v ? h - Hq - Hkv : h - Hq) * head_stride;
    const int tp = slot & 15;
    if (is_v) {
#pragma unroll
      for (int j = 0; j < 8; ++j) blk[16 * D + (i0 + j) * 16 + tp] = f2e4m3(o[j] * v_scale_inv);
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = bf2f(__float2bfloat16(o[j])) * k_scale_inv;
      // the lane's dims are half of a 16-byte core-matrix row
      *reinterpret_cast<uint2*>(blk + (tp >> 3) * 8 * D + (i0 >> 4) * 128 + (tp & 7) * 16 + (i0 & 15)) =
          make_uint2(pack_e4m3x4_f(o[0], o[1], o[2], o[3]), pack_e4m3x4_f(o[4], o[5], o[6], o[7]));
    }
  }
}

// Elementwise kernels on bf16, V elements per access: 8 or 4 where pointers and sizes allow, else 1 (see each_width).
template <int V> struct EachWord { typedef uint4 type; };
template <> struct EachWord<4> { typedef uint2 type; };
template <> struct EachWord<1> { typedef __nv_bfloat16 type; };
// out[i] = f(a[i], b[i]) for i < n (out may be a)
template <int V, typename F>
__device__ __forceinline__ void each(const __nv_bfloat16* a, const __nv_bfloat16* b, __nv_bfloat16* out, size_t n, size_t first, size_t step, F f) {
  typedef typename EachWord<V>::type W;
  for (size_t i = first; i < n / V; i += step) {
    const W wa = reinterpret_cast<const W*>(a)[i], wb = reinterpret_cast<const W*>(b)[i];
    W wo;
    const __nv_bfloat16 *x = reinterpret_cast<const __nv_bfloat16*>(&wa), *y = reinterpret_cast<const __nv_bfloat16*>(&wb);
    __nv_bfloat16* z = reinterpret_cast<__nv_bfloat16*>(&wo);
#pragma unroll
    for (int j = 0; j < V; ++j) z[j] = __float2bfloat16(f(bf2f(x[j]), bf2f(y[j])));
    reinterpret_cast<W*>(out)[i] = wo;
  }
}
// (the division sets the pace: wider accesses make a thread's divisions wait for one another, 1.1 - 1.4 times as long up to 10 M elements)
__global__ void mul_sigmoid_kernel(__nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ gate, size_t n) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    x[i] = __float2bfloat16(bf2f(x[i]) / (1.f + __expf(-bf2f(gate[i]))));
}
template <int V>
__global__ void add_kernel(const __nv_bfloat16* a, const __nv_bfloat16* b, __nv_bfloat16* out, size_t n) {
  each<V>(a, b, out, n, (size_t)blockIdx.x * blockDim.x + threadIdx.x, (size_t)gridDim.x * blockDim.x, [](float x, float y) { return x + y; });
}
// out[t, :] = a[t, :] + b[t, :] * bf16(sigmoid(gate_logit[t]))
template <int V>
__global__ void add_sigmoid_scaled_kernel(const __nv_bfloat16* a, const __nv_bfloat16* b, const __nv_bfloat16* gl,
                                          __nv_bfloat16* out, int H) {
  const size_t row = (size_t)blockIdx.x * H;
  const float s = bf2f(__float2bfloat16(1.f / (1.f + __expf(-bf2f(gl[blockIdx.x])))));
  each<V>(a + row, b + row, out + row, H, threadIdx.x, blockDim.x, [s](float x, float y) { return x + y * s; });
}
__global__ void gather_rows_kernel(const __nv_bfloat16* __restrict__ x, const int* __restrict__ rows,
                                   __nv_bfloat16* __restrict__ out, int H) {
  const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)rows[blockIdx.x] * H);
  uint4* dst = reinterpret_cast<uint4*>(out + (size_t)blockIdx.x * H);
  for (int i = threadIdx.x; i < H / 8; i += blockDim.x) dst[i] = src[i];
}

// argmax over fp32 rows, lowest index wins ties; writes int64 ids (and optionally the max value)
__global__ void argmax_kernel(const float* __restrict__ logits, long long* __restrict__ out, float* __restrict__ out_val,
                              int V, long long ld, int index_offset) {
  pdl_trigger();
  pdl_wait();
  __shared__ float sv[32];
  __shared__ int si[32];
  const float* row = logits + (size_t)blockIdx.x * ld;
  float best = -INFINITY;
  int bi = 0x7fffffff;
  for (int i = threadIdx.x; i < V; i += blockDim.x) {
    const float x = row[i];
    if (x > best || (x == best && i < bi)) { best = x; bi = i; }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) { sv[warp] = best; si[warp] = bi; }
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
    best = lane < nw ? sv[lane] : -INFINITY;
    bi = lane < nw ? si[lane] : 0x7fffffff;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
    if (lane == 0) {
      out[blockIdx.x] = (long long)(bi == 0x7fffffff ? 0 : bi) + index_offset;
      if (out_val) out_val[blockIdx.x] = best;
    }
  }
}

// Reduce the per-tile (value, column) pairs of the greedy head: one warp per row, ties to the lower column.
__global__ void argmax_parts_kernel(const float* __restrict__ val, const int* __restrict__ idx, int tiles, int M,
                                    long long* __restrict__ out, float* __restrict__ out_val, int index_offset) {
  pdl_trigger();
  pdl_wait();
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= M) return;
  float bv = -INFINITY;
  int bi = 0x7fffffff;
  for (int t = lane; t < tiles; t += 32) {
    const float v = val[(size_t)t * M + row];
    const int i = idx[(size_t)t * M + row];
    if (v > bv || (v == bv && i < bi)) { bv = v; bi = i; }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
  }
  if (lane == 0) {
    out[row] = (long long)bi + index_offset;
    if (out_val) out_val[row] = bv;
  }
}

}  // namespace blz

using namespace blz;
typedef __nv_bfloat16 bf16;

// Rows of more than 40 KB (beyond 20480 elements) in shared memory, on any device of the process.
static cudaError_t allow_smem(size_t bytes) {
  if (bytes <= 40 * 1024) return cudaSuccess;
  static PerDeviceOnce once[7];
  constexpr int MOST = 100 * 1024;
  cudaError_t e = once[0].smem_limit(swiglu_kernel<1>, MOST);
  if (e == cudaSuccess) e = once[1].smem_limit(swiglu_kernel<2>, MOST);
  if (e == cudaSuccess) e = once[2].smem_limit(rmsnorm_kernel<0>, MOST);
  if (e == cudaSuccess) e = once[3].smem_limit(rmsnorm_kernel<1>, MOST);
  if (e == cudaSuccess) e = once[4].smem_limit(rmsnorm_kernel<2>, MOST);
  if (e == cudaSuccess) e = once[5].smem_limit(rmsnorm_row16_kernel<1, 6>, MOST);
  if (e == cudaSuccess) e = once[6].smem_limit(rmsnorm_row16_kernel<2, 6>, MOST);
  return e;
}

// threads and chunks per thread of the register-resident row kernels; chunks == 0: width not covered
// Few rows (a decode step) cannot fill the GPU with 256-thread CTAs: they get up to 512 threads per row, which shortens
// each row's dependency chain; BLAZE_ROW_THREADS=256 restores one shape for all.
static inline void reg_shape(int W, int T, int* threads, int* chunks) {
  static int wide_rows = -1;
  if (wide_rows < 0) { const char* e = getenv("BLAZE_ROW_THREADS"); wide_rows = (e && atoi(e) == 256) ? 0 : 1; }
  *threads = W <= 12288 ? 256 : 512;
  if (wide_rows && T <= 1024 && W >= 4096) *threads = 512;
  const int ch = (W + *threads * 8 - 1) / (*threads * 8);
  *chunks = (W % 32 == 0 && ch <= 6) ? ch : 0;
}

#define BLZ_CH_SWITCH(ch, CALL)                                                                    \
  switch (ch) {                                                                                     \
    case 1: CALL(1); break; case 2: CALL(2); break; case 3: CALL(3); break; case 4: CALL(4); break; \
    case 5: CALL(5); break; default: CALL(6); break;                                                \
  }

// The quantising row kernels with 16 elements per thread: rows of up to 6 chunks of 256 threads.  At any number of rows where rows are
// normed or are activations already (but for few long norms and few rows of 513 - 1024, see there) (us before / now: 8192 rows of 12288 activations, NVFP4, 77 / 46, 1 row 3.35 / 3.10; norms, from
// cold caches, of 825 rows of 4096 14.3 / 12.3, 3000 of 5120 34.8 / 28.7, 2000 of 12320 76 / 49), for gated rows from 512 on (825 rows of 12288 19.8 / 17.1, 256 rows 7.6 / 8.3: their
// activation is the longer chain per thread there; the experts' short gated rows likewise 43.7 / 46.2).
constexpr int ROW16_MOST = 6 * 256 * 16;
static inline int row16_threads(int W, int chunks) { return (W / 16 + chunks * 32 - 1) / (chunks * 32) * 32; }

static inline int norm_threads(int H) {
  int t = H / 8;
  t = (t + 31) / 32 * 32;
  return t < 32 ? 32 : (t > 1024 ? 1024 : t);
}

BLZ_API int blz_embed(const void* table, const int* tokens, void* out, int T, int H, int vocab, cudaStream_t s) {
  if (T == 0) return 0;
  launch_pdl(embed_kernel, dim3(T), dim3(256), 0, s, (const bf16*)table, tokens, (bf16*)out, H, vocab);
  return (int)cudaGetLastError();
}

// quant: 0 → bf16 `out`; 1 → NVFP4 (q_out [T, H/2], sf_out tiled, row_scale [T]); 2 → MXFP8 (q_out [T, H], sf_out tiled)
BLZ_API int blz_rmsnorm(void* x, void* residual, const void* w, void* out, void* q_out, void* sf_out,
                        float* row_scale, int T, int H, float eps, int zero_centered, int quant, int zero_src, cudaStream_t s) {
  if (H % 32 || T < 0) return (int)cudaErrorInvalidValue;
  if (T == 0) return 0;
  const int thr = norm_threads(H);
  const size_t sm = (size_t)H * 2;
  if (cudaError_t e = allow_smem(sm)) return (int)e;
  const int ct = quant == 1 ? (H + 63) / 64 : (H + 127) / 128;
  int rt, ch;
  reg_shape(H, T, &rt, &ch);
  // Few long rows: the sums of rmsnorm_row16_kernel go by way of shared memory there, with two more barriers (us, 8 / 16 elements a
  // thread: MXFP8 1 row of 5120 3.50 / 3.81, of 7168 3.50 / 4.00, 64 rows of 12288 4.51 / 5.12, 96 of 24576 7.42 / 8.01; NVFP4 16 rows of
  // 4096 3.03 / 3.32, 1 of 12288 4.47 / 4.92; 150 rows of 5120 5.13 / 4.78, of 12288 6.84 / 6.42).  Few rows of two warps: see swiglu_impl.
  const bool few = T <= 128 && (H >= 4096 || (H > 512 && H <= 1024));
  if (quant && H <= ROW16_MOST && !few) {
    const int c16 = (H + 4095) / 4096;
    const size_t sm16 = c16 == 1 && H / 8 <= rt ? 0 : sm;          // (see rmsnorm_row16_kernel)
#define BLZ_RN(C)                                                                                                              \
  if (quant == 1) launch_pdl(rmsnorm_row16_kernel<1, C>, dim3(T), dim3(row16_threads(H, C)), sm16, s, (bf16*)x, (bf16*)residual, (const bf16*)w, (uint8_t*)q_out, (uint8_t*)sf_out, row_scale, H, eps, zero_centered, ct, zero_src, rt); \
  else launch_pdl(rmsnorm_row16_kernel<2, C>, dim3(T), dim3(row16_threads(H, C)), sm16, s, (bf16*)x, (bf16*)residual, (const bf16*)w, (uint8_t*)q_out, (uint8_t*)sf_out, row_scale, H, eps, zero_centered, ct, zero_src, rt)
    BLZ_CH_SWITCH(c16, BLZ_RN)
#undef BLZ_RN
    return (int)cudaGetLastError();
  }
  if (ch) {
#define BLZ_RN2(Q, C) launch_pdl(rmsnorm_reg_kernel<Q, C>, dim3(T), dim3(rt), 0, s, (bf16*)x, (bf16*)residual, (const bf16*)w, (bf16*)out, (uint8_t*)q_out, (uint8_t*)sf_out, row_scale, H, eps, zero_centered, ct, zero_src)
#define BLZ_RN(C) if (quant == 0) BLZ_RN2(0, C); else if (quant == 1) BLZ_RN2(1, C); else BLZ_RN2(2, C)
    BLZ_CH_SWITCH(ch, BLZ_RN)
#undef BLZ_RN
#undef BLZ_RN2
    return (int)cudaGetLastError();
  }
  if (quant == 0)
    rmsnorm_kernel<0><<<T, thr, sm, s>>>((bf16*)x, (bf16*)residual, (const bf16*)w, (bf16*)out, nullptr, nullptr, nullptr, H, eps, zero_centered, 0, zero_src);
  else if (quant == 1)
    rmsnorm_kernel<1><<<T, thr, sm, s>>>((bf16*)x, (bf16*)residual, (const bf16*)w, nullptr, (uint8_t*)q_out, (uint8_t*)sf_out, row_scale, H, eps, zero_centered, ct, zero_src);
  else
    rmsnorm_kernel<2><<<T, thr, sm, s>>>((bf16*)x, (bf16*)residual, (const bf16*)w, nullptr, (uint8_t*)q_out, (uint8_t*)sf_out, row_scale, H, eps, zero_centered, ct, zero_src);
  return (int)cudaGetLastError();
}

// mode as `quant` above; src_is_act = 1 quantises the [T, I] input as is (no SwiGLU), 2: gate and up values in groups of 16 | 16.  blz_swiglu_live: T entries of row_list
// name the rows to process (-1 = skip): the live rows of the routed experts' padded row space.
static int swiglu_impl(const void* gu, void* out, void* q_out, void* sf_out, float* row_scale, int T, int I,
                       int mode, int src_is_act, const int* row_list, cudaStream_t s);
BLZ_API int blz_swiglu(const void* gu, void* out, void* q_out, void* sf_out, float* row_scale, int T, int I,
                       int mode, int src_is_act, cudaStream_t s) {
  return swiglu_impl(gu, out, q_out, sf_out, row_scale, T, I, mode, src_is_act, nullptr, s);
}
BLZ_API int blz_swiglu_live(const void* gu, void* out, void* q_out, void* sf_out, float* row_scale, int T, int I,
                            int mode, int src_is_act, const int* row_list, cudaStream_t s) {
  return swiglu_impl(gu, out, q_out, sf_out, row_scale, T, I, mode, src_is_act, row_list, s);
}
static int swiglu_impl(const void* gu, void* out, void* q_out, void* sf_out, float* row_scale, int T, int I,
                       int mode, int src_is_act, const int* row_list, cudaStream_t s) {
  const int il = src_is_act == 2;
  if (il) src_is_act = 0;
  if (I % 32 || T < 0) return (int)cudaErrorInvalidValue;
  if (T == 0) return 0;
  const int thr = norm_threads(I);
  const size_t sm = (size_t)I * 2;
  if (cudaError_t e = allow_smem(sm)) return (int)e;
  const int ct = mode == 1 ? (I + 63) / 64 : (I + 127) / 128;
  {
    // Two warps of 16 elements a thread lose to three or four of 8 while all rows are few (us, 8 / 16 elements a thread: NVFP4 4 rows of 768
    // 2.40 / 2.76, 512 rows 2.44 / 2.90, 1024 rows 2.74 / 2.93, 4 rows of 1024 2.22 / 2.48, 150 rows 2.52 / 2.74; MXFP8 4 rows of 768
    // 2.04 / 2.43; but 4096 rows of 1024 in NVFP4 6.25 / 4.20); one warp does not (4 rows of 512 2.30 / 2.39).
    const int tpr16 = (I / 16 + 31) / 32 * 32;
    if (mode && src_is_act && I <= 1024 && (I <= 512 || (long long)T * I > 3 << 18)) {
      const int per = 256 / tpr16;
      const dim3 grid((T + per - 1) / per), block(per * tpr16);
      if (mode == 1) launch_pdl(quant_rows16_kernel<1>, grid, block, 0, s, (const bf16*)gu, (uint8_t*)q_out, (uint8_t*)sf_out, row_scale, I, ct, row_list, T, tpr16);
      else launch_pdl(quant_rows16_kernel<2>, grid, block, 0, s, (const bf16*)gu, (uint8_t*)q_out, (uint8_t*)sf_out, row_scale, I, ct, row_list, T, tpr16);
      return (int)cudaGetLastError();
    }
    const int tpr = (I / 8 + 31) / 32 * 32, rows_per = tpr <= 128 ? 256 / tpr : 1;
    if (I <= 1024 && rows_per >= 2) {
      const dim3 grid((T + rows_per - 1) / rows_per), block(rows_per * tpr);
      if (mode == 0) launch_pdl(swiglu_rows_kernel<0>, grid, block, 0, s, (const bf16*)gu, (bf16*)out, (uint8_t*)nullptr, (uint8_t*)nullptr, (float*)nullptr, I, src_is_act, il, 0, row_list, T, tpr);
      else if (mode == 1) launch_pdl(swiglu_rows_kernel<1>, grid, block, 0, s, (const bf16*)gu, (bf16*)nullptr, (uint8_t*)q_out, (uint8_t*)sf_out, row_scale, I, src_is_act, il, ct, row_list, T, tpr);
      else launch_pdl(swiglu_rows_kernel<2>, grid, block, 0, s, (const bf16*)gu, (bf16*)nullptr, (uint8_t*)q_out, (uint8_t*)sf_out, row_scale, I, src_is_act, il, ct, row_list, T, tpr);
      return (int)cudaGetLastError();
    }
  }
  int rt, ch;
  reg_shape(I, T, &rt, &ch);
  if (mode && I <= ROW16_MOST && (src_is_act || T >= 512)) {
    const int c16 = (I + 4095) / 4096;
#define BLZ_SW2(Q, C, ACT) launch_pdl(swiglu_row16_kernel<Q, C, ACT>, dim3(T), dim3(row16_threads(I, C)), 0, s, (const bf16*)gu, (uint8_t*)q_out, (uint8_t*)sf_out, row_scale, I, il, ct, row_list)
#define BLZ_SW(C) if (mode == 1) { if (src_is_act) BLZ_SW2(1, C, true); else BLZ_SW2(1, C, false); } else { if (src_is_act) BLZ_SW2(2, C, true); else BLZ_SW2(2, C, false); }
    BLZ_CH_SWITCH(c16, BLZ_SW)
#undef BLZ_SW
#undef BLZ_SW2
    return (int)cudaGetLastError();
  }
  if (ch && !(mode && src_is_act)) {
#define BLZ_SW(C)                                                                                                              \
  if (src_is_act) launch_pdl(swiglu_reg_kernel<0, C, true>, dim3(T), dim3(rt), 0, s, (const bf16*)gu, (bf16*)out, (uint8_t*)nullptr, (uint8_t*)nullptr, (float*)nullptr, I, il, 0, row_list); \
  else if (mode == 0) launch_pdl(swiglu_reg_kernel<0, C, false>, dim3(T), dim3(rt), 0, s, (const bf16*)gu, (bf16*)out, (uint8_t*)nullptr, (uint8_t*)nullptr, (float*)nullptr, I, il, 0, row_list); \
  else if (mode == 1) launch_pdl(swiglu_reg_kernel<1, C, false>, dim3(T), dim3(rt), 0, s, (const bf16*)gu, (bf16*)nullptr, (uint8_t*)q_out, (uint8_t*)sf_out, row_scale, I, il, ct, row_list); \
  else launch_pdl(swiglu_reg_kernel<2, C, false>, dim3(T), dim3(rt), 0, s, (const bf16*)gu, (bf16*)nullptr, (uint8_t*)q_out, (uint8_t*)sf_out, row_scale, I, il, ct, row_list)
    BLZ_CH_SWITCH(ch, BLZ_SW)
#undef BLZ_SW
    return (int)cudaGetLastError();
  }
  if (mode == 0) swiglu_kernel<0><<<T, thr, 0, s>>>((const bf16*)gu, (bf16*)out, nullptr, nullptr, nullptr, I, src_is_act, il, 0, row_list);
  else if (mode == 1) swiglu_kernel<1><<<T, thr, sm, s>>>((const bf16*)gu, nullptr, (uint8_t*)q_out, (uint8_t*)sf_out, row_scale, I, src_is_act, il, ct, row_list);
  else swiglu_kernel<2><<<T, thr, sm, s>>>((const bf16*)gu, nullptr, (uint8_t*)q_out, (uint8_t*)sf_out, row_scale, I, src_is_act, il, ct, row_list);
  return (int)cudaGetLastError();
}

// longest: the most new tokens of a sequence (host knowledge): a page that one step fills takes 16.
BLZ_API int blz_attn_prep_runs(const void* qkv, void* q_out, void* gate_out, void* kv_pool, const int* positions,
                               const int* slot_mapping, const float* inv_freq, const void* q_norm_w, const void* k_norm_w,
                               int T, int Hq, int Hkv, int D, int rot_dim, float eps, float rope_scale, int gated,
                               int zero_centered, float k_scale, float v_scale, long long page_stride, long long head_stride,
                               int rotate, long long pos_stride, int mrope0, int mrope1, int longest, cudaStream_t s) {
  if (T == 0) return 0;
  const int half = rot_dim / 2, vpl = D / 32;
  if ((D != 64 && D != 128 && D != 256) || rot_dim > D || half % vpl || ((half / vpl) & (half / vpl - 1)) || half / vpl > 16)
    return (int)cudaErrorInvalidValue;
  // decode-sized steps: more warps per token shorten the per-token chain (launch bound of the kernel: 512 threads)
  int wpb = (Hq + 2 * Hkv) >= 8 ? 8 : (Hq + 2 * Hkv);
  { static int wide = -1; if (wide < 0) { const char* e = getenv("BLAZE_ROW_THREADS"); wide = (e && atoi(e) == 256) ? 0 : 1; }
    if (wide && T <= 1024 && (Hq + 2 * Hkv) >= 16) wpb = 16; }
  // 8 dims per lane: head_dim 128 and 256, no rotation, the rotated pairs a whole number of lanes apart, rows on 16 bytes
  const bool on16 = !((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(q_out) | reinterpret_cast<uintptr_t>(gate_out) |
                       reinterpret_cast<uintptr_t>(q_norm_w) | reinterpret_cast<uintptr_t>(k_norm_w) | reinterpret_cast<uintptr_t>(kv_pool)) & 15);
  // ... except for many single tokens of few heads, which the kernel by single heads spreads over more warps (8 + 2 x 8 heads of 128,
  // 700 tokens of decode steps: 11.0 us there, 12.2 here).
  const int heads = Hq + 2 * Hkv, sms = sm_count();
  if (D != 64 && !rotate && half % 8 == 0 && half > 0 && on16 && page_stride % 16 == 0 && head_stride % 16 == 0 &&
      (longest >= 16 || heads > 24 || T <= sms)) {
    // Values in blocks of their own where the step may fill pages, from 64 tokens on.  A warp for every pass over the heads as long as
    // there is a block per SM, so that nothing waits in turn; then blocks of eight warps, and of four from some four blocks per SM
    // on.  Over the kernel by single heads, 4 / 8 / 12 / 16 warps: 32 + 2 x 8 heads of 128, prompts of 128 tokens 0.85 / 0.73 / 0.66 /
    // 0.70, 384 tokens 0.61 / 0.59 / 0.82 / 0.78, 1024 tokens 0.48 / 0.56 / 0.73 / 0.79; 700 single tokens 1.01 / 1.02 / 1.11 / 1.15;
    // 16 + 2 x 2 gated heads of 256, 700 tokens 0.50 / 0.63 / 0.77 / 1.07.
    const int v_blocks = T >= 64 && longest >= 16 ? (T + 15) / 16 : 0, hpw = 256 / D;
    const int passes = (heads + hpw - 1) / hpw, most = T <= sms ? 12 : T <= 4 * sms ? 8 : 4;
    const int warps = passes < 4 ? 4 : passes > most ? most : passes;
#define BLZ_PREP(DD)                                                                                                 \
  launch_pdl(attn_prep_heads_kernel<DD>, dim3(T + v_blocks), dim3(warps * 32), 0, s, (const bf16*)qkv, (bf16*)q_out,     \
             (bf16*)gate_out, (uint8_t*)kv_pool, positions, slot_mapping, inv_freq, (const bf16*)q_norm_w,              \
             (const bf16*)k_norm_w, T, Hq, Hkv, rot_dim, eps, rope_scale, gated, zero_centered, 1.f / k_scale,          \
             1.f / v_scale, page_stride > 0 ? page_stride : (long long)Hkv * 2 * 16 * D,                                \
             head_stride > 0 ? head_stride : (long long)2 * 16 * D, v_blocks, pos_stride, mrope0, mrope1)
    if (D == 128) BLZ_PREP(128); else BLZ_PREP(256);
#undef BLZ_PREP
    return (int)cudaGetLastError();
  }
  const int grid = T;
#define BLZ_PREP(DD)                                                                                                 \
  launch_pdl(attn_prep_kernel<DD>, dim3(grid), dim3(wpb * 32), 0, s, (const bf16*)qkv, (bf16*)q_out, (bf16*)gate_out,  \
             (uint8_t*)kv_pool, positions, slot_mapping, inv_freq, (const bf16*)q_norm_w, (const bf16*)k_norm_w, T, Hq, \
             Hkv, rot_dim, eps, rope_scale, gated, zero_centered, 1.f / k_scale, 1.f / v_scale,                         \
             page_stride > 0 ? page_stride : (long long)Hkv * 2 * 16 * D, head_stride > 0 ? head_stride : (long long)2 * 16 * D, \
             rotate, pos_stride, mrope0, mrope1)
  if (D == 64) BLZ_PREP(64); else if (D == 128) BLZ_PREP(128); else BLZ_PREP(256);
#undef BLZ_PREP
  return (int)cudaGetLastError();
}

BLZ_API int blz_attn_prep(const void* qkv, void* q_out, void* gate_out, void* kv_pool, const int* positions,
                          const int* slot_mapping, const float* inv_freq, const void* q_norm_w, const void* k_norm_w,
                          int T, int Hq, int Hkv, int D, int rot_dim, float eps, float rope_scale, int gated,
                          int zero_centered, float k_scale, float v_scale, long long page_stride, long long head_stride,
                          int rotate, long long pos_stride, int mrope0, int mrope1, cudaStream_t s) {
  return blz_attn_prep_runs(qkv, q_out, gate_out, kv_pool, positions, slot_mapping, inv_freq, q_norm_w, k_norm_w, T, Hq, Hkv, D, rot_dim,
                            eps, rope_scale, gated, zero_centered, k_scale, v_scale, page_stride, head_stride, rotate, pos_stride, mrope0,
                            mrope1, T, s);
}

namespace blz {
// Copy the K and V rows of KV slot src[m] to slot dst[m] in every KV head of one layer's pool (page layout of the
// attention kernels: K as 8-row x 16-byte core matrices, V transposed).  Used after a draft tree has been verified: the
// accepted path's rows move down to consecutive positions.  Moves seg[i] .. seg[i+1]-1 belong to sequence i and run in
// list order inside one CTA (a later move may overwrite the source of an earlier one: row 2 -> 1, then row 5 -> 2);
// different sequences never share a slot.  Reference: blz_move_rows (kernels/src/cuda/tree.cu :142).
__global__ void kv_move_rows_kernel(uint8_t* pool, const int* __restrict__ src, const int* __restrict__ dst,
                                    const int* __restrict__ seg, int D, long long page_stride, long long head_stride) {
  for (int m = seg[blockIdx.x]; m < seg[blockIdx.x + 1]; ++m) {
    const int s = src[m], d = dst[m];
    if (s != d && s >= 0 && d >= 0) {
      const uint8_t* sb = pool + (size_t)(s >> 4) * page_stride + (size_t)blockIdx.y * head_stride;
      uint8_t* db = pool + (size_t)(d >> 4) * page_stride + (size_t)blockIdx.y * head_stride;
      const int st = s & 15, dt = d & 15;
      for (int c = threadIdx.x; c < D / 16; c += blockDim.x)
        *reinterpret_cast<uint4*>(db + (dt >> 3) * 8 * D + c * 128 + (dt & 7) * 16) =
            *reinterpret_cast<const uint4*>(sb + (st >> 3) * 8 * D + c * 128 + (st & 7) * 16);
      for (int i = threadIdx.x; i < D; i += blockDim.x) db[16 * D + i * 16 + dt] = sb[16 * D + i * 16 + st];
    }
    __syncthreads();
  }
}

}  // namespace blz
BLZ_API int blz_kv_move_rows(void* pool, const int* src, const int* dst, const int* seg, int num_seqs, int Hkv, int D,
                             long long page_stride, long long head_stride, cudaStream_t s) {
  if (num_seqs <= 0) return 0;
  if (D % 16 || Hkv <= 0 || page_stride <= 0 || head_stride <= 0 || page_stride % 16 || head_stride % 16)
    return (int)cudaErrorInvalidValue;
  blz::kv_move_rows_kernel<<<dim3(num_seqs, Hkv), 128, 0, s>>>((uint8_t*)pool, src, dst, seg, D, page_stride, head_stride);
  return (int)cudaGetLastError();
}

// Elements per access that n elements at these places allow.  One block per 256 accesses and rows' blocks without idle passes: sum of
// 256 x 4096 2.5 us with single elements, 2.3 with eight (3.3 with a grid for single elements), 8192 x 4096 78 and 32; rows with a
// gate 1000 x 5120 7.2 and 5.4 (8.8 in blocks of 256 threads), 8192 x 4096 75 and 41.
static int each_width(long long n, const void* a, const void* b, const void* c) {
  const uintptr_t at = reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c);
  return n % 8 == 0 && !(at & 15) ? 8 : n % 4 == 0 && !(at & 7) ? 4 : 1;
}
#define BLZ_EACH(V, CALL) { if (V == 8) { constexpr int W = 8; CALL; } else if (V == 4) { constexpr int W = 4; CALL; } else { constexpr int W = 1; CALL; } }
BLZ_API int blz_mul_sigmoid(void* x, const void* gate, long long n, cudaStream_t s) {
  if (n == 0) return 0;
  mul_sigmoid_kernel<<<(int)((n + 1023) / 1024 > 4096 ? 4096 : (n + 1023) / 1024), 256, 0, s>>>((bf16*)x, (const bf16*)gate, (size_t)n);
  return (int)cudaGetLastError();
}
BLZ_API int blz_add(const void* a, const void* b, void* out, long long n, cudaStream_t s) {
  if (n == 0) return 0;
  const int v = each_width(n, a, b, out);
  const long long blocks = (n / v + 255) / 256, most = 1 << 20;
  BLZ_EACH(v, (add_kernel<W><<<(unsigned)(blocks < most ? blocks : most), 256, 0, s>>>((const bf16*)a, (const bf16*)b, (bf16*)out, (size_t)n)))
  return (int)cudaGetLastError();
}
BLZ_API int blz_add_sigmoid_scaled(const void* a, const void* b, const void* gl, void* out, int T, int H, cudaStream_t s) {
  if (T == 0) return 0;
  // blocks of up to 512 threads, of 256 where there are rows for all SMs several times over
  const int v = each_width(H, a, b, out), items = H / v, most = T >= 2048 ? 256 : 512, passes = (items + most - 1) / most;
  const int threads = passes ? ((items + passes - 1) / passes + 31) / 32 * 32 : 32;
  BLZ_EACH(v, (add_sigmoid_scaled_kernel<W><<<T, threads, 0, s>>>((const bf16*)a, (const bf16*)b, (const bf16*)gl, (bf16*)out, H)))
  return (int)cudaGetLastError();
}
#undef BLZ_EACH
BLZ_API int blz_gather_rows(const void* x, const int* rows, void* out, int R, int H, cudaStream_t s) {
  if (R == 0) return 0;
  if (H % 8) return (int)cudaErrorInvalidValue;
  gather_rows_kernel<<<R, 256, 0, s>>>((const bf16*)x, rows, (bf16*)out, H);
  return (int)cudaGetLastError();
}
BLZ_API int blz_argmax(const float* logits, long long* out, float* out_val, int R, int V, long long ld, int index_offset,
                       cudaStream_t s) {
  if (R == 0) return 0;
  launch_pdl(argmax_kernel, dim3(R), dim3(1024), 0, s, logits, out, out_val, V, ld, index_offset);
  return (int)cudaGetLastError();
}

BLZ_API int blz_argmax_parts(const float* val, const int* idx, int tiles, int M, long long* out, float* out_val, int index_offset,
                             cudaStream_t s) {
  if (M <= 0 || tiles <= 0) return 0;
  return (int)launch_pdl(argmax_parts_kernel, dim3((M + 7) / 8), dim3(256), 0, s, val, idx, tiles, M, out, out_val, index_offset);
}
