// Pieces shared by the block-scaled GEMM kernels: e4m3 conversions and their e8m0 scales, the weight tensor map.
#pragma once
#include "gemm_tc_common.cuh"
#include <cuda_fp4.h>
#include <cuda_fp8.h>

// e4m3 output (the next GEMM's activations): round to nearest, saturating at +-448 like the MMA's own conversions
template <> __device__ __forceinline__ __nv_fp8_e4m3 from_f32<__nv_fp8_e4m3>(float v) {
  __nv_fp8_e4m3 r;
  r.__x = __nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3);
  return r;
}

namespace {

__device__ __forceinline__ uint32_t f32x2_to_e4m3x2(float lo, float hi) {       // low byte <- lo, high byte <- hi
  uint16_t r;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ float2 e4m3x2_to_f32x2(uint32_t v) {
  uint32_t h2;
  asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h2) : "h"((uint16_t)v));
  return __half22float2(*reinterpret_cast<__half2*>(&h2));
}
__device__ __forceinline__ float2 e2m1x2_to_f32x2(uint32_t c) {
  const __half2_raw h = __nv_cvt_fp4x2_to_halfraw2((__nv_fp4x2_storage_t)c, __NV_E2M1);
  return __half22float2(__half2(h));
}
// e8m0 byte s with 2^(s-127) >= amax / 448 (smallest such power of two), and the exact factors 2^(s-127), 2^(127-s)
__device__ __forceinline__ void mx8_scale(float amax, uint32_t& sb, float& scale, float& inv) {
  const float ds = amax * (1.0f / 448.0f);
  uint32_t u = (__float_as_uint(ds) + 0x007FFFFFu) & 0x7F800000u;
  sb = u >> 23;
  if (amax == 0.0f) sb = 127u;
  sb = min(max(sb, 1u), 253u);
  scale = __uint_as_float(sb << 23);
  inv = __uint_as_float((254u - sb) << 23);
}

__device__ __forceinline__ uint32_t f32x2_to_e2m1x2(float lo, float hi) {       // `lo` in bits 0..3
  return (uint32_t)__nv_cvt_float2_to_fp4x2(make_float2(lo, hi), __NV_E2M1, cudaRoundNearest);
}
// e8m0 byte s with 2^(s-127) >= amax / 6, and the exact factors 2^(s-127), 2^(127-s)
__device__ __forceinline__ void mx4_scale(float amax, uint32_t& sb, float& scale, float& inv) {
  // amax / 6 rounded UP to a power of two; the product with a constant just above 1/6 is never below the quotient, so
  // every value of the group still fits (it doubles the scale where amax is within an ulp of 6 * 2^e, which costs nothing
  // that matters here) and the division is off the chain
  const float ds = amax * 0.16666668f;
  uint32_t u = (__float_as_uint(ds) + 0x007FFFFFu) & 0x7F800000u;
  sb = u >> 23;
  if (amax == 0.0f) sb = 127u;
  sb = min(max(sb, 1u), 253u);
  scale = __uint_as_float(sb << 23);
  inv = __uint_as_float((254u - sb) << 23);
}
// What a term leaves of a value, in one rounding.  A product by itself is past the largest number where the group's maximum is near it (2.98e38), and
// left to the compiler some of a lane's values got one and others not.
__device__ __forceinline__ float left_over(float v, float code, float scale) { return fmaf(-code, scale, v); }
// Term t of N values of a 32-group (v: what the terms before left over, and leaves); its maximum comes from `all`.  -> scale byte
// A value that is not finite has its code in the first term and leaves nothing, so that the others keep the rest of their terms.
template <int N, typename F>
__device__ __forceinline__ uint32_t e2m1_term(int t, float (&v)[N], const bool (&nan)[N], uint32_t& codes, F all) {
  // (first term: NaN ranks above Inf where four neighbouring values are NaN, and is caught below)
  uint32_t top = 0;
#pragma unroll
  for (int i = 0; i < N; i += 4)
    top = max(top, __float_as_uint(fmaxf(fmaxf(fabsf(v[i]), fabsf(v[i + 1])), fmaxf(fabsf(v[i + 2]), fabsf(v[i + 3])))));
  float amax = __uint_as_float(all(top));
  if (t == 0 && !(amax < 3.0e38f)) amax = 3.0e38f;                 // Inf / NaN in the group: keep the scale finite
  uint32_t sb; float s, inv;
  mx4_scale(amax, sb, s, inv);
  codes = 0;
#pragma unroll
  for (int i = 0; i < N; i += 2) {
    const uint32_t c = f32x2_to_e2m1x2(nan[i] ? 0.0f : v[i] * inv, nan[i + 1] ? 0.0f : v[i + 1] * inv);
    codes |= c << (4 * i);
    const float2 f = e2m1x2_to_f32x2(c);
    v[i] = left_over(v[i], f.x, s);
    v[i + 1] = left_over(v[i + 1], f.y, s);
    if (t == 0) {
      if (!(fabsf(v[i]) < INFINITY)) v[i] = 0.0f;
      if (!(fabsf(v[i + 1]) < INFINITY)) v[i + 1] = 0.0f;
    }
  }
  return sb;
}

// cuTensorMapEncodeTiled with the defaults of these kernels
inline int encode_map(CUtensorMap* map, CUtensorMapDataType type, int rank, const void* base, const cuuint64_t* dims, const cuuint64_t* strides,
                      const cuuint32_t* box, CUtensorMapSwizzle swizzle, const char* what) {
  static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
  static std::mutex mu;
  {
    std::lock_guard<std::mutex> lk(mu);
    if (!encode) {
      void* fn = nullptr;
      cudaDriverEntryPointQueryResult qr;
      MOE_CHECK_CUDA(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &qr));
      if (qr != cudaDriverEntryPointSuccess || !fn) {
        moe_set_error("moe_grouped_gemm: the driver does not provide cuTensorMapEncodeTiled");
        return MOE_ERR_UNSUPPORTED;
      }
      encode = (PFN_cuTensorMapEncodeTiled_v12000)fn;
    }
  }
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  const CUresult r = encode(map, type, rank, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    moe_set_error("moe_grouped_gemm: cuTensorMapEncodeTiled (%s) failed with code %d", what, (int)r);
    return MOE_ERR_CUDA;
  }
  return MOE_OK;
}

// Tensor map over the value tiles of the block-scaled layout, boxes of n_blocks tiles.  [tile][128 rows][128 e2m1 = 64 bytes];
// `packed`: the 64-byte rows as they are, 64-byte swizzle; else the TMA unit writes 16 elements per 16 bytes of shared memory
// (128-byte rows, 128-byte swizzle), the operand form of kind::mxf8f6f4.
inline int make_w_map(const MoeGemmArgs& a, int KT, int NB, bool packed, int n_blocks, CUtensorMap* map) {
  const cuuint64_t inner = packed ? 64 : 128;
  const cuuint64_t dims[3] = {inner, 128, (cuuint64_t)a.E * (cuuint64_t)KT * (cuuint64_t)NB};
  const cuuint64_t strides[2] = {64, 64 * 128};
  const cuuint32_t box[3] = {(cuuint32_t)inner, 128, (cuuint32_t)n_blocks};
  return encode_map(map, packed ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_16U4_ALIGN16B, 3, a.w, dims, strides, box,
                    packed ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B, "packed e2m1 weights");
}

// ---- copies issued by a warp that runs its loop as a whole: the instruction is guarded by an election next to it and its operands
// live in uniform registers (issued by a single thread of a divergent branch, a copy cost about 150 cycles)
__device__ __forceinline__ void elect_bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\telect.sync _|q, 0xFFFFFFFF;\n\t"
      "@q cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n\t}" ::"r"(dst),
      "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void elect_tile_3d(uint32_t dst, const CUtensorMap* tmap, int x, int y, int z, uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\telect.sync _|q, 0xFFFFFFFF;\n\t"
      "@q cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n\t}" ::"r"(dst),
      "l"(tmap), "r"(x), "r"(y), "r"(z), "r"(bar)
      : "memory");
}
// the same with a cache policy
__device__ __forceinline__ void elect_tile_3d_hint(uint32_t dst, const CUtensorMap* tmap, int x, int y, int z, uint32_t bar, uint64_t policy) {
  asm volatile(
      "{\n\t.reg .pred q;\n\telect.sync _|q, 0xFFFFFFFF;\n\t"
      "@q cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3, %4}], [%5], %6;\n\t}" ::"r"(dst),
      "l"(tmap), "r"(x), "r"(y), "r"(z), "r"(bar), "l"(policy)
      : "memory");
}
__device__ __forceinline__ void elect_bulk_g2s_hint(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar, uint64_t policy) {
  asm volatile(
      "{\n\t.reg .pred q;\n\telect.sync _|q, 0xFFFFFFFF;\n\t"
      "@q cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;\n\t}" ::"r"(dst),
      "l"(src), "r"(bytes), "r"(bar), "l"(policy)
      : "memory");
}
__device__ __forceinline__ void elect_tile_4d_hint(uint32_t dst, const CUtensorMap* tmap, int x, int y, int z, int w, uint32_t bar, uint64_t policy) {
  asm volatile(
      "{\n\t.reg .pred q;\n\telect.sync _|q, 0xFFFFFFFF;\n\t"
      "@q cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3, %4, %5}], [%6], %7;\n\t}" ::"r"(dst),
      "l"(tmap), "r"(x), "r"(y), "r"(z), "r"(w), "r"(bar), "l"(policy)
      : "memory");
}

__device__ __forceinline__ void elect_tile_4d(uint32_t dst, const CUtensorMap* tmap, int x, int y, int z, int w, uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\telect.sync _|q, 0xFFFFFFFF;\n\t"
      "@q cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];\n\t}" ::"r"(dst),
      "l"(tmap), "r"(x), "r"(y), "r"(z), "r"(w), "r"(bar)
      : "memory");
}

}  // namespace
