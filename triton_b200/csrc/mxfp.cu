// MXFP4 quantiser / dequantiser for sm_100a: e2m1 values packed two per byte (element 2i in the low
// nibble) with one e8m0 scale byte per 32 elements along the quantised axis.
//
// Arithmetic (bit-exact with triton_kernels numerics_details/mxfp_details/_downcast_to_mxfp.py:33-147
// and _upcast_from_mxfp.py:8-53, 109-220):
//   m      = max |x| over the 32-group, in fp32
//   ds     = m / 6 (ROUND_UP) or m / 4 (ROUND_DOWN), IEEE round-to-nearest division
//   u      = (bits(ds) + 0x007FFFFF) & 0x7F800000  (ROUND_UP: next power of two)
//            bits(ds) & 0x7F800000                  (ROUND_DOWN)
//   scale  = u >> 23 ;  inv = (u == 0) ? 0 : 1 / float(u)
//   code   = RTNE_e2m1(x * inv), saturating at +-6
// Both kernels are HBM-bound: 16-byte loads/stores, one thread per 32-group on the contiguous path (one division and
// one scale per group, 16 bytes of codes per store).
#include "common.cuh"
#include <cuda_fp4.h>
#include <type_traits>

namespace {

__device__ __forceinline__ uint32_t scale_bits(float m, int mode) {
  if (mode == MOE_ROUND_UP) {
    float ds = __fdiv_rn(m, 6.0f);
    return (__float_as_uint(ds) + 0x007FFFFFu) & 0x7F800000u;
  }
  float ds = __fdiv_rn(m, 4.0f);
  return __float_as_uint(ds) & 0x7F800000u;
}

// 1 / u for u = 2^(e - 127) stored as e << 23: the exponent mirrored around the bias, exactly what an IEEE division
// returns.  e = 0 (group of zeros) gives 0 as in the reference; e <= 253 always holds because max|x| / 4 < 2^127.
__device__ __forceinline__ float inv_scale(uint32_t u) {
  return (u == 0u) ? 0.0f : __uint_as_float(0x7F000000u - u);
}

// Position of a grid-stride loop over [rows][chunks per row] without a division per iteration.
template <typename I> struct RowCursorT {
  I row, c, step_row, step_c, per_row;
  __device__ __forceinline__ RowCursorT(int64_t first, int64_t stride, int64_t chunks_per_row) {
    per_row = (I)chunks_per_row;
    row = (I)(first / chunks_per_row); c = (I)(first - (int64_t)row * chunks_per_row);
    step_row = (I)(stride / chunks_per_row); step_c = (I)(stride - (int64_t)step_row * chunks_per_row);
  }
  __device__ __forceinline__ void next() {
    row += step_row; c += step_c;
    if (c >= per_row) { c -= per_row; ++row; }
  }
};
using RowCursor = RowCursorT<int64_t>;

// two fp32 -> one byte: `lo` in bits 0..3, `hi` in bits 4..7 (round-to-nearest-even, saturating)
__device__ __forceinline__ uint32_t e2m1x2(float lo, float hi) {
  return (uint32_t)__nv_cvt_float2_to_fp4x2(make_float2(lo, hi), __NV_E2M1, cudaRoundNearest);
}

// ---- contiguous path: quant axis has unit stride, rows 16-byte aligned ------------------------------
// One thread owns whole 32-groups: 64 (or 128) contiguous input bytes as 16-byte loads, one division and one scale
// per group, one 16-byte store of the 32 codes and one byte of scale.  GROUPS_UNROLL groups are loaded before the first
// is converted, so that enough bytes are in flight per SM to cover the HBM latency.
constexpr int GROUPS_UNROLL = 2, DENSE_BLOCKS = 4;

template <typename T> __device__ __forceinline__ void unpack16(const uint4& r, float* v);
template <> __device__ __forceinline__ void unpack16<__nv_bfloat16>(const uint4& r, float* v) {
  const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    v[2 * j] = __uint_as_float(w[j] << 16);
    v[2 * j + 1] = __uint_as_float(w[j] & 0xFFFF0000u);
  }
}
template <> __device__ __forceinline__ void unpack16<__half>(const uint4& r, float* v) {
  const __half2* h = reinterpret_cast<const __half2*>(&r);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 f = __half22float2(h[j]);
    v[2 * j] = f.x;
    v[2 * j + 1] = f.y;
  }
}
template <> __device__ __forceinline__ void unpack16<float>(const uint4& r, float* v) {
  v[0] = __uint_as_float(r.x); v[1] = __uint_as_float(r.y); v[2] = __uint_as_float(r.z); v[3] = __uint_as_float(r.w);
}

// max |x| of a group; NaN operands lose, as with fmaxf.  Two-byte types by packed maxima of the pairs.
template <typename T> struct Two;
template <> struct Two<__nv_bfloat16> { using type = __nv_bfloat162; };
template <> struct Two<__half> { using type = __half2; };
template <typename T, int VPG> __device__ __forceinline__ float group_absmax(const uint4 (&raw)[VPG]) {
  if constexpr (sizeof(T) == 2) {
    using T2 = typename Two<T>::type;
    T2 m[4];
#pragma unroll
    for (int k = 0; k < VPG; ++k) {
      const uint32_t w[4] = {raw[k].x, raw[k].y, raw[k].z, raw[k].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const T2 v = __habs2(*reinterpret_cast<const T2*>(&w[j]));
        m[j] = k == 0 ? v : __hmax2(m[j], v);
      }
    }
    const T2 t = __hmax2(__hmax2(m[0], m[1]), __hmax2(m[2], m[3]));
    return fmaxf(fmaxf(0.0f, to_f32<T>(t.x)), to_f32<T>(t.y));
  } else {
    float m = 0.0f;
#pragma unroll
    for (int k = 0; k < VPG; ++k) {
      float v[32 / VPG];
      unpack16<T>(raw[k], v);
#pragma unroll
      for (int j = 0; j < 32 / VPG; ++j) m = fmaxf(m, fabsf(v[j]));
    }
    return m;
  }
}

// the 32 values of a group as VPG raw 16-byte vectors -> scale bits and 16 bytes of codes.  The vectors are unpacked
// twice (once for the maximum, once for the codes) instead of holding 32 floats across the division.
template <typename T, int VPG>
__device__ __forceinline__ uint4 quantise_raw(const uint4 (&raw)[VPG], int mode, uint32_t& sc) {
  constexpr int EPV = 32 / VPG;
  const float m = group_absmax<T, VPG>(raw);
  sc = scale_bits(m, mode);
  const float inv = inv_scale(sc);
  uint32_t w[4];
  if constexpr (EPV == 8) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float v[8];
      unpack16<T>(raw[k], v);
      const uint32_t b0 = e2m1x2(v[0] * inv, v[1] * inv), b1 = e2m1x2(v[2] * inv, v[3] * inv);
      const uint32_t b2 = e2m1x2(v[4] * inv, v[5] * inv), b3 = e2m1x2(v[6] * inv, v[7] * inv);
      w[k] = __byte_perm(b0 | (b1 << 8), b2 | (b3 << 8), 0x5410);
    }
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float v[8];
      unpack16<T>(raw[2 * k], v);
      unpack16<T>(raw[2 * k + 1], v + 4);
      const uint32_t b0 = e2m1x2(v[0] * inv, v[1] * inv), b1 = e2m1x2(v[2] * inv, v[3] * inv);
      const uint32_t b2 = e2m1x2(v[4] * inv, v[5] * inv), b3 = e2m1x2(v[6] * inv, v[7] * inv);
      w[k] = __byte_perm(b0 | (b1 << 8), b2 | (b3 << 8), 0x5410);
    }
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

template <typename T, typename I>
__global__ void __launch_bounds__(256, sizeof(T) == 2 ? 3 : 2) downcast_rows_kernel(const T* x, int64_t n_rows, int64_t quant,
                                                            int64_t outer, int64_t sx_batch, int64_t sx_outer,
                                                            uint8_t* q, uint8_t* scale,
                                                            int mode) {
  pdl_begin();
  constexpr int EPV = 16 / (int)sizeof(T);               // elements per 16-byte vector
  constexpr int VPG = 32 / EPV;                          // vectors per group
  const int64_t groups_per_row = quant >> 5;
  const int64_t total = n_rows * groups_per_row;
  const int64_t stride = (int64_t)gridDim.x * (GROUPS_UNROLL * 256);
  const int64_t tile0 = (int64_t)blockIdx.x * (GROUPS_UNROLL * 256);
  RowCursorT<I> cur[GROUPS_UNROLL] = {RowCursorT<I>(tile0 + threadIdx.x, stride, groups_per_row),
                                      RowCursorT<I>(tile0 + 256 + threadIdx.x, stride, groups_per_row)};
  const bool one_batch = outer == n_rows;
  for (int64_t tile = tile0; tile < total; tile += stride) {
    uint4 raw[GROUPS_UNROLL][VPG];
    bool live[GROUPS_UNROLL];
#pragma unroll
    for (int u = 0; u < GROUPS_UNROLL; ++u) {
      live[u] = tile + u * 256 + threadIdx.x < total;
      if (live[u]) {
        const int64_t row = cur[u].row, c = cur[u].c;
        int64_t b = 0, o = row;
        if (!one_batch) { b = row / outer; o = row - b * outer; }
        const uint4* src = reinterpret_cast<const uint4*>(x + b * sx_batch + o * sx_outer + c * 32);
#pragma unroll
        for (int k = 0; k < VPG; ++k) raw[u][k] = __ldcs(src + k);       // read once: L2 keeps the codes for their reader (8192 x 8192 and back 64.7 -> 62.1 us)
      }
    }
#pragma unroll
    for (int u = 0; u < GROUPS_UNROLL; ++u) {
      if (live[u]) {
        uint32_t sc;
        const uint4 codes = quantise_raw<T, VPG>(raw[u], mode, sc);
        const int64_t row = cur[u].row, c = cur[u].c;
        *reinterpret_cast<uint4*>(q + row * (quant >> 1) + c * 16) = codes;
        scale[row * groups_per_row + c] = (uint8_t)(sc >> 23);
      }
      cur[u].next();
    }
  }
}

// Rows that follow one another without a gap: groups are numbered through, so a thread has one index where the kernel above keeps a row and a chunk
// for each of its groups and multiplies three pitches: 64 registers, so a fourth block per SM.  8192 x 8192 bf16 to codes and back 62.1 -> 51.0 us with
// this kernel and upcast_dense_kernel (with three blocks per SM 51.1, with five and spills 53.5).
template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 2 ? DENSE_BLOCKS : 2) downcast_dense_kernel(const T* x, int64_t total, uint8_t* q, uint8_t* scale, int mode) {
  pdl_begin();
  constexpr int VPG = 2 * (int)sizeof(T);                // vectors per group
  const int64_t stride = (int64_t)gridDim.x * (GROUPS_UNROLL * 256);
  for (int64_t g0 = (int64_t)blockIdx.x * (GROUPS_UNROLL * 256) + threadIdx.x; g0 < total; g0 += stride) {
    uint4 raw[GROUPS_UNROLL][VPG];
#pragma unroll
    for (int u = 0; u < GROUPS_UNROLL; ++u)
      if (g0 + u * 256 < total) {
        const uint4* src = reinterpret_cast<const uint4*>(x + (g0 + u * 256) * 32);
#pragma unroll
        for (int k = 0; k < VPG; ++k) raw[u][k] = __ldcs(src + k);
      }
#pragma unroll
    for (int u = 0; u < GROUPS_UNROLL; ++u)
      if (g0 + u * 256 < total) {
        uint32_t sc;
        reinterpret_cast<uint4*>(q)[g0 + u * 256] = quantise_raw<T, VPG>(raw[u], mode, sc);
        scale[g0 + u * 256] = (uint8_t)(sc >> 23);
      }
  }
}

// ---- quantised axis strided, the other axis contiguous (expert weights quantised along K, axis 0 of a row-major matrix) --
// HBM-bound.  A block takes 64 columns x 8 groups (256 elements of the quantised axis): warp = group, lane = two
// neighbouring columns, so a warp load is 128 (bf16 / fp16) contiguous bytes and all 32 of a thread are in flight at once;
// the raw pairs stay packed in registers (two columns' maxima by one packed max) and are unpacked only for the conversion.
// Codes and scales meet in shared memory and leave as 128-byte runs of codes and 8-byte runs of scales per column:
// stored from registers they were lone 16-byte and single-byte writes at the pitch of an output row (16 x 2880 x 5760
// bf16, 671 MB moved: 221 us).
constexpr int CT_COLS = 64, CT_GROUPS = 8;
constexpr int CT_PITCH = CT_COLS * 16 + 16;          // bytes of one group's codes [column][16 B]; padded: a column's 8 groups on distinct banks

template <typename T> struct Pair { using Raw = uint32_t; };
template <> struct Pair<float> { using Raw = float2; };
template <typename T> __device__ __forceinline__ float2 unpack_pair(typename Pair<T>::Raw w);
template <> __device__ __forceinline__ float2 unpack_pair<__nv_bfloat16>(uint32_t w) {
  return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u));
}
template <> __device__ __forceinline__ float2 unpack_pair<__half>(uint32_t w) {
  return __half22float2(*reinterpret_cast<const __half2*>(&w));
}
template <> __device__ __forceinline__ float2 unpack_pair<float>(float2 w) { return w; }
// running |max| of both columns; NaN operands lose, as with fmaxf
template <typename T> __device__ __forceinline__ float2 pair_absmax(const typename Pair<T>::Raw (&raw)[32]);
template <> __device__ __forceinline__ float2 pair_absmax<__nv_bfloat16>(const uint32_t (&raw)[32]) {
  __nv_bfloat162 m = __float2bfloat162_rn(0.0f);
#pragma unroll
  for (int j = 0; j < 32; ++j) m = __hmax2(m, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&raw[j])));
  return make_float2(__low2float(m), __high2float(m));
}
template <> __device__ __forceinline__ float2 pair_absmax<__half>(const uint32_t (&raw)[32]) {
  __half2 m = __float2half2_rn(0.0f);
#pragma unroll
  for (int j = 0; j < 32; ++j) m = __hmax2(m, __habs2(*reinterpret_cast<const __half2*>(&raw[j])));
  return make_float2(__low2float(m), __high2float(m));
}
template <> __device__ __forceinline__ float2 pair_absmax<float>(const float2 (&raw)[32]) {
  float2 m = make_float2(0.0f, 0.0f);
#pragma unroll
  for (int j = 0; j < 32; ++j) m = make_float2(fmaxf(m.x, fabsf(raw[j].x)), fmaxf(m.y, fabsf(raw[j].y)));
  return m;
}

template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 2 ? 4 : 2) downcast_cols_kernel(
    const T* __restrict__ x, int64_t outer, int groups, int col_blocks, int group_blocks, int64_t sx_batch, int64_t sx_quant,
    uint8_t* __restrict__ q, uint8_t* __restrict__ scale, int mode) {
  using Raw = typename Pair<T>::Raw;
  __shared__ __align__(16) uint8_t s_q[CT_GROUPS * CT_PITCH];
  __shared__ uint8_t s_s[CT_COLS * CT_GROUPS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cb = (int)(blockIdx.x % (unsigned)col_blocks);
  const unsigned t = blockIdx.x / (unsigned)col_blocks;
  const int gb = (int)(t % (unsigned)group_blocks);
  const int64_t b = t / (unsigned)group_blocks;
  const int64_t c0 = (int64_t)cb * CT_COLS;
  const int g0 = gb * CT_GROUPS, g = g0 + warp;
  const int64_t col = c0 + lane * 2;
  if (g < groups && col < outer) {
    const T* src = x + b * sx_batch + (int64_t)g * 32 * sx_quant + col;
    Raw raw[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) raw[j] = __ldcs(reinterpret_cast<const Raw*>(src + j * sx_quant));
    const float2 m = pair_absmax<T>(raw);
    const uint32_t u0 = scale_bits(m.x, mode), u1 = scale_bits(m.y, mode);
    const float i0 = inv_scale(u0), i1 = inv_scale(u1);
    uint32_t w0[4], w1[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      uint32_t b0[4], b1[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const float2 v = unpack_pair<T>(raw[8 * k + 2 * h]), n = unpack_pair<T>(raw[8 * k + 2 * h + 1]);
        b0[h] = e2m1x2(v.x * i0, n.x * i0);
        b1[h] = e2m1x2(v.y * i1, n.y * i1);
      }
      w0[k] = __byte_perm(b0[0] | (b0[1] << 8), b0[2] | (b0[3] << 8), 0x5410);
      w1[k] = __byte_perm(b1[0] | (b1[1] << 8), b1[2] | (b1[3] << 8), 0x5410);
    }
    uint8_t* dst = s_q + warp * CT_PITCH + lane * 32;
    *reinterpret_cast<uint4*>(dst) = make_uint4(w0[0], w0[1], w0[2], w0[3]);
    *reinterpret_cast<uint4*>(dst + 16) = make_uint4(w1[0], w1[1], w1[2], w1[3]);
    s_s[lane * 16 + warp] = (uint8_t)(u0 >> 23);
    s_s[lane * 16 + 8 + warp] = (uint8_t)(u1 >> 23);
  }
  __syncthreads();
  const int64_t row_bytes = (int64_t)groups * 16;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int p = threadIdx.x + i * 256, c = p >> 3, gi = p & 7;
    if (c0 + c < outer && g0 + gi < groups) {
      const int64_t row = b * outer + c0 + c;
      *reinterpret_cast<uint4*>(q + row * row_bytes + (int64_t)(g0 + gi) * 16) = *reinterpret_cast<const uint4*>(s_q + gi * CT_PITCH + c * 16);
      scale[row * groups + g0 + gi] = s_s[c * 8 + gi];
    }
  }
}

// ---- strided path: any strides; consecutive threads walk the `outer` axis ---------------------------
template <typename T>
__global__ void __launch_bounds__(256) downcast_strided_kernel(const T* x, int64_t batch, int64_t outer,
                                                               int64_t quant, int64_t sx_batch, int64_t sx_outer,
                                                               int64_t sx_quant, uint8_t* q,
                                                               uint8_t* scale, int mode) {
  pdl_begin();
  const int64_t groups = quant >> 5;
  const int64_t total = batch * outer * groups;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const int64_t o = i % outer;
    const int64_t t = i / outer;
    const int64_t g = t % groups;
    const int64_t b = t / groups;
    const T* src = x + b * sx_batch + o * sx_outer + g * 32 * sx_quant;
    float v[32];
    float m = 0.0f;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      v[j] = to_f32<T>(src[j * sx_quant]);
      m = fmaxf(m, fabsf(v[j]));
    }
    const uint32_t u = scale_bits(m, mode);
    const float inv = inv_scale(u);
    uint32_t w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      uint32_t p = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) p |= e2m1x2(v[8 * k + 2 * j] * inv, v[8 * k + 2 * j + 1] * inv) << (8 * j);
      w[k] = p;
    }
    const int64_t row = b * outer + o;
    *reinterpret_cast<uint4*>(q + row * (quant >> 1) + g * 16) = make_uint4(w[0], w[1], w[2], w[3]);
    scale[row * groups + g] = (uint8_t)(u >> 23);
  }
}

__device__ __forceinline__ float e2m1_to_f32(uint32_t code) {
  // magnitude bits e1 e0 m: 0, .5, 1, 1.5, 2, 3, 4, 6
  const uint32_t mag = code & 7u;
  uint32_t bits = (mag == 0) ? 0u : (mag == 1) ? 0x3F000000u : (((mag >> 1) + 126u) << 23) | ((mag & 1u) << 22);
  return __uint_as_float(bits | ((code & 8u) << 28));
}

template <typename T> __device__ __forceinline__ float finite_max();
template <> __device__ __forceinline__ float finite_max<float>() { return 3.4028234663852886e+38f; }
template <> __device__ __forceinline__ float finite_max<__nv_bfloat16>() { return 3.3895313892515355e+38f; }
template <> __device__ __forceinline__ float finite_max<__half>() { return 65504.0f; }

template <typename T>
__device__ __forceinline__ T dequant_one(uint32_t code, float s, bool nan_scale) {
  float r = e2m1_to_f32(code) * s;
  const float mx = finite_max<T>();
  r = fminf(fmaxf(r, -mx), mx);
  if (nan_scale) r = __uint_as_float(0x7FC00000u);
  return from_f32<T>(r);
}

// bf16 fast path: the three magnitude bits of a code placed at bf16 bits 8:6 are value * 2^-126, and one
// bf16x2 multiply by 2^(sb - 1) gives value * 2^(sb - 127) exactly (every product is representable; sb = 0 multiplies
// by zero as the reference's scale bits 0 << 23 do).  Scale bytes from 253 up can overflow and take the general path.
__device__ __forceinline__ uint32_t bf16x2_mul_rn(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
// codes k and k + 4 of word w (nibble p holds element p) -> bf16x2 (low half: element k) of value * 2^-126
template <int K> __device__ __forceinline__ uint32_t e2m1_pair_k(uint32_t w) {
  const uint32_t mag = (K < 2 ? (w << (6 - 4 * K)) : (w >> (4 * K - 6))) & 0x01C001C0u;
  const uint32_t sgn = (w << (12 - 4 * K)) & 0x80008000u;
  return mag | sgn;
}
__device__ __forceinline__ uint4 upcast8_bf16(uint32_t w, uint32_t sb) {
  uint32_t c2, r[4];
  if (sb <= 128u) {
    c2 = (sb ? ((sb + 126u) << 7) : 0u) * 0x10001u;
    r[0] = bf16x2_mul_rn(e2m1_pair_k<0>(w), c2); r[1] = bf16x2_mul_rn(e2m1_pair_k<1>(w), c2);
    r[2] = bf16x2_mul_rn(e2m1_pair_k<2>(w), c2); r[3] = bf16x2_mul_rn(e2m1_pair_k<3>(w), c2);
  } else {                                           // 2^(sb - 1) is not a bf16: multiply by 2^126, then by 2^(sb - 127)
    const uint32_t k2 = 0x7E807E80u, s2 = (sb << 7) * 0x10001u;
    r[0] = bf16x2_mul_rn(bf16x2_mul_rn(e2m1_pair_k<0>(w), k2), s2); r[1] = bf16x2_mul_rn(bf16x2_mul_rn(e2m1_pair_k<1>(w), k2), s2);
    r[2] = bf16x2_mul_rn(bf16x2_mul_rn(e2m1_pair_k<2>(w), k2), s2); r[3] = bf16x2_mul_rn(bf16x2_mul_rn(e2m1_pair_k<3>(w), k2), s2);
  }
  // r[k] = (element k, element k + 4): back to element order
  return make_uint4(__byte_perm(r[0], r[1], 0x5410), __byte_perm(r[2], r[3], 0x5410), __byte_perm(r[0], r[1], 0x7632),
                    __byte_perm(r[2], r[3], 0x7632));
}

// Eight codes by table look-up: a byte permute takes four codes as its selectors, bits 0-2 the magnitude, and picks the low or high bytes of
// their values; bit 3 asks for the sign of a byte of ones instead.  Then a multiplication by the scale, exact where `looks_up` says so: products and
// scale are normal or subnormal numbers of the type and none has to be clamped.  (fp32 values are bf16 values and sixteen zero bits.)
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
  return d;
}
template <typename T> __device__ __forceinline__ bool looks_up(uint32_t sb);
template <> __device__ __forceinline__ bool looks_up<__nv_bfloat16>(uint32_t sb) { return sb < 253u; }
template <> __device__ __forceinline__ bool looks_up<float>(uint32_t sb) { return sb < 253u; }
template <> __device__ __forceinline__ bool looks_up<__half>(uint32_t sb) { return sb - 113u <= 140u - 113u; }      // 2^-14 .. 2^13
// values of the codes in bits 0-15 of w, two to a word (fp32: as bf16)
template <typename T> __device__ __forceinline__ void lookup4(uint32_t w, uint32_t& r0, uint32_t& r1) {
  const uint32_t mag = w & 0x7777u;
  const uint32_t sign = (prmt(0x80808080u, 0x80808080u, w) << 1) & 0x80808080u;      // 0xFF for a negative code, else 0x80
  if constexpr (std::is_same<T, __half>::value) {
    const uint32_t hi = prmt(0x3E3C3800u, 0x46444240u, mag) | sign;         // of 0, .5, 1, 1.5 and 2, 3, 4, 6; low bytes are zero
    r0 = prmt(hi, 0u, 0x1404u);
    r1 = prmt(hi, 0u, 0x3424u);
  } else {
    const uint32_t lo = prmt(0xC0800000u, 0xC0804000u, mag), hi = prmt(0x3F3F3F00u, 0x40404040u, mag) | sign;
    r0 = prmt(lo, hi, 0x5140u);
    r1 = prmt(lo, hi, 0x7362u);
  }
}
// eight elements, scaled
template <typename T> __device__ __forceinline__ void lookup8(uint32_t w, uint32_t sb, uint32_t (&r)[2 * sizeof(T)]) {
  uint32_t v[4];
  lookup4<T>(w, v[0], v[1]);
  lookup4<T>(w >> 16, v[2], v[3]);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if constexpr (std::is_same<T, __nv_bfloat16>::value) {
      r[i] = bf16x2_mul_rn(v[i], (sb << 7) * 0x10001u);
    } else if constexpr (std::is_same<T, __half>::value) {
      const uint32_t s2 = ((sb - 112u) << 10) * 0x10001u;
      const __half2 p = __hmul2(*reinterpret_cast<const __half2*>(&v[i]), *reinterpret_cast<const __half2*>(&s2));
      r[i] = *reinterpret_cast<const uint32_t*>(&p);
    } else {
      const float s = __uint_as_float(sb << 23);
      r[2 * i] = __float_as_uint(__uint_as_float(v[i] << 16) * s);
      r[2 * i + 1] = __float_as_uint(__uint_as_float(v[i] & 0xFFFF0000u) * s);
    }
  }
}

// Rows that follow one another without a gap: a thread 64 bytes, numbered through.  The kernel below issues 0.78 instructions a cycle and waits for the
// integer pipe (35 us for 8192 x 8192 bf16): two thirds of them are positions, shifts and masks.  us for 8192 x 8192 to codes and back, before and now:
// bf16 62.1 -> 51.0, fp16 92 -> 51.0, fp32 138 -> 110; 2048 x 2048 bf16 10.2 -> 5.8.  (With 32 bytes a thread bf16 52.4 and 7.3, with 128 fp32 122.)
constexpr int UP_DENSE_UNROLL = 2;
template <typename T>
__global__ void __launch_bounds__(256) upcast_dense_kernel(const uint8_t* q, const uint8_t* scale, T* out, int64_t total) {
  pdl_begin();
  constexpr int N = 64 / (int)sizeof(T), W = N / 8;      // elements of a thread, words of their codes
  using Codes = std::conditional_t<W == 4, uint4, uint2>;
  const int64_t stride = (int64_t)gridDim.x * (UP_DENSE_UNROLL * 256);
  for (int64_t i0 = (int64_t)blockIdx.x * (UP_DENSE_UNROLL * 256) + threadIdx.x; i0 < total; i0 += stride) {
    Codes w[UP_DENSE_UNROLL];
    uint32_t sb[UP_DENSE_UNROLL];
#pragma unroll
    for (int u = 0; u < UP_DENSE_UNROLL; ++u)
      if (i0 + u * 256 < total) {
        w[u] = reinterpret_cast<const Codes*>(q)[i0 + u * 256];
        sb[u] = scale[(i0 + u * 256) * N / 32];
      }
#pragma unroll
    for (int u = 0; u < UP_DENSE_UNROLL; ++u)
      if (i0 + u * 256 < total) {
        const uint32_t* word = reinterpret_cast<const uint32_t*>(&w[u]);
        T* dst = out + (i0 + u * 256) * N;
        auto store = [&](const uint4* v) {
          st_v8(dst, v[0], v[1]);
          st_v8(dst + N / 2, v[2], v[3]);
        };
        if (looks_up<T>(sb[u])) {
          uint32_t r[W][2 * sizeof(T)];
#pragma unroll
          for (int k = 0; k < W; ++k) lookup8<T>(word[k], sb[u], r[k]);
          store(reinterpret_cast<const uint4*>(r));
        } else {
          const float s = __uint_as_float(sb[u] << 23);
          alignas(16) T e[N];
#pragma unroll
          for (int k = 0; k < N; ++k) e[k] = dequant_one<T>((word[k / 8] >> (4 * (k % 8))) & 0xFu, s, sb[u] == 0xFFu);
          store(reinterpret_cast<const uint4*>(e));
        }
      }
  }
}

// HBM-bound, four fifths of it writes: with 16-byte stores (a sector in two) 8192 x 8192 to bf16 took 45.3 us on cold inputs, with
// a sector per lane 35.6 (4.8 TB/s over 169.9 MB).
constexpr int ROWS_UNROLL = 4;
// contiguous output: thread owns U units of 8 elements (4 input bytes each) of each of ROWS_UNROLL chunks per iteration; a
// chunk of two units of a 2-byte type, or of one of fp32, leaves as one 32-byte store (WIDE)
template <typename T, bool WIDE>
__global__ void __launch_bounds__(256) upcast_rows_kernel(const uint8_t* q,
                                                          const uint8_t* scale, T* out,
                                                          int64_t n_rows, int64_t quant, int64_t outer,
                                                          int64_t so_batch, int64_t so_outer) {
  pdl_begin();
  constexpr int U = WIDE && sizeof(T) == 2 ? 2 : 1;
  const int64_t chunks_per_row = quant / (8 * U);
  const int64_t total = n_rows * chunks_per_row;
  const int64_t stride = (int64_t)gridDim.x * (ROWS_UNROLL * 256);
  const int64_t tile0 = (int64_t)blockIdx.x * (ROWS_UNROLL * 256);
  RowCursor cur[ROWS_UNROLL] = {RowCursor(tile0 + threadIdx.x, stride, chunks_per_row),
                                RowCursor(tile0 + 256 + threadIdx.x, stride, chunks_per_row),
                                RowCursor(tile0 + 512 + threadIdx.x, stride, chunks_per_row),
                                RowCursor(tile0 + 768 + threadIdx.x, stride, chunks_per_row)};
  const bool one_batch = outer == n_rows;
  for (int64_t tile = tile0; tile < total; tile += stride) {
    uint32_t w[ROWS_UNROLL][U], sb[ROWS_UNROLL];
#pragma unroll
    for (int u = 0; u < ROWS_UNROLL; ++u) {
      const bool live = tile + u * 256 + threadIdx.x < total;
      const int64_t row = live ? cur[u].row : 0, c = live ? cur[u].c : 0;
      const uint8_t* src = q + row * (quant >> 1) + c * (4 * U);
      if constexpr (U == 2) {
        const uint2 two = *reinterpret_cast<const uint2*>(src);
        w[u][0] = two.x; w[u][1] = two.y;
      } else {
        w[u][0] = *reinterpret_cast<const uint32_t*>(src);
      }
      sb[u] = scale[row * (quant >> 5) + c * U / 4];
    }
#pragma unroll
    for (int u = 0; u < ROWS_UNROLL; ++u) {
      const bool live = tile + u * 256 + threadIdx.x < total;
      const int64_t row = cur[u].row, c = cur[u].c;
      cur[u].next();
      if (!live) continue;
      int64_t b = 0, o = row;
      if (!one_batch) { b = row / outer; o = row - b * outer; }
      T* dst = out + b * so_batch + o * so_outer + c * (8 * U);
      uint4 v[U * 8 * sizeof(T) / 16];
      bool done = false;
      if constexpr (std::is_same<T, __nv_bfloat16>::value) {
        if (sb[u] < 253u) {
#pragma unroll
          for (int i = 0; i < U; ++i) v[i] = upcast8_bf16(w[u][i], sb[u]);
          done = true;
        }
      }
      if (!done) {
        const float s = __uint_as_float(sb[u] << 23);
        const bool nan_scale = sb[u] == 0xFFu;
        alignas(16) T e[8 * U];
#pragma unroll
        for (int j = 0; j < 8 * U; ++j) e[j] = dequant_one<T>((w[u][j / 8] >> (4 * (j % 8))) & 0xFu, s, nan_scale);
#pragma unroll
        for (int i = 0; i < (int)(sizeof(v) / 16); ++i) v[i] = reinterpret_cast<const uint4*>(e)[i];
      }
      if constexpr (WIDE) {
        st_v8(dst, v[0], v[1]);
      } else {
#pragma unroll
        for (int i = 0; i < (int)(sizeof(v) / 16); ++i) reinterpret_cast<uint4*>(dst)[i] = v[i];
      }
    }
  }
}

// The inverse of downcast_cols_kernel: output contiguous along the other axis.  A block reads 64 columns x 8 groups of codes
// (128-byte runs) through shared memory; warp = group, lane = two neighbouring columns, every store of a warp is 128
// contiguous bytes (fp32: 256).  A thread per column and group stored 64-byte runs from loads at the pitch of a row.
template <typename T>
__global__ void __launch_bounds__(256) upcast_cols_kernel(const uint8_t* q, const uint8_t* scale,
                                                          T* out, int64_t outer, int groups, int col_blocks,
                                                          int group_blocks, int64_t so_batch, int64_t so_quant) {
  pdl_begin();
  __shared__ __align__(16) uint8_t s_q[CT_GROUPS * CT_PITCH];
  __shared__ uint8_t s_s[CT_COLS * CT_GROUPS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cb = (int)(blockIdx.x % (unsigned)col_blocks);
  const unsigned t = blockIdx.x / (unsigned)col_blocks;
  const int gb = (int)(t % (unsigned)group_blocks);
  const int64_t b = t / (unsigned)group_blocks;
  const int64_t c0 = (int64_t)cb * CT_COLS;
  const int g0 = gb * CT_GROUPS, g = g0 + warp;
  const int64_t row_bytes = (int64_t)groups * 16;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int p = threadIdx.x + i * 256, c = p >> 3, gi = p & 7;
    if (c0 + c < outer && g0 + gi < groups) {
      const int64_t row = b * outer + c0 + c;
      *reinterpret_cast<uint4*>(s_q + gi * CT_PITCH + c * 16) = *reinterpret_cast<const uint4*>(q + row * row_bytes + (int64_t)(g0 + gi) * 16);
      s_s[c * 8 + gi] = scale[row * groups + g0 + gi];
    }
  }
  __syncthreads();
  const int64_t col = c0 + lane * 2;
  if (g >= groups || col >= outer) return;
  const uint4 a0 = *reinterpret_cast<const uint4*>(s_q + warp * CT_PITCH + lane * 32);
  const uint4 a1 = *reinterpret_cast<const uint4*>(s_q + warp * CT_PITCH + lane * 32 + 16);
  const uint32_t sb0 = s_s[lane * 16 + warp], sb1 = s_s[lane * 16 + 8 + warp];
  const uint32_t w0[4] = {a0.x, a0.y, a0.z, a0.w}, w1[4] = {a1.x, a1.y, a1.z, a1.w};
  T* dst = out + b * so_batch + (int64_t)g * 32 * so_quant + col;
  if (looks_up<T>(sb0) && looks_up<T>(sb1)) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      uint32_t p0[2 * sizeof(T)], p1[2 * sizeof(T)];               // eight elements of either column
      lookup8<T>(w0[k], sb0, p0);
      lookup8<T>(w1[k], sb1, p1);
#pragma unroll
      for (int h = 0; h < 8; ++h) {
        T* at = dst + (8 * k + h) * so_quant;
        if constexpr (sizeof(T) == 2) *reinterpret_cast<uint32_t*>(at) = __byte_perm(p0[h >> 1], p1[h >> 1], h & 1 ? 0x7632 : 0x5410);
        else *reinterpret_cast<uint2*>(at) = make_uint2(p0[h], p1[h]);
      }
    }
    return;
  }
  const float f0 = __uint_as_float(sb0 << 23), f1 = __uint_as_float(sb1 << 23);
  const bool n0 = sb0 == 0xFFu, n1 = sb1 == 0xFFu;
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    T e[2] = {dequant_one<T>((w0[j >> 3] >> (4 * (j & 7))) & 0xFu, f0, n0), dequant_one<T>((w1[j >> 3] >> (4 * (j & 7))) & 0xFu, f1, n1)};
    *reinterpret_cast<typename Pair<T>::Raw*>(dst + j * so_quant) = *reinterpret_cast<const typename Pair<T>::Raw*>(e);
  }
}

template <typename T>
__global__ void __launch_bounds__(256) upcast_strided_kernel(const uint8_t* q,
                                                             const uint8_t* scale, T* out,
                                                             int64_t batch, int64_t outer, int64_t quant,
                                                             int64_t so_batch, int64_t so_outer, int64_t so_quant) {
  pdl_begin();
  const int64_t groups = quant >> 5;
  const int64_t total = batch * outer * groups;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const int64_t o = i % outer;
    const int64_t t = i / outer;
    const int64_t g = t % groups;
    const int64_t b = t / groups;
    const int64_t row = b * outer + o;
    const uint4 raw = *reinterpret_cast<const uint4*>(q + row * (quant >> 1) + g * 16);
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
    const uint32_t sb = scale[row * groups + g];
    const float s = __uint_as_float(sb << 23);
    const bool nan_scale = sb == 0xFFu;
    T* dst = out + b * so_batch + o * so_outer + g * 32 * so_quant;
#pragma unroll
    for (int j = 0; j < 32; ++j) dst[j * so_quant] = dequant_one<T>((w[j >> 3] >> (4 * (j & 7))) & 0xFu, s, nan_scale);
  }
}

int64_t col_tiles(int64_t batch, int64_t outer, int64_t quant) {       // blocks of the column kernels
  return batch * cdiv64(outer, CT_COLS) * cdiv64(quant >> 5, CT_GROUPS);
}

int grid_for(int64_t total, int threads) {
  int64_t blocks = cdiv64(total, threads);
  int64_t cap = (int64_t)moe_sm_count() * 16;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  return (int)blocks;
}

}  // namespace

extern "C" __attribute__((visibility("default"))) int moe_downcast_mxfp4(const void* x, int src_dtype, int64_t batch, int64_t outer, int64_t quant,
                                  int64_t sx_batch, int64_t sx_outer, int64_t sx_quant, uint8_t* q, uint8_t* scale,
                                  int rounding_mode, void* stream) {
  MOE_CHECK_ARG(batch >= 0 && outer >= 0 && quant >= 0, "moe_downcast_mxfp4: negative extent");
  MOE_CHECK_ARG(quant % 32 == 0, "moe_downcast_mxfp4: quantised axis (%lld) must be a multiple of 32", (long long)quant);
  MOE_CHECK_ARG(rounding_mode == MOE_ROUND_UP || rounding_mode == MOE_ROUND_DOWN, "moe_downcast_mxfp4: bad rounding mode");
  if (batch * outer * quant == 0) return MOE_OK;
  MOE_CHECK_ARG(x && q && scale, "moe_downcast_mxfp4: NULL pointer");
  cudaStream_t st = (cudaStream_t)stream;
  MOE_DISPATCH_FLOAT(src_dtype, T, {
    const int64_t align = 16 / (int64_t)sizeof(T);
    const bool rows_ok = sx_quant == 1 && ((uintptr_t)x % 16 == 0) && (sx_outer % align == 0) &&
                         (sx_batch % align == 0) && ((uintptr_t)q % 4 == 0);
    // two columns per thread: 4- or 8-byte loads
    const bool cols_ok = sx_outer == 1 && sx_quant != 1 && outer % 2 == 0 && ((uintptr_t)x % (2 * sizeof(T)) == 0) &&
                         (sx_quant % 2 == 0) && (sx_batch % 2 == 0) && ((uintptr_t)q % 16 == 0) &&
                         col_tiles(batch, outer, quant) < 2147483647LL;
    if (rows_ok && (uintptr_t)q % 16 == 0 && sx_outer == quant && (batch == 1 || sx_batch == outer * quant)) {
      const int64_t total = batch * outer * (quant >> 5);
      MOE_CHECK_CUDA(launch_pdl(downcast_dense_kernel<T>, dim3(grid_for(total, GROUPS_UNROLL * 256)), dim3(256), 0, st, (const T*)x, total, q, scale,
                                rounding_mode));
    } else if (rows_ok && (uintptr_t)q % 16 == 0) {
      const int64_t total = batch * outer * (quant >> 5);
      if (total + (int64_t)GROUPS_UNROLL * 256 * moe_sm_count() * 16 < 2147483647LL)       // 32-bit row / group counters
        MOE_CHECK_CUDA(launch_pdl(downcast_rows_kernel<T, int32_t>, dim3(grid_for(total, GROUPS_UNROLL * 256)), dim3(256), 0, st,
                                  (const T*)x, batch * outer, quant, outer, sx_batch, sx_outer, q, scale, rounding_mode));
      else
        MOE_CHECK_CUDA(launch_pdl(downcast_rows_kernel<T, int64_t>, dim3(grid_for(total, GROUPS_UNROLL * 256)), dim3(256), 0, st,
                                  (const T*)x, batch * outer, quant, outer, sx_batch, sx_outer, q, scale, rounding_mode));
    } else if (cols_ok) {
      const int groups = (int)(quant >> 5);
      downcast_cols_kernel<T><<<(unsigned)col_tiles(batch, outer, quant), 256, 0, st>>>(
          (const T*)x, outer, groups, (int)cdiv64(outer, CT_COLS), (int)cdiv64(groups, CT_GROUPS), sx_batch, sx_quant, q, scale,
          rounding_mode);
    } else {
      MOE_CHECK_ARG((uintptr_t)q % 16 == 0, "moe_downcast_mxfp4: q must be 16-byte aligned");
      const int64_t total = batch * outer * (quant >> 5);
      MOE_CHECK_CUDA(launch_pdl(downcast_strided_kernel<T>, dim3(grid_for(total, 256)), dim3(256), 0, st, (const T*)x, batch, outer,
                                quant, sx_batch, sx_outer, sx_quant, q, scale, rounding_mode));
    }
  });
  MOE_CHECK_LAUNCH();
  return MOE_OK;
}

extern "C" __attribute__((visibility("default"))) int moe_upcast_mxfp4(const uint8_t* q, const uint8_t* scale, void* out, int dst_dtype, int64_t batch,
                                int64_t outer, int64_t quant, int64_t so_batch, int64_t so_outer, int64_t so_quant,
                                void* stream) {
  MOE_CHECK_ARG(batch >= 0 && outer >= 0 && quant >= 0, "moe_upcast_mxfp4: negative extent");
  MOE_CHECK_ARG(quant % 32 == 0, "moe_upcast_mxfp4: quantised axis (%lld) must be a multiple of 32", (long long)quant);
  if (batch * outer * quant == 0) return MOE_OK;
  MOE_CHECK_ARG(q && scale && out, "moe_upcast_mxfp4: NULL pointer");
  cudaStream_t st = (cudaStream_t)stream;
  MOE_DISPATCH_FLOAT(dst_dtype, T, {
    const int64_t align = 16 / (int64_t)sizeof(T);
    const bool rows_ok = so_quant == 1 && ((uintptr_t)out % 16 == 0) && (so_outer % align == 0) &&
                         (so_batch % align == 0) && ((uintptr_t)q % 4 == 0);
    const bool wide = rows_ok && (uintptr_t)out % 32 == 0 && so_outer % (2 * align) == 0 && so_batch % (2 * align) == 0 &&
                      (uintptr_t)q % 8 == 0;
    if (wide && (uintptr_t)q % 16 == 0 && so_outer == quant && (batch == 1 || so_batch == outer * quant)) {
      const int64_t total = batch * outer * (quant * (int64_t)sizeof(T) >> 6);
      MOE_CHECK_CUDA(launch_pdl(upcast_dense_kernel<T>, dim3(grid_for(total, UP_DENSE_UNROLL * 256)), dim3(256), 0, st, q, scale, (T*)out, total));
    } else if (wide) {
      const int64_t total = batch * outer * (quant * (int64_t)sizeof(T) >> 5);
      MOE_CHECK_CUDA(launch_pdl(upcast_rows_kernel<T, true>, dim3(grid_for(total, ROWS_UNROLL * 256)), dim3(256), 0, st, q, scale,
                                (T*)out, batch * outer, quant, outer, so_batch, so_outer));
    } else if (rows_ok) {
      const int64_t total = batch * outer * (quant >> 3);
      MOE_CHECK_CUDA(launch_pdl(upcast_rows_kernel<T, false>, dim3(grid_for(total, ROWS_UNROLL * 256)), dim3(256), 0, st, q, scale,
                                (T*)out, batch * outer, quant, outer, so_batch, so_outer));
    } else if (so_outer == 1 && so_quant % 2 == 0 && so_batch % 2 == 0 && outer % 2 == 0 && (uintptr_t)q % 16 == 0 &&
               (uintptr_t)out % (2 * sizeof(T)) == 0 && col_tiles(batch, outer, quant) < 2147483647LL) {
      const int groups = (int)(quant >> 5);
      MOE_CHECK_CUDA(launch_pdl(upcast_cols_kernel<T>, dim3((unsigned)col_tiles(batch, outer, quant)), dim3(256), 0, st, q, scale,
                                (T*)out, outer, groups, (int)cdiv64(outer, CT_COLS), (int)cdiv64(groups, CT_GROUPS), so_batch, so_quant));
    } else {
      MOE_CHECK_ARG((uintptr_t)q % 16 == 0, "moe_upcast_mxfp4: q must be 16-byte aligned");
      const int64_t total = batch * outer * (quant >> 5);
      MOE_CHECK_CUDA(launch_pdl(upcast_strided_kernel<T>, dim3(grid_for(total, 256)), dim3(256), 0, st, q, scale, (T*)out, batch, outer,
                                quant, so_batch, so_outer, so_quant));
    }
  });
  MOE_CHECK_LAUNCH();
  return MOE_OK;
}
