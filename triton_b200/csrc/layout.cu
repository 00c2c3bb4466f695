// One-time re-layout of canonical MXFP4 weights into the tile-contiguous form the tcgen05 kernel streams.
//
// Canonical (what moe_downcast_mxfp4 writes for w[E,K,N] quantised along K): values [E][N][K/2] bytes,
// byte b of a row holding k = 2b (low nibble) and 2b+1 (high nibble); scales [E][N][K/32] (any strides).
// Tiled: tiles of 128 n x 128 k ordered [E][n_tile][k_tile].
//   value tile: 8 KB = [4 scale groups][128 rows][16 bytes]: the 16 bytes of (group g, row r) are the 32 k values
//               k = 32g .. 32g+31 of that row, so that 8 consecutive lanes reading 8 consecutive rows of one
//               group touch 128 contiguous bytes.  Inside, 32-bit word q covers k = 32g + 8q .. +7 with nibble p
//               holding k + {0,2,4,6,1,3,5,7}[p], so that (word >> 4i) & 0x000F000F yields the pair (2i, 2i+1) in
//               the low and high half-word.
//   scale tile: 128 rows x 4 bytes (the four 32-groups of the k tile).
// Out-of-range n or k is zero (value 0, scale byte 0).
#include "common.cuh"

namespace {

constexpr int TN = 128, TK = 128;

__device__ __forceinline__ uint32_t nibble_interleave(uint32_t w) {   // natural -> (evens | odds << 16)
  uint32_t ev = w & 0x0F0F0F0Fu, od = (w >> 4) & 0x0F0F0F0Fu;          // k = 2a and k = 2a + 1 in byte a
  ev = (ev | (ev >> 4)) & 0x00FF00FFu;
  od = (od | (od >> 4)) & 0x00FF00FFu;
  return ((ev | (ev >> 8)) & 0xFFFFu) | ((od | (od >> 8)) << 16);
}
__device__ __forceinline__ uint32_t nibble_deinterleave(uint32_t r) {
  uint32_t w = 0;
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    w |= ((r >> (4 * a)) & 0xFu) << (8 * a);
    w |= ((r >> (16 + 4 * a)) & 0xFu) << (8 * a + 4);
  }
  return w;
}

// 16 bytes (the 32 k of one scale group) of a source row; VEC: rows are 16-byte aligned
template <bool VEC> __device__ __forceinline__ uint4 load_group(const uint8_t* src) {
  if constexpr (VEC) {
    return *reinterpret_cast<const uint4*>(src);
  } else {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      w[i] = (uint32_t)src[4 * i] | ((uint32_t)src[4 * i + 1] << 8) | ((uint32_t)src[4 * i + 2] << 16) | ((uint32_t)src[4 * i + 3] << 24);
    return make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// Value tiles of both layouts.  HBM-bound copy: a block takes a tile, a thread two of its 512 16-byte pieces (row, scale
// group), four neighbouring lanes the 64 bytes of a row.  SCALED: the block-scaled layout (tiles [E][k_tile][n_block],
// rows of 64 bytes as they are), else [E][n_tile][k_tile] with the [group][row] order and interleaved nibbles described above.
template <bool SCALED, bool VEC>
__global__ void __launch_bounds__(256) to_tiles_values(const uint8_t* __restrict__ q, int64_t q_stride_e, int64_t q_stride_n,
                                                       int E, int K, int N, int NT, int KT, uint4* __restrict__ out) {
  const int64_t tiles = (int64_t)E * NT * KT;
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int kt = SCALED ? (int)(tile / NT % KT) : (int)(tile % KT);
    const int nt = SCALED ? (int)(tile % NT) : (int)(tile / KT % NT);
    const int64_t e = tile / ((int64_t)NT * KT);
    uint4* dst = out + tile * (TN * 4);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int p = threadIdx.x + i * 256, r = p >> 2, g = p & 3;
      const int n = nt * TN + r, k = kt * TK + g * 32;             // K is a multiple of 32: a group is in or out as a whole
      uint4 v = make_uint4(0, 0, 0, 0);
      if (n < N && k < K) v = load_group<VEC>(q + e * q_stride_e + (int64_t)n * q_stride_n + (k >> 1));
      if constexpr (SCALED)
        dst[p] = v;
      else
        dst[g * TN + r] = make_uint4(nibble_interleave(v.x), nibble_interleave(v.y), nibble_interleave(v.z), nibble_interleave(v.w));
    }
  }
}

// Scales stored K-innermost and dense ([E][N][K / 32], what the quantiser returns along K), either layout: a block takes the rows of
// one weight block, contiguous in memory, through shared memory and writes their tiles of all k steps.  A word per thread read four
// lone bytes at the pitch of a row (16 x 2880 x 5760: 15.5 us, so 8.5).  MX: the block-scaled order [E][k step][block].
constexpr int SCALE_ROWS_SMEM = 48 * 1024;
template <bool MX>
__global__ void __launch_bounds__(256) scales_from_rows(const uint8_t* __restrict__ s, int64_t s_stride_e, int groups, int N, int NB, int KT,
                                                        uint32_t* __restrict__ out) {
  extern __shared__ __align__(16) uint32_t s_words[];              // [rows][groups] bytes
  const int nb = blockIdx.x % NB, e = blockIdx.x / NB, rows = min(TN, N - nb * TN);
  const uint8_t* src = s + (int64_t)e * s_stride_e + (int64_t)nb * TN * groups;       // 4-byte aligned: TN is a multiple of 4
  const int bytes = rows * groups;
  int done = 0;                                      // words copied, 16 bytes at a time where they start on such a boundary
  if ((uintptr_t)src % 16 == 0) {
    done = bytes >> 4 << 2;
#pragma unroll 4
    for (int i = threadIdx.x; i < done >> 2; i += 256) reinterpret_cast<uint4*>(s_words)[i] = reinterpret_cast<const uint4*>(src)[i];
  }
  for (int i = done + threadIdx.x; i < bytes >> 2; i += 256) s_words[i] = reinterpret_cast<const uint32_t*>(src)[i];
  uint8_t* s_bytes = reinterpret_cast<uint8_t*>(s_words);
  if ((int)threadIdx.x < (bytes & 3)) s_bytes[(bytes & ~3) + threadIdx.x] = src[(bytes & ~3) + threadIdx.x];
  __syncthreads();
  for (int i = threadIdx.x; i < KT * TN; i += 256) {
    const int c = i & (TN - 1), kt = i >> 7;
    const int r = MX ? (c >> 2) + 32 * (c & 3) : c;  // block-scaled word: (r % 32) * 4 + r / 32
    uint32_t w = 0;
    if (r < rows) {                                  // four bytes at any place, from the two words that hold them (with bytes one by one and 4-byte copies in 8.7 and 9.3 us in place, so 7.5 and 7.9)
      const int at = r * groups + kt * 4, live = min(4, groups - kt * 4);
      w = __funnelshift_r(s_words[at >> 2], s_words[min((at >> 2) + 1, (bytes - 1) >> 2)], 8 * (at & 3));
      if (live < 4) w &= (1u << (8 * live)) - 1u;
    }
    const int64_t tile = MX ? ((int64_t)e * KT + kt) * NB + nb : ((int64_t)e * NB + nb) * KT + kt;
    out[tile * TN + c] = w;
  }
}
// false: the scales are laid out in some other way
template <bool MX>
bool launch_scales_from_rows(const uint8_t* s, int64_t s_stride_e, int64_t s_stride_k, int64_t s_stride_n, int E, int K, int N, int NB, int KT,
                             uint32_t* out, cudaStream_t st) {
  const int groups = K / 32, smem = TN * groups;
  if (K % 32 || s_stride_k != 1 || s_stride_n != groups || s_stride_e % 4 || (uintptr_t)s % 4 || smem > SCALE_ROWS_SMEM ||
      (int64_t)E * NB >= 2147483647LL)
    return false;
  scales_from_rows<MX><<<(unsigned)(E * NB), 256, smem, st>>>(s, s_stride_e, groups, N, NB, KT, out);
  return true;
}

__global__ void __launch_bounds__(256) to_b200_scales(const uint8_t* __restrict__ s, int64_t s_stride_e,
                                                      int64_t s_stride_k, int64_t s_stride_n, int E, int K, int N,
                                                      int NT, int KT, uint32_t* __restrict__ out) {
  const int64_t total = (int64_t)E * NT * KT * TN;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int r = (int)(i & (TN - 1));
    int64_t t = i >> 7;
    const int kt = (int)(t % KT); t /= KT;
    const int nt = (int)(t % NT);
    const int e = (int)(t / NT);
    const int n = nt * TN + r;
    uint32_t w = 0;
    if (n < N) {
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const int kg = kt * 4 + g;
        if (kg * 32 < K)
          w |= (uint32_t)s[(int64_t)e * s_stride_e + (int64_t)kg * s_stride_k + (int64_t)n * s_stride_n] << (8 * g);
      }
    }
    out[i] = w;
  }
}

__global__ void __launch_bounds__(256) from_b200_kernel(const uint32_t* __restrict__ values,
                                                        const uint8_t* __restrict__ scales, int E, int K, int N, int NT,
                                                        int KT, uint8_t* __restrict__ q, uint8_t* __restrict__ s) {
  const int64_t words_per_row = K >> 3;
  const int64_t total = (int64_t)E * N * words_per_row;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t wj = i % words_per_row;
    int64_t t = i / words_per_row;
    const int n = (int)(t % N);
    const int e = (int)(t / N);
    const int k = (int)(wj * 8);
    const int nt = n / TN, r = n % TN, kt = k / TK, j = (k % TK) / 8;
    const int64_t tile = ((int64_t)e * NT + nt) * KT + kt;
    if (q) {
      const uint32_t w = nibble_deinterleave(values[tile * (TN * 16) + (j >> 2) * (TN * 4) + r * 4 + (j & 3)]);
      uint8_t* dst = q + ((int64_t)e * N + n) * (K >> 1) + (k >> 1);
      dst[0] = (uint8_t)w; dst[1] = (uint8_t)(w >> 8); dst[2] = (uint8_t)(w >> 16); dst[3] = (uint8_t)(w >> 24);
    }
    if (s && (k & 31) == 0)
      s[((int64_t)e * N + n) * (K >> 5) + (k >> 5)] = scales[tile * (TN * 4) + r * 4 + ((k % TK) >> 5)];
  }
}

template <bool SCALED>
void launch_to_tiles(const uint8_t* q, int64_t q_stride_e, int64_t q_stride_n, int E, int K, int N, int NT, int KT, uint8_t* out,
                     cudaStream_t st) {
  const int64_t tiles = (int64_t)E * NT * KT, cap = (int64_t)moe_sm_count() * 32;
  const int grid = (int)(tiles < cap ? tiles : cap);
  if ((uintptr_t)q % 16 == 0 && q_stride_e % 16 == 0 && q_stride_n % 16 == 0)
    to_tiles_values<SCALED, true><<<grid, 256, 0, st>>>(q, q_stride_e, q_stride_n, E, K, N, NT, KT, (uint4*)out);
  else
    to_tiles_values<SCALED, false><<<grid, 256, 0, st>>>(q, q_stride_e, q_stride_n, E, K, N, NT, KT, (uint4*)out);
}

int grid_for(int64_t total) {
  int64_t blocks = cdiv64(total, 256);
  int64_t cap = (int64_t)moe_sm_count() * 16;
  if (blocks > cap) blocks = cap;
  return (int)(blocks < 1 ? 1 : blocks);
}

}  // namespace

extern "C" __attribute__((visibility("default"))) size_t moe_weight_b200_value_bytes(int E, int K, int N) {
  return (size_t)E * (size_t)cdiv64(N, TN) * (size_t)cdiv64(K, TK) * (size_t)(TN * TK / 2);
}
extern "C" __attribute__((visibility("default"))) size_t moe_weight_b200_scale_bytes(int E, int K, int N) {
  return (size_t)E * (size_t)cdiv64(N, TN) * (size_t)cdiv64(K, TK) * (size_t)(TN * 4);
}

extern "C" __attribute__((visibility("default"))) int moe_weight_layout_to_b200(const uint8_t* q, int64_t q_stride_e, int64_t q_stride_n, const uint8_t* scale,
                                         int64_t s_stride_e, int64_t s_stride_k, int64_t s_stride_n, int E, int K, int N,
                                         uint8_t* out_values, uint8_t* out_scales, void* stream) {
  MOE_CHECK_ARG(E > 0 && K > 0 && N > 0 && K % 32 == 0, "moe_weight_layout_to_b200: need K %% 32 == 0 (K=%d)", K);
  MOE_CHECK_ARG((q != nullptr) == (out_values != nullptr) && (scale != nullptr) == (out_scales != nullptr) &&
                    (q || scale),
                "moe_weight_layout_to_b200: pass (q, out_values) and/or (scale, out_scales)");
  MOE_CHECK_ARG((uintptr_t)out_values % 16 == 0 && (uintptr_t)out_scales % 16 == 0,
                "moe_weight_layout_to_b200: outputs must be 16-byte aligned");
  const int NT = (int)cdiv64(N, TN), KT = (int)cdiv64(K, TK);
  cudaStream_t st = (cudaStream_t)stream;
  if (q) {
    launch_to_tiles<false>(q, q_stride_e, q_stride_n, E, K, N, NT, KT, out_values, st);
    MOE_CHECK_LAUNCH();
  }
  if (scale) {
    if (!launch_scales_from_rows<false>(scale, s_stride_e, s_stride_k, s_stride_n, E, K, N, NT, KT, (uint32_t*)out_scales, st))
      to_b200_scales<<<grid_for((int64_t)E * NT * KT * TN), 256, 0, st>>>(scale, s_stride_e, s_stride_k, s_stride_n, E, K,
                                                                         N, NT, KT, (uint32_t*)out_scales);
    MOE_CHECK_LAUNCH();
  }
  return MOE_OK;
}

extern "C" __attribute__((visibility("default"))) int moe_weight_layout_from_b200(const uint8_t* values, const uint8_t* scales, int E, int K, int N,
                                           uint8_t* q, uint8_t* scale, void* stream) {
  MOE_CHECK_ARG(E > 0 && K > 0 && N > 0 && K % 32 == 0, "moe_weight_layout_from_b200: need K %% 32 == 0 (K=%d)", K);
  MOE_CHECK_ARG((values != nullptr) == (q != nullptr) && (scales != nullptr) == (scale != nullptr) && (q || scale),
                "moe_weight_layout_from_b200: pass (values, q) and/or (scales, scale)");
  const int NT = (int)cdiv64(N, TN), KT = (int)cdiv64(K, TK);
  from_b200_kernel<<<grid_for((int64_t)E * N * (K >> 3)), 256, 0, (cudaStream_t)stream>>>(
      (const uint32_t*)values, scales, E, K, N, NT, KT, q, scale);
  MOE_CHECK_LAUNCH();
  return MOE_OK;
}

// ---- block-scaled layout (what the kind::mxf8f6f4 kernel streams) --------------------------------------------------
// Tiles of 128 n x 128 k ordered [E][k_tile][n_block]: the blocks a CTA tile needs in one k step are neighbours.
//   value tile: 128 rows x 64 bytes, byte b of a row holding k = 2b (low nibble) and 2b + 1 (high nibble) -- plain
//               packed e2m1, which the TMA unit expands to one byte per element on its way into shared memory;
//   scale tile: 512 bytes, the scale of (row r, group g) at (r % 32) * 16 + (r / 32) * 4 + g: the order tcgen05.cp
//               (32x128b.warpx4) moves into tensor memory, the same 128 x 4 packed block as BlackwellMXScaleLayout of
//               the reference (tensor_details/layout_details/blackwell_scale.py:165-175).
// Out-of-range n or k is zero (value 0, scale byte 0 = 2^-127).
namespace {

__global__ void __launch_bounds__(256) to_b200mx_scales(const uint8_t* __restrict__ s, int64_t s_stride_e,
                                                        int64_t s_stride_k, int64_t s_stride_n, int E, int K, int N,
                                                        int NB, int KT, uint32_t* __restrict__ out) {
  const int64_t total = (int64_t)E * KT * NB * TN;                  // one 32-bit word = the 4 groups of a row
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int c = (int)(i & (TN - 1));                 // word inside the tile: (r % 32) * 4 + r / 32
    const int r = (c >> 2) + 32 * (c & 3);
    int64_t t = i >> 7;
    const int nb = (int)(t % NB); t /= NB;
    const int kt = (int)(t % KT);
    const int e = (int)(t / KT);
    const int n = nb * TN + r;
    uint32_t w = 0;
    if (n < N) {
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const int kg = kt * 4 + g;
        if (kg * 32 < K)
          w |= (uint32_t)s[(int64_t)e * s_stride_e + (int64_t)kg * s_stride_k + (int64_t)n * s_stride_n] << (8 * g);
      }
    }
    out[i] = w;
  }
}

__global__ void __launch_bounds__(256) from_b200mx_kernel(const uint32_t* __restrict__ values,
                                                          const uint8_t* __restrict__ scales, int E, int K, int N, int NB,
                                                          int KT, uint8_t* __restrict__ q, uint8_t* __restrict__ s) {
  const int64_t words_per_row = K >> 3;
  const int64_t total = (int64_t)E * N * words_per_row;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t wj = i % words_per_row;
    int64_t t = i / words_per_row;
    const int n = (int)(t % N);
    const int e = (int)(t / N);
    const int k = (int)(wj * 8);
    const int nb = n / TN, r = n % TN, kt = k / TK, j = (k % TK) / 8;
    const int64_t tile = ((int64_t)e * KT + kt) * NB + nb;
    if (q) {
      const uint32_t w = values[tile * (TN * 16) + r * 16 + j];
      uint8_t* dst = q + ((int64_t)e * N + n) * (K >> 1) + (k >> 1);
      dst[0] = (uint8_t)w; dst[1] = (uint8_t)(w >> 8); dst[2] = (uint8_t)(w >> 16); dst[3] = (uint8_t)(w >> 24);
    }
    if (s && (k & 31) == 0)
      s[((int64_t)e * N + n) * (K >> 5) + (k >> 5)] = scales[tile * 512 + (r & 31) * 16 + (r >> 5) * 4 + ((k % TK) >> 5)];
  }
}

}  // namespace

extern "C" __attribute__((visibility("default"))) int moe_weight_layout_to_b200mx(const uint8_t* q, int64_t q_stride_e, int64_t q_stride_n, const uint8_t* scale,
                                         int64_t s_stride_e, int64_t s_stride_k, int64_t s_stride_n, int E, int K, int N,
                                         uint8_t* out_values, uint8_t* out_scales, void* stream) {
  MOE_CHECK_ARG(E > 0 && K > 0 && N > 0 && K % 32 == 0, "moe_weight_layout_to_b200mx: need K %% 32 == 0 (K=%d)", K);
  MOE_CHECK_ARG((q != nullptr) == (out_values != nullptr) && (scale != nullptr) == (out_scales != nullptr) &&
                    (q || scale),
                "moe_weight_layout_to_b200mx: pass (q, out_values) and/or (scale, out_scales)");
  MOE_CHECK_ARG((uintptr_t)out_values % 32 == 0 && (uintptr_t)out_scales % 16 == 0,
                "moe_weight_layout_to_b200mx: values must be 32-byte and scales 16-byte aligned");
  const int NB = (int)cdiv64(N, TN), KT = (int)cdiv64(K, TK);
  cudaStream_t st = (cudaStream_t)stream;
  if (q) {
    launch_to_tiles<true>(q, q_stride_e, q_stride_n, E, K, N, NB, KT, out_values, st);
    MOE_CHECK_LAUNCH();
  }
  if (scale) {
    if (!launch_scales_from_rows<true>(scale, s_stride_e, s_stride_k, s_stride_n, E, K, N, NB, KT, (uint32_t*)out_scales, st))
      to_b200mx_scales<<<grid_for((int64_t)E * NB * KT * TN), 256, 0, st>>>(scale, s_stride_e, s_stride_k, s_stride_n, E, K,
                                                                           N, NB, KT, (uint32_t*)out_scales);
    MOE_CHECK_LAUNCH();
  }
  return MOE_OK;
}

extern "C" __attribute__((visibility("default"))) int moe_weight_layout_from_b200mx(const uint8_t* values, const uint8_t* scales, int E, int K, int N,
                                           uint8_t* q, uint8_t* scale, void* stream) {
  MOE_CHECK_ARG(E > 0 && K > 0 && N > 0 && K % 32 == 0, "moe_weight_layout_from_b200mx: need K %% 32 == 0 (K=%d)", K);
  MOE_CHECK_ARG((values != nullptr) == (q != nullptr) && (scales != nullptr) == (scale != nullptr) && (q || scale),
                "moe_weight_layout_from_b200mx: pass (values, q) and/or (scales, scale)");
  const int NB = (int)cdiv64(N, TN), KT = (int)cdiv64(K, TK);
  from_b200mx_kernel<<<grid_for((int64_t)E * N * (K >> 3)), 256, 0, (cudaStream_t)stream>>>(
      (const uint32_t*)values, scales, E, K, N, NB, KT, q, scale);
  MOE_CHECK_LAUNCH();
  return MOE_OK;
}
