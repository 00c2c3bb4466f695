// Two products of a layer in a row: the first one's epilogue leaves its SwiGLU rows in the operand form of the second (what that
// product's pack kernel would make of them, byte for byte), so they are neither written and read again as rows nor packed by a
// launch of their own.  The forms: two e4m3 terms (or e4m3 rows as one) in the lines of the pair kernel or the chunks of the
// decode kernel, four e2m1 terms in such chunks.
//
// Measured, us per layer step with pack launch and without: 8 experts of 512 x 2048, 256 tokens 37.4 -> 29.8; 128 experts of 2880 x 5760,
// 300 tokens 324 -> 306 (its pack: 11), 16384 tokens 3260 -> 3147 (137, of 767 MB through HBM), e4m3 8192 tokens, 32 experts 974 -> 914.
#pragma once
#include "gemm_mx_common.cuh"

namespace {

// output types of a GEMM kernel that writes tokens: e4m3 rows, bf16 rows as two e4m3 terms, bf16 rows as four e2m1 terms
struct Tok1 { uint8_t byte; };
struct Tok2 { uint16_t half; };
struct Tok4 { uint16_t half; };
template <typename TY> constexpr int TOK_TERMS = 0;
template <> constexpr int TOK_TERMS<Tok1> = 1;
template <> constexpr int TOK_TERMS<Tok2> = 2;
template <> constexpr int TOK_TERMS<Tok4> = 4;

// first padded row of an expert in the pair kernel's lines: a multiple of 32, and never before the end of the previous expert's last
// group of 32
__device__ __forceinline__ int64_t padded_base(int e, int off) { return (int64_t)(off & ~31) + 32 * (int64_t)e; }

// Values (one line of 64 or 128 bytes) and scales of row r of expert e, whose rows start at `off`, at k step 0.  first_block:
// chunk form, o.block_offs[e].
__device__ __forceinline__ void token_addr(const TokenOut& o, int e, int off, int first_block, int r, uint8_t*& q, uint8_t*& s) {
  if (o.tb == 0) {
    const int64_t prow = padded_base(e, off) + r, line = o.terms * (prow & ~(int64_t)7) + (prow & 7);
    q = o.q + line * 128;
    s = o.s + line * 4;
  } else {
    const int j = r / o.tb, rr = r - j * o.tb;
    const int64_t at = (int64_t)(first_block + j) * o.block_bytes;
    q = o.q + at + rr * (o.terms == 4 ? 64 : 128);
    s = o.s + at + (rr & 31) * 16 + (rr >> 5) * 4;
  }
}

// N values of a 32-group as two e4m3 terms, N / 8 words of eight codes each in the order of k; the group's maxima come from `all`
template <int N, typename F>
__device__ __forceinline__ void two_terms(float (&v)[N], F all, uint32_t (&h)[N / 4], uint32_t (&l)[N / 4], uint32_t& sh, uint32_t& sl, float& amax) {
  float m = 0.0f;
#pragma unroll
  for (int i = 0; i < N; ++i) m = fmaxf(m, fabsf(v[i]));
  amax = m = all(m);
  float s_hi, i_hi;
  mx8_scale(m, sh, s_hi, i_hi);
  float rm = 0.0f;
#pragma unroll
  for (int i = 0; i < N / 2; ++i) {
    const uint32_t c = f32x2_to_e4m3x2(v[2 * i] * i_hi, v[2 * i + 1] * i_hi);
    const float2 f = e4m3x2_to_f32x2(c);
    v[2 * i] -= f.x * s_hi;
    v[2 * i + 1] -= f.y * s_hi;
    rm = fmaxf(rm, fmaxf(fabsf(v[2 * i]), fabsf(v[2 * i + 1])));
    h[i >> 1] = (i & 1) ? (h[i >> 1] | (c << 16)) : c;
  }
  rm = all(rm);
  if (!(rm < 3.0e38f)) rm = 0.0f;
  float s_lo, i_lo;
  mx8_scale(rm, sl, s_lo, i_lo);
#pragma unroll
  for (int i = 0; i < N / 4; ++i)
    l[i] = f32x2_to_e4m3x2(v[4 * i] * i_lo, v[4 * i + 1] * i_lo) | (f32x2_to_e4m3x2(v[4 * i + 2] * i_lo, v[4 * i + 3] * i_lo) << 16);
}

// ---- epilogue ------------------------------------------------------------------------------------------------------
// Accumulator [weight row = lane][token = column], gate and linear in neighbouring lanes: the lane pair swaps halves of a 16-token
// chunk, and lane `odd` gets the outputs of tokens 8 odd .. + 7 of the pair's column.
__device__ __forceinline__ void swiglu_chunk(const GemmParams& p, const uint32_t (&raw)[16], float bias, int odd, float (&y)[8]) {
  float v[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(raw[j]) + bias;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float recv = __shfl_xor_sync(0xFFFFFFFFu, odd ? v[j] : v[8 + j], 1);
    y[j] = gemm_swiglu(odd ? recv : v[j], odd ? v[8 + j] : recv, p.act_alpha, p.act_limit, p.act_has_limit);
  }
}

// Two warps hold a group of 32 outputs (64 weight rows) of 16 tokens.  They meet in shared memory ([token][72 bytes]: rows of 18
// words keep the lanes of a warp on distinct banks), then four lanes take a token, eight outputs each.
constexpr int TOK_PITCH = 72, TOK_STAGE = 16 * TOK_PITCH;
struct TokStage {
  uint32_t at;                   // shared memory of the pair of warps
  int bar;                       // their named barrier
  int i;                         // thread 0 .. 63 of the pair
  __device__ __forceinline__ void sync() const { asm volatile("bar.sync %0, 64;" ::"r"(bar) : "memory"); }
  // the same answer in both warps, so that neither leaves the other at a barrier
  __device__ __forceinline__ bool all(bool ok) const {
    int r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbar.red.and.pred q, %2, 64, p;\n\tselp.b32 %0, 1, 0, q;\n\t}"
                 : "=r"(r) : "r"((int)ok), "r"(bar) : "memory");
    return r != 0;
  }
};
__device__ __forceinline__ uint2 lds64(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
  return v;
}

// y[u]: outputs of tokens 8 odd .. + 7 in column `col` (0 .. 31) of group g + 2 u, for `live` of the U neighbouring weight blocks (a
// stage each, their chains side by side); q, s: lines of token i >> 2 of the chunk at k step 0 (q NULL: not stored).  zero_next: the
// group two past the last block's is past K too, and zero.
template <typename TY, int U>
__device__ __forceinline__ void emit_tokens(const TokenOut& o, const TokStage& st, const float (&y)[U][8], int live, int col, int odd, int g,
                                            uint8_t* q, uint8_t* s, bool zero_next) {
  constexpr int TERMS = TOK_TERMS<TY>;
  const uint32_t w = st.at + (uint32_t)(odd * 8 * TOK_PITCH + col * (TERMS == 1 ? 1 : 2));
#pragma unroll
  for (int u = 0; u < U; ++u)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint32_t at = w + (uint32_t)(u * TOK_STAGE + j * TOK_PITCH);
      if constexpr (TERMS == 1)
        asm volatile("st.shared.u8 [%0], %1;" ::"r"(at), "r"((uint32_t)from_f32<__nv_fp8_e4m3>(y[u][j]).__x) : "memory");
      else
        asm volatile("st.shared.u16 [%0], %1;" ::"r"(at), "h"(__bfloat16_as_ushort(__float2bfloat16_rn(y[u][j]))) : "memory");
    }
  st.sync();
  const int token = st.i >> 2, l4 = st.i & 3;
  const uint32_t r = st.at + (uint32_t)(token * TOK_PITCH + l4 * (TERMS == 1 ? 8 : 16));
  uint2 lo[U], hi[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    lo[u] = lds64(r + (uint32_t)(u * TOK_STAGE));
    if constexpr (TERMS != 1) hi[u] = lds64(r + (uint32_t)(u * TOK_STAGE) + 8u);
  }
  st.sync();                                           // the stage may be written again
  const int x7 = token & 7;                            // (chunks start at multiples of 8 rows)
  // the value bytes of these lanes in group gg, its scale
  auto value = [&](int gg) {
    uint8_t* line = q + (gg >> 2) * o.q_step;
    if constexpr (TERMS == 4) return line + (((gg & 3) ^ (x7 >> 1 & 3)) << 4) + l4 * 4;
    else return line + (((2 * (gg & 3) + (l4 >> 1)) ^ x7) << 4) + (l4 & 1) * 8;
  };
  auto scale = [&](int gg) { return s + (gg >> 2) * o.s_step + (gg & 3); };
  if constexpr (TERMS == 1) {
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (q && u < live) {
        *reinterpret_cast<uint2*>(value(g + 2 * u)) = lo[u];
        if (l4 == 0) *scale(g + 2 * u) = 127;          // 1.0
      }
  } else {
    float v[U][8];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t raw[4] = {lo[u].x, lo[u].y, hi[u].x, hi[u].y};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        v[u][2 * j] = __uint_as_float(raw[j] << 16);
        v[u][2 * j + 1] = __uint_as_float(raw[j] & 0xFFFF0000u);
      }
    }
    if constexpr (TERMS == 4) {
      bool nan[U][8];
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int j = 0; j < 8; ++j) nan[u][j] = v[u][j] != v[u][j];
#pragma unroll
      for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int u = 0; u < U; ++u) {
          uint32_t codes;
          const uint32_t sb = e2m1_term(t, v[u], nan[u], codes, [](uint32_t top) {
            top = max(top, __shfl_xor_sync(0xFFFFFFFFu, top, 1));
            return max(top, __shfl_xor_sync(0xFFFFFFFFu, top, 2));
          });
          if (q && u < live) {
            *reinterpret_cast<uint32_t*>(value(g + 2 * u) + t * o.lo_q) = codes;
            if (l4 == 0) scale(g + 2 * u)[(t & 1) * 256 + (t >> 1) * 4] = (uint8_t)sb;      // row t * 16 + r of the chunk
          }
        }
    } else {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        uint32_t h[2], l[2], sh, sl;
        float amax;
        two_terms<8>(v[u], [](float m) {
          m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, 1));
          return fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, 2));
        }, h, l, sh, sl, amax);
        if (o.permuted) {                              // k inside eight: even, then odd
          const uint32_t h0 = __byte_perm(h[0], h[1], 0x6420), l0 = __byte_perm(l[0], l[1], 0x6420);
          h[1] = __byte_perm(h[0], h[1], 0x7531); h[0] = h0;
          l[1] = __byte_perm(l[0], l[1], 0x7531); l[0] = l0;
        }
        if (q && u < live) {
          uint8_t* d = value(g + 2 * u);
          *reinterpret_cast<uint2*>(d) = make_uint2(h[0], h[1]);
          *reinterpret_cast<uint2*>(d + o.lo_q) = make_uint2(l[0], l[1]);
          if (l4 == 0) {
            scale(g + 2 * u)[0] = (uint8_t)sh;
            scale(g + 2 * u)[o.lo_s] = (uint8_t)sl;
          }
        }
      }
    }
  }
  if (zero_next && q) {
    const int gz = g + 2 * live;
#pragma unroll
    for (int t = 0; t < TERMS; ++t) {
      uint8_t* d = value(gz) + t * o.lo_q;
      if constexpr (TERMS == 4) *reinterpret_cast<uint32_t*>(d) = 0;
      else *reinterpret_cast<uint2*>(d) = make_uint2(0, 0);
      if (l4 == 0) scale(gz)[TERMS == 4 ? (t & 1) * 256 + (t >> 1) * 4 : t * o.lo_s] = 127;
    }
  }
}

}  // namespace
