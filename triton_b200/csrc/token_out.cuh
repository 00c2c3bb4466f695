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

// Lines a term of a token block of `rows` rows takes in its chunk where chunks fit their rows: 16, 32 or 64.
__device__ __forceinline__ int chunk_lines(int rows) { return rows <= 16 ? 16 : rows <= 32 ? 32 : 64; }
// scale of line r of a chunk, from the start of its scales
__device__ __forceinline__ int chunk_scale(int r) { return (r & 31) * 16 + (r >> 5) * 4; }

// Values (one line of 64 or 128 bytes) and scales of row r of expert e, whose `size` rows start at `off`, at k step 0.  first_block:
// chunk form, o.block_offs[e].  The low two bits of s: log2 of the lines of a term / 8 (chunk form of several terms).
__device__ __forceinline__ void token_addr(const TokenOut& o, int e, int off, int size, int first_block, int r, uint8_t*& q, uint8_t*& s) {
  if (o.tb == 0) {
    const int64_t prow = padded_base(e, off) + r, line = o.terms * (prow & ~(int64_t)7) + (prow & 7);
    q = o.q + line * 128;
    s = o.s + line * 4;
  } else {
    const int j = r / o.tb, rr = r - j * o.tb, row = o.terms == 4 ? 64 : 128;
    const int lines = o.fit ? chunk_lines(min(o.tb, size - j * o.tb)) : o.tb;
    uint8_t* chunk = o.q + (int64_t)(first_block + j) * o.block_bytes;
    q = chunk + rr * row;
    s = chunk + (o.terms == 1 ? o.n_one : o.terms * lines) * row + chunk_scale(rr) + (o.terms == 1 ? 0 : 28 - __clz(lines));
  }
}
// from a term's line and scale to the next term's (scale: two terms)
__device__ __forceinline__ void token_strides(const TokenOut& o, const uint8_t* s, int& lo_q, int& lo_s) {
  const int lines = 8 << ((uintptr_t)s & 3u);
  lo_q = o.tb == 0 ? 1024 : lines * (o.terms == 4 ? 64 : 128);
  lo_s = o.tb == 0 ? 32 : lines < 32 ? lines * 16 : lines / 8;
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
    v[2 * i] = left_over(v[2 * i], f.x, s_hi);
    v[2 * i + 1] = left_over(v[2 * i + 1], f.y, s_hi);
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
// Accumulator [weight row = lane][token = column], gate and linear in neighbouring lanes: the lane pair swaps halves of N tokens, and lane
// `odd` gets the outputs of tokens N / 2 odd .. of the pair's column.
template <int N>
__device__ __forceinline__ void swiglu_chunk(const GemmParams& p, const uint32_t (&raw)[N], float bias, int odd, float (&y)[N / 2]) {
  float v[N];
#pragma unroll
  for (int j = 0; j < N; ++j) v[j] = __uint_as_float(raw[j]) + bias;
#pragma unroll
  for (int j = 0; j < N / 2; ++j) {
    const float recv = __shfl_xor_sync(0xFFFFFFFFu, odd ? v[j] : v[N / 2 + j], 1);
    y[j] = gemm_swiglu(odd ? recv : v[j], odd ? v[N / 2 + j] : recv, p.act_alpha, p.act_limit, p.act_has_limit);
  }
}

// Two warps hold a group of 32 outputs (64 weight rows) of 16 tokens.  They meet in shared memory ([token][72 bytes]: rows of 18
// words keep the lanes of a warp on distinct banks), then four lanes take a row of a group, eight outputs each.
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

// outputs of tokens token0 .. + N - 1 in column `col` (0 .. 31) of the group staged at `at`
template <typename TY, int N>
__device__ __forceinline__ void stage_tokens(uint32_t at, const float (&y)[N], int token0, int col) {
  const uint32_t w = at + (uint32_t)(token0 * TOK_PITCH + col * (TOK_TERMS<TY> == 1 ? 1 : 2));
#pragma unroll
  for (int j = 0; j < N; ++j) {
    if constexpr (TOK_TERMS<TY> == 1)
      asm volatile("st.shared.u8 [%0], %1;" ::"r"(w + (uint32_t)(j * TOK_PITCH)), "r"((uint32_t)from_f32<__nv_fp8_e4m3>(y[j]).__x) : "memory");
    else
      asm volatile("st.shared.u16 [%0], %1;" ::"r"(w + (uint32_t)(j * TOK_PITCH)), "h"(__bfloat16_as_ushort(__float2bfloat16_rn(y[j]))) : "memory");
  }
}

// This lane's eight values (l4: which) of a staged row
struct StagedRow { uint2 lo, hi; };
template <typename TY> __device__ __forceinline__ StagedRow staged_row(uint32_t at, int token, int l4) {
  const uint32_t r = at + (uint32_t)(token * TOK_PITCH + l4 * (TOK_TERMS<TY> == 1 ? 8 : 16));
  StagedRow v{lds64(r), make_uint2(0, 0)};
  if constexpr (TOK_TERMS<TY> != 1) v.hi = lds64(r + 8u);
  return v;
}

// The row, group g of its token: q, s are the token's line and scales at k step 0 (q NULL: not stored), x7 its row mod 8.  All 32 lanes
// call, four neighbouring ones a row.  zero_next: group g + 2 is past the last weight block, and zero.
template <typename TY>
__device__ __forceinline__ void emit_group(const TokenOut& o, const StagedRow& row, int l4, int x7, int g, uint8_t* q, uint8_t* s, bool zero_next) {
  constexpr int TERMS = TOK_TERMS<TY>;
  int lo_q, lo_s;
  token_strides(o, s, lo_q, lo_s);
  s = (uint8_t*)((uintptr_t)s & ~(uintptr_t)3);
  // scale of term t: with four terms line 16 t + r of the chunk
  auto term_scale = [&](int t) { return TERMS == 4 ? (t & 1) * 256 + (t >> 1) * 4 : t * lo_s; };
  // the value bytes of these lanes in group gg
  auto value = [&](int gg) {
    uint8_t* line = q + (gg >> 2) * o.q_step;
    if constexpr (TERMS == 4) return line + (((gg & 3) ^ (x7 >> 1 & 3)) << 4) + l4 * 4;
    else return line + (((2 * (gg & 3) + (l4 >> 1)) ^ x7) << 4) + (l4 & 1) * 8;
  };
  uint8_t *d = value(g), *sd = s + (g >> 2) * o.s_step + (g & 3);
  if constexpr (TERMS == 1) {
    if (q) {
      *reinterpret_cast<uint2*>(d) = row.lo;
      if (l4 == 0) sd[0] = 127;                        // 1.0
    }
  } else {
    const uint32_t raw[4] = {row.lo.x, row.lo.y, row.hi.x, row.hi.y};
    float v[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      v[2 * j] = __uint_as_float(raw[j] << 16);
      v[2 * j + 1] = __uint_as_float(raw[j] & 0xFFFF0000u);
    }
    if constexpr (TERMS == 4) {
      bool nan[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) nan[j] = v[j] != v[j];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        uint32_t codes;
        const uint32_t sb = e2m1_term(t, v, nan, codes, [](uint32_t top) {
          top = max(top, __shfl_xor_sync(0xFFFFFFFFu, top, 1));
          return max(top, __shfl_xor_sync(0xFFFFFFFFu, top, 2));
        });
        if (q) {
          *reinterpret_cast<uint32_t*>(d + t * lo_q) = codes;
          if (l4 == 0) sd[term_scale(t)] = (uint8_t)sb;
        }
      }
    } else {
      uint32_t h[2], l[2], sh, sl;
      float amax;
      two_terms<8>(v, [](float m) {
        m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, 1));
        return fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, 2));
      }, h, l, sh, sl, amax);
      if (o.permuted) {                                // k inside eight: even, then odd
        const uint32_t h0 = __byte_perm(h[0], h[1], 0x6420), l0 = __byte_perm(l[0], l[1], 0x6420);
        h[1] = __byte_perm(h[0], h[1], 0x7531); h[0] = h0;
        l[1] = __byte_perm(l[0], l[1], 0x7531); l[0] = l0;
      }
      if (q) {
        *reinterpret_cast<uint2*>(d) = make_uint2(h[0], h[1]);
        *reinterpret_cast<uint2*>(d + lo_q) = make_uint2(l[0], l[1]);
        if (l4 == 0) {
          sd[0] = (uint8_t)sh;
          sd[lo_s] = (uint8_t)sl;
        }
      }
    }
  }
  if (zero_next && q) {
    uint8_t* z = value(g + 2);
#pragma unroll 1
    for (int t = 0; t < TERMS; ++t) {
      if constexpr (TERMS == 4) *reinterpret_cast<uint32_t*>(z + t * lo_q) = 0;
      else *reinterpret_cast<uint2*>(z + t * lo_q) = make_uint2(0, 0);
      if (l4 == 0) sd[term_scale(t) + 2] = 127;
    }
  }
}

}  // namespace
