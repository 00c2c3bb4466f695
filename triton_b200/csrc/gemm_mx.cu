// Ragged grouped GEMM on the block-scaled tensor-core path of sm_100a:
//   tcgen05.mma.kind::mxf8f6f4.block_scale -- e2m1 weights with their e8m0 scales go into the MMA as they are
//   stored (no software dequantisation), activations are e4m3 with e8m0 scales per 32 k.
//
// What the reference reaches through `PrecisionConfig(a_mx_scale=..., b_mx_scale=...)` and fp8 activations
// (triton_kernels matmul.py:130-132, 311-336; matmul_details/_p_matmul.py:399-407): its MXFP4 weights feed
// tl.dot_scaled, which lowers to this instruction kind.
//
// Operand roles are swapped with respect to the bf16 kernel: the WEIGHTS are the M = 128 operand (a tile is 128
// weight rows x 128 k) and the TOKENS are the N operand (16 .. 128 columns), so that a handful of tokens costs a
// handful of accumulator columns.  A CTA tile is MB (1 to 3) weight blocks x one block of tokens; the token block
// stays in shared memory per k step and is shared by the MB weight blocks.
//
// bf16 activations are split into two e4m3 terms, hi = mxfp8(x) and lo = mxfp8(x - hi), each with its own e8m0
// scale per 32 k (error about 2^-8 of the group maximum, inside the tolerance of the bf16 path).  Both terms sit
// side by side as N columns of ONE MMA ([hi tokens | lo tokens], every column has its own scale), the epilogue adds the
// two accumulator columns of a token.  e4m3 / MXFP8 activations enter as they are (one term).
//
// With at most 16 token rows per block (decode) bf16 activations take a second form: FOUR e2m1 terms, each the MXFP4
// quantisation of what the terms before it left over (about 2^-14 of the group maximum after four), and the MMA is
//   tcgen05.mma.kind::mxf4.block_scale.scale_vec::2X -- K = 64 per instruction and both operands packed, so a
// weight tile stays 8 KB in shared memory (plain TMA copy, 64-byte swizzle) instead of the 16 KB of the byte-per-
// element form, and a k step costs half the MMA instructions.  Twice the bytes in flight per SM and half the
// instruction count are what a weight-streaming step is short of; the four terms are four groups of N columns.
//
// Data flow of one k step (128 k):
//   weights     one TMA tensor copy: MB x (128 rows x 64 packed bytes) from the tile-contiguous layout of
//               moe_weight_layout_to_b200mx, unpacked by the TMA unit (CU_TENSOR_MAP_DATA_TYPE_16U4_ALIGN16B) into the
//               byte-per-element, 128-byte-swizzled operand the MMA reads;
//   w scales    one bulk copy of MB x 512 B, already in the [32 lanes][4 quarters][4 k groups] order;
//   tokens      one bulk copy of a chunk the pack kernel below prepared per (token block, k step): the e4m3 rows in
//               the swizzled operand layout followed by their 512 B of scales;
//   scales -> tensor memory through registers (tcgen05.st by four loader warps), then MB x 4 MMAs of K = 32.
// Warps: 0 producer, 1 MMA issue + tensor-memory owner, 2-5 epilogue, 6-9 scale loaders.  Every mbarrier
// wait is bounded.
#include "token_out.cuh"
#include <type_traits>

namespace {

constexpr int MX_THREADS = 320;               // warp 0 producer, 1 MMA, 2-5 epilogue, 6-9 scale loaders
constexpr int MX_MAX_STAGES = 8;
constexpr int MX_W_TILE = 128 * 128;           // one weight block of a stage in shared memory (byte per element)
constexpr int MX_W_TILE_TX = 128 * 64;         // what its copy reports to the mbarrier: the packed bytes read; also the
                                               // size of a weight block that stays packed (four-term form)
constexpr int MX_WS_TILE = 512;                // its scales
constexpr int MX_SF_COLS = 16;                 // tensor-memory columns of scales per stage (MB x 4 + 4)
constexpr int MX_SF_BASE = 512 - MX_MAX_STAGES * MX_SF_COLS;    // 384: accumulators live below
constexpr int MX_SMEM_LIMIT = 227 * 1024;
constexpr int MX_CTL_BARS = 3 * MX_MAX_STAGES + 5;          // full, empty, scales-ready rings; 2 + 2 accumulator; drain
constexpr int MX_CTL_BYTES = MX_CTL_BARS * 8 + 16 + MX_MAX_STAGES * 4;      // + tensor-memory base, abort flag, columns of the tile that starts with a stage
// rows on their way to the next product's tokens: a stage per two epilogue warps and weight block of the tile
template <typename TY> constexpr int MX_TOK_BYTES = TOK_TERMS<TY> ? 6 * TOK_STAGE : 0;

struct MxParams {
  const uint8_t* xq;            // packed token chunks: [slot][k step][lines of the terms | 512 B of scales], at most chunk_bytes
  int64_t chunk_bytes;
  int n_mma;                    // MMA N at most: token columns (hi and lo when split); accumulators are this far apart
  int tb;                       // token rows per block (16, 32, 64 or 128)
  int split;                    // terms of a token: 1, 2 (bf16 as hi + lo e4m3) or 4 (bf16 as e2m1 terms); term t of
                                // token j is column t * lines + j, lines = tb or (FIT) what the block's rows need
  int KT, NB;                   // 128-k steps, 128-row weight blocks
  int stages, stage_bytes;
  int acc_bufs;
  int64_t grid_m;               // static bound on token blocks (dense problems: exact)
  int once;                     // weights are read about once: they are the first to leave L2
  uint32_t hint_m;              // and on the entries of the schedule that may be read before they are known to be written
  TokenOut out;                 // the rows as the next product's tokens
};

inline bool mx_fits(int split, int mb) { return split == 2 && mb > 1; }

struct MxMaps {
  CUtensorMap m[3];             // boxes of 1, 2 and 3 weight blocks
};

// The tiles of one CTA, in the order every role walks them.  A tile is one token block x up to MB consecutive weight
// blocks; tile = (weight group, token block) with token blocks varying fastest, dealt out round robin, so that CTAs
// running at the same time share a weight group (large problems: the group is read from HBM once).  (Equal contiguous
// ranges of weight blocks per CTA, which leave no partly filled last wave, were measured 5-12 % slower at 16 and 64
// tokens and, after the issuing warps got cheaper, 0-10 %: they cut more tiles short of MB blocks, and a k step costs about the same
// whatever it carries.  Slices of K per
// tile with fp32 partial sums in global memory -- red.global.add, the slice that arrives last runs the epilogue -- were
// correct and 20-35 % slower at 4 to 64 tokens: 48 scalar reductions per thread and slice, their fence and the counter
// round trip take longer than a slice of a few k steps, and the epilogue warps become the bottleneck.)
//
// The tiles that do not fill a last round are dealt out block by block where that is one round.  A block by itself has two k steps to
// a stage: a stage takes its way through copy, scales and MMA whatever it carries, with one k step a block took as long as
// three do.  (fc1 of 300 tokens, 1380 tiles: 158 -> 152 us; of 4 tokens, 150 tiles, with the code of the epilogue: 24 -> 20.)
struct MxSched {
  uint32_t useful_m, cur, end, whole, wide;      // tiles dealt out whole, tiles of MB blocks; `end` counts blocks behind the whole tiles
  int NB, MB;
  bool narrow = false;                           // the tile is a block by itself: two k steps a stage
  __device__ __forceinline__ MxSched(uint32_t useful_m_, int NB_, int MB_) : useful_m(useful_m_), cur(blockIdx.x), NB(NB_), MB(MB_) {
    const uint32_t rest = (uint32_t)(NB % MB), n = useful_m * (uint32_t)((NB + MB - 1) / MB);
    wide = useful_m * (uint32_t)(NB / MB);
    whole = end = n;
    const uint32_t last = n % gridDim.x, last_wide = wide + last > n ? wide + last - n : 0u;      // of the last round: tiles, wide ones
    const uint32_t blocks = last_wide * (uint32_t)MB + (last - last_wide) * rest;
    if (MB == 3 && last && blocks <= gridDim.x) {
      whole = n - last;
      end = whole + blocks;
    }
  }
  __device__ __forceinline__ bool next(int64_t& pid_m, int& nb0, int& mb_live) {
    if (cur >= end) return false;
    uint32_t tile = cur, block = 0;
    if (cur >= whole) {                          // block `block` of a tile of the last round, the wide ones first
      const uint32_t i = cur - whole, in_wide = (wide > whole ? wide - whole : 0u) * (uint32_t)MB;
      const uint32_t per = i < in_wide ? (uint32_t)MB : (uint32_t)(NB % MB), j = i < in_wide ? i : i - in_wide;
      tile = (i < in_wide ? whole : max(wide, whole)) + j / per;
      block = j % per;
    }
    const uint32_t grp = tile / useful_m;
    pid_m = tile - grp * useful_m;
    nb0 = (int)grp * MB + (int)block;
    mb_live = cur >= whole ? 1 : min(MB, NB - nb0);
    narrow = MB == 3 && mb_live == 1;
    cur += gridDim.x;
    return true;
  }
};

// ---- token block -> (expert, first row, rows) through the block schedule of the block size in use -----------
__device__ __forceinline__ bool mx_map_block(const GemmParams& p, int tb, int64_t pid_m, int& e, int64_t& row0, int& rows) {
  if (p.slice_sizes == nullptr) {
    e = 0;
    row0 = pid_m * tb;
    if (row0 >= p.M) return false;
    rows = (int)min((int64_t)tb, p.M - row0);
    return true;
  }
  const uint32_t ent = (uint32_t)p.block_sched[pid_m];
  if (ent == 0xFFFFFFFFu) return false;
  e = (int)(ent & 0xFFFFu);
  const int blk = (int)(ent >> 16);
  row0 = (int64_t)p.slice_offs[e] + (int64_t)blk * tb;
  rows = min(tb, p.slice_sizes[e] - blk * tb);
  return rows > 0;
}

// ============================================================================================================
// Pack kernel: token rows -> per (token block, k step) chunks in the operand layout of the MMA.
//   line r of the chunk (term t of row j: r = t * lines + j) is 128 bytes = 128 e4m3 values of k = 128 kt .. +127, its 16-byte pieces XOR-
//   swizzled with (r & 7) like a 128-byte-swizzled TMA tile; the scale of (row r, group g) is byte
//   (r % 32) * 16 + (r / 32) * 4 + g of the 512 bytes that follow the rows.
// grid = (token blocks, k steps); a warp takes a row at a time, a lane 4 consecutive k.
// ============================================================================================================
struct PackParams {
  const void* x; int64_t ld_x; int64_t rows_x;        // source rows; ld in elements
  const uint8_t* x_scale; int64_t ld_xs;              // e8m0 [rows_x, K / 32] for MXFP8 sources, else NULL
  const int32_t* gather;
  int K, KT, tb, n_mma, fit;
  int64_t chunk_bytes;
  uint8_t* out;
};

// four consecutive values of row `src` (lane l of a warp: k = 128 kt + 4 l), 0 where there are none
__device__ __forceinline__ void pack_load4(const PackParams& a, int64_t src, int k, bool live, float (&v)[4]) {
  uint2 raw = make_uint2(0, 0);
  if (live) raw = *reinterpret_cast<const uint2*>((const __nv_bfloat16*)a.x + src * a.ld_x + k);
  v[0] = __uint_as_float(raw.x << 16); v[1] = __uint_as_float(raw.x & 0xFFFF0000u);
  v[2] = __uint_as_float(raw.y << 16); v[3] = __uint_as_float(raw.y & 0xFFFF0000u);
}
__device__ __forceinline__ void pack_load1(const PackParams& a, int64_t src, int k, bool live, uint32_t& word, uint32_t& s) {
  word = 0;
  s = 127;
  if (live) {
    word = *reinterpret_cast<const uint32_t*>((const uint8_t*)a.x + src * a.ld_x + k);
    if (a.x_scale) s = a.x_scale[src * a.ld_xs + (k >> 5)];
  }
}
struct TwoTerms { uint32_t hi, lo, s_hi, s_lo; };
__device__ __forceinline__ void pack_two_terms(const float (&v)[4], TwoTerms& q) {
  float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
#pragma unroll
  for (int o = 1; o <= 4; o <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, o));
  if (!(amax < 3.0e38f)) amax = 3.0e38f;          // Inf / NaN in the group: keep the scale finite
  float s_hi, i_hi;
  mx8_scale(amax, q.s_hi, s_hi, i_hi);
  const uint32_t h01 = f32x2_to_e4m3x2(v[0] * i_hi, v[1] * i_hi), h23 = f32x2_to_e4m3x2(v[2] * i_hi, v[3] * i_hi);
  const float2 f01 = e4m3x2_to_f32x2(h01), f23 = e4m3x2_to_f32x2(h23);
  float rs[4] = {left_over(v[0], f01.x, s_hi), left_over(v[1], f01.y, s_hi), left_over(v[2], f23.x, s_hi), left_over(v[3], f23.y, s_hi)};
  float rmax = fmaxf(fmaxf(fabsf(rs[0]), fabsf(rs[1])), fmaxf(fabsf(rs[2]), fabsf(rs[3])));
#pragma unroll
  for (int o = 1; o <= 4; o <<= 1) rmax = fmaxf(rmax, __shfl_xor_sync(0xFFFFFFFFu, rmax, o));
  if (!(rmax < 3.0e38f)) rmax = 0.0f;
  float s_lo, i_lo;
  mx8_scale(rmax, q.s_lo, s_lo, i_lo);
  const uint32_t l01 = f32x2_to_e4m3x2(rs[0] * i_lo, rs[1] * i_lo), l23 = f32x2_to_e4m3x2(rs[2] * i_lo, rs[3] * i_lo);
  q.hi = h01 | (h23 << 16);
  q.lo = l01 | (l23 << 16);
}
// a lane's four e4m3 codes in line `line` of a chunk of `lines` lines, and its group's scale
__device__ __forceinline__ void pack_store8(uint8_t* chunk, int lines, int line, uint32_t g, int lane, uint32_t codes, uint32_t s) {
  const uint32_t piece = (uint32_t)(lane >> 2), within = (uint32_t)(lane & 3) * 4u;
  *reinterpret_cast<uint32_t*>(chunk + line * 128 + ((piece ^ (uint32_t)(line & 7)) << 4) + within) = codes;
  if ((lane & 7) == 0) chunk[lines * 128 + (line & 31) * 16 + (line >> 5) * 4 + g] = (uint8_t)s;
}

template <bool SPLIT>
__global__ void __launch_bounds__(256) mx_pack_x_kernel(const GemmParams p, const PackParams a) {
  pdl_begin();
  const int64_t slot = blockIdx.x;
  const int kt = blockIdx.y;
  int e; int64_t row0; int rows;
  if (!mx_map_block(p, a.tb, slot, e, row0, rows)) return;
  uint8_t* chunk = a.out + (slot * a.KT + kt) * a.chunk_bytes;
  const int lines = !SPLIT ? a.n_mma : a.fit ? chunk_lines(rows) : a.tb;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k = kt * 128 + lane * 4;
  const uint32_t g = (uint32_t)(lane >> 3);
  for (int r = warp; r < rows; r += 8) {
    const int64_t m = row0 + r;
    int64_t src = a.gather ? (int64_t)a.gather[m] : m;
    if (src >= a.rows_x) src = -1;
    const bool live = src >= 0 && k < a.K;        // K % 32 == 0: a lane's four values are in or out together
    if constexpr (SPLIT) {
      float v[4];
      pack_load4(a, src, k, live, v);
      TwoTerms q;
      pack_two_terms(v, q);
      pack_store8(chunk, 2 * lines, r, g, lane, q.hi, q.s_hi);
      pack_store8(chunk, 2 * lines, lines + r, g, lane, q.lo, q.s_lo);
    } else {
      uint32_t word, s;
      pack_load1(a, src, k, live, word, s);
      pack_store8(chunk, lines, r, g, lane, word, s);
    }
  }
}

// ---- four e2m1 terms -----------------------------------------------------------------------------------------
// Chunk of the four-term form: line r (r < 4 tb; term t of token j is line t * tb + j) is 64 bytes = 128 e2m1 values, low
// nibble first, its 16-byte pieces XOR-swizzled with ((r >> 1) & 3) like a 64-byte-swizzled TMA tile; scales as above.
// Two values at a time by the conversion instructions (round to nearest, ties to the even code; |q| <= 6 but for Inf, which
// saturates): with compares and selects per value, and a warp reduction under four masks, the pack of 64 tokens for 128 experts
// took 13.6-14.4 us, so 10.5-11.1.
__device__ __forceinline__ uint32_t group_max_bits(uint32_t top) {        // over the 8 lanes that hold a group
#pragma unroll
  for (int o = 1; o <= 4; o <<= 1) top = max(top, __shfl_xor_sync(0xFFFFFFFFu, top, o));
  return top;
}
// a lane's four e2m1 codes in line `line` of a chunk of `lines` lines, and its group's scale
__device__ __forceinline__ void pack_store4(uint8_t* chunk, int lines, int line, uint32_t g, int lane, uint32_t codes, uint32_t sb) {
  *reinterpret_cast<uint16_t*>(chunk + line * 64 + ((g ^ (uint32_t)((line >> 1) & 3)) << 4) + (uint32_t)(lane & 7) * 2u) = (uint16_t)codes;      // a 32-group is one 16-byte piece
  if ((lane & 7) == 0) chunk[lines * 64 + (line & 31) * 16 + (line >> 5) * 4 + (int)g] = (uint8_t)sb;
}
// The pass by position, a warp a row at a time.
// (16 warps over the rows of eight k steps, for a third of the blocks: 2.6 x slower at 64 tokens, the blocks of 16 rows decide;
// four warps instead of eight: 8 % slower.)  (A warp per (token block, k step, four rows) with the rows' chains side by side, and dead warps grouped into whole
// CTAs, was tried in place of the loop over rows below: 2.3 x slower.  A row's four-term chain is latency, and four of
// them in one warp add up where eight warps of a CTA overlap them.)
__global__ void __launch_bounds__(256) mx_pack_x4_kernel(const GemmParams p, const PackParams a) {
  pdl_begin();
  const int64_t slot = blockIdx.x;
  const int kt = blockIdx.y;
  int e; int64_t row0; int rows;
  if (!mx_map_block(p, a.tb, slot, e, row0, rows)) return;
  uint8_t* chunk = a.out + (slot * a.KT + kt) * a.chunk_bytes;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k = kt * 128 + lane * 4;
  const uint32_t g = (uint32_t)(lane >> 3);
  for (int r = warp; r < rows; r += 8) {
    const int64_t m = row0 + r;
    int64_t src = a.gather ? (int64_t)a.gather[m] : m;
    if (src >= a.rows_x) src = -1;
    float v[4];
    pack_load4(a, src, k, src >= 0 && k < a.K, v);
    const bool nan[4] = {v[0] != v[0], v[1] != v[1], v[2] != v[2], v[3] != v[3]};      // e2m1 has no NaN: such a value counts as 0
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      uint32_t codes;
      const uint32_t sb = e2m1_term(t, v, nan, codes, group_max_bits);
      pack_store4(chunk, a.n_mma, t * a.tb + r, g, lane, codes, sb);
    }
  }
}

// The same with the tokens of x in turn, given the positions of every one (positions, experts: k per token): a warp takes a token's k step,
// quantises it once and writes its lines for each of the k positions.  The pass is a chain of latencies: by position it runs a block
// for every (token block, k step) the schedule may hold, most of them without rows, and a warp's rows follow one another.  64 tokens of 128
// experts 7.2 -> 4.0 us of a step, 300 tokens 10.3 -> 5.1; steps of 64 tokens of 128 and 32 experts 159.2 -> 155.3 and 100.5 -> 97.9.
struct PackRows {
  const int32_t* positions; const int16_t* experts;      // [rows_x, k]
  int k;
};
// chunk (at its k step) and lines of a term of pick `at` of [rows_x, k], and the row in its block; no chunk where the pick is not a row of
// one of the experts (dropped ones are -1)
struct PickChunk { uint8_t* chunk; int r, lines; };
__device__ __forceinline__ PickChunk pick_chunk(const GemmParams& p, const PackParams& a, const PackRows& w, int64_t at, int kt, bool split) {
  // (the loads side by side: with the block's behind the check a step of 4 tokens of 8 experts took 0.4 us longer)
  const int pick = w.experts[at], m = w.positions[at], e = (unsigned)pick < (unsigned)p.E ? pick : 0;
  const int rows = p.slice_sizes[e], off = p.slice_offs[e], first = p.block_offs[e];
  const int rr = m - off, j = rr / a.tb;
  PickChunk c;
  c.r = rr - j * a.tb;
  c.lines = !split ? a.n_mma : a.fit ? chunk_lines(min(a.tb, rows - j * a.tb)) : a.tb;
  uint8_t* chunk = a.out + ((int64_t)(first + j) * a.KT + kt) * a.chunk_bytes;
  c.chunk = e == pick && rr >= 0 && rr < rows ? chunk : nullptr;
  return c;
}
// `store`(chunk, r, lines) for each pick of token t that has a chunk, by the whole warp
template <typename F>
__device__ __forceinline__ void each_pick(const GemmParams& p, const PackParams& a, const PackRows& w, int64_t t, int kt, bool split, F store) {
  const int lane = threadIdx.x & 31;
  for (int j0 = 0; j0 < w.k; j0 += 32) {
    PickChunk own{nullptr, 0, 0};
    if (j0 + lane < w.k) own = pick_chunk(p, a, w, t * w.k + j0 + lane, kt, split);
    for (int j = 0; j < min(32, w.k - j0); ++j) {
      uint8_t* chunk = (uint8_t*)__shfl_sync(0xFFFFFFFFu, (unsigned long long)own.chunk, j);
      const int r = __shfl_sync(0xFFFFFFFFu, own.r, j), lines = __shfl_sync(0xFFFFFFFFu, own.lines, j);
      if (chunk) store(chunk, r, lines);
    }
  }
}
// FORM: terms of a token
template <int FORM>
__global__ void __launch_bounds__(256) mx_pack_rows_kernel(const GemmParams p, const PackParams a, const PackRows w) {
  pdl_begin();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t unit = (int64_t)blockIdx.x * 8 + warp, t = unit / a.KT;
  if (t >= a.rows_x) return;
  const int kt = (int)(unit - t * a.KT), k = kt * 128 + lane * 4;
  const bool live = k < a.K;
  const uint32_t g = (uint32_t)(lane >> 3);
  if constexpr (FORM == 4) {
    float v[4];
    pack_load4(a, t, k, live, v);
    const bool nan[4] = {v[0] != v[0], v[1] != v[1], v[2] != v[2], v[3] != v[3]};
    uint32_t codes[4], sb[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) sb[i] = e2m1_term(i, v, nan, codes[i], group_max_bits);
    each_pick(p, a, w, t, kt, true, [&](uint8_t* chunk, int r, int lines) {
#pragma unroll
      for (int i = 0; i < 4; ++i) pack_store4(chunk, a.n_mma, i * lines + r, g, lane, codes[i], sb[i]);
    });
  } else if constexpr (FORM == 2) {
    float v[4];
    pack_load4(a, t, k, live, v);
    TwoTerms q;
    pack_two_terms(v, q);
    each_pick(p, a, w, t, kt, true, [&](uint8_t* chunk, int r, int lines) {
      pack_store8(chunk, 2 * lines, r, g, lane, q.hi, q.s_hi);
      pack_store8(chunk, 2 * lines, lines + r, g, lane, q.lo, q.s_lo);
    });
  } else {
    uint32_t word, s;
    pack_load1(a, t, k, live, word, s);
    each_pick(p, a, w, t, kt, false, [&](uint8_t* chunk, int r, int lines) { pack_store8(chunk, lines, r, g, lane, word, s); });
  }
}

// ============================================================================================================
// PTX pieces of the block-scaled path
// ============================================================================================================
// instruction descriptor of kind::mxf8f6f4: A = e2m1 (code 5), B = e4m3 (code 0), both K-major, e8m0 scales,
// M = 128, N = n; sf selects the byte (k group) of the scale words for A and B
__device__ __forceinline__ uint32_t mx_idesc(int n, uint32_t sf) {
  return (sf << 4) | (5u << 7) | (0u << 10) | ((uint32_t)(n >> 3) << 17) | (1u << 23) | (1u << 27) | (sf << 29);
}
// kind::mxf4: A and B e2m1 (code 1), packed, K-major, K = 64; sf selects the byte PAIR (0 or 2) of the scale words
__device__ __forceinline__ uint32_t mx4_idesc(int n, uint32_t sf) {
  return (sf << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | (1u << 23) | (1u << 27) | (sf << 29);
}
// One block-scaled MMA of either kind, issued by an elected lane while the whole warp runs the loop: the
// operands of tcgen05.mma live in uniform registers, and computed by a single thread of a divergent branch each of them took a
// move from a vector register first (87-95 cycles per instruction; a block-scaled MMA of up to 64 columns runs 45).  Of a
// shared-memory descriptor only the low word varies.
constexpr uint32_t MX_DESC_LO = 1u << 16;                                              // leading byte offset (unused)
constexpr uint32_t MX_DESC_HI_SW128 = (1024u >> 4) | (1u << 14) | (2u << 29);          // 8-row groups 1024 B apart, 128-byte swizzle
constexpr uint32_t MX_DESC_HI_SW64 = (512u >> 4) | (1u << 14) | (4u << 29);            // 64-byte rows and swizzle
template <bool F4>
__device__ __forceinline__ void mma_mx(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t sfa, uint32_t sfb,
                                       uint32_t accumulate) {
  if constexpr (F4)
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %7};\n\tmov.b64 db, {%2, %7};\n\t"
        "setp.ne.b32 p, %6, 0;\n\telect.sync _|q, 0xFFFFFFFF;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], da, db, %3, [%4], [%5], p;\n\t}" ::"r"(d_tmem),
        "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(sfa), "r"(sfb), "r"(accumulate), "n"(MX_DESC_HI_SW64)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %7};\n\tmov.b64 db, {%2, %7};\n\t"
        "setp.ne.b32 p, %6, 0;\n\telect.sync _|q, 0xFFFFFFFF;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale.scale_vec::1X [%0], da, db, %3, [%4], [%5], p;\n\t}" ::"r"(d_tmem),
        "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(sfa), "r"(sfb), "r"(accumulate), "n"(MX_DESC_HI_SW128)
        : "memory");
}

// Asks L2 for the weights of this CTA's first stages (a warp, ahead of its wait for the kernel before, whose CTA on this SM may have left
// long before its last one does).  Decode of one token 38.2 -> 36.9 us per step, 16 tokens of 32 experts 70.8 -> 68.1.  (With the
// metadata read ahead of the wait for good, and the first weights loaded into shared memory there: 34.8 and 64.3, but
// only the wait makes visible what the stream's kernels wrote, those further back included.)
template <int NACC>
__device__ __forceinline__ void mx_hint_weights(const GemmParams& p, const MxParams& q, int narrow_steps, int lane) {
  const int KT = q.KT, NB = q.NB;
  uint32_t useful_m = (uint32_t)q.grid_m;
  if (p.slice_sizes) useful_m = min((uint32_t)ld_hint(p.block_offs + p.E), q.hint_m);
  MxSched sched(useful_m, NB, NACC);
  int64_t pid_m;
  int nb0, mb_live;
  if (!sched.next(pid_m, nb0, mb_live)) return;
  const int e = p.slice_sizes ? ld_hint(p.block_sched + pid_m) & 0xFFFF : 0;
  if (e >= p.E) return;
  const int steps = min(KT, q.stages * (NACC == 1 || sched.narrow ? narrow_steps : 1));
  for (int kt = lane; kt < steps; kt += 32) {
    const int64_t tile = ((int64_t)e * KT + kt) * NB + nb0;
    l2_hint((const uint8_t*)p.w + tile * MX_W_TILE_TX, (uint32_t)(mb_live * MX_W_TILE_TX));
    l2_hint(p.w_scale + tile * MX_WS_TILE, (uint32_t)(mb_live * MX_WS_TILE));
  }
}

// sums of N tokens over their terms, smallest first
__device__ __forceinline__ void tmem_ld_n(uint32_t taddr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld_n(uint32_t taddr, uint32_t (&r)[16]) { tmem_ld16(taddr, r); }
template <bool F4, int N>
__device__ __forceinline__ void mx_sums(uint32_t taddr, int split, int lines, uint32_t (&sum)[N]) {
  uint32_t t1[N], t2[N], t3[N];
  tmem_ld_n(taddr, sum);
  if (split > 1) tmem_ld_n(taddr + (uint32_t)lines, t1);
  if constexpr (F4) {
    tmem_ld_n(taddr + 2u * (uint32_t)lines, t2);
    tmem_ld_n(taddr + 3u * (uint32_t)lines, t3);
  }
  tmem_ld_wait();
#pragma unroll
  for (int j = 0; j < N; ++j) {
    float a = __uint_as_float(sum[j]), b = split > 1 ? __uint_as_float(t1[j]) : 0.0f;
    if constexpr (F4) {
      a += __uint_as_float(t3[j]);
      b += __uint_as_float(t2[j]);
    }
    if (split > 1) a += b;
    sum[j] = __float_as_uint(a);
  }
}

// ============================================================================================================
// The GEMM kernel
// ============================================================================================================
// F4: the four-term form (packed operands, kind::mxf4); otherwise byte-per-element operands, kind::mxf8f6f4
// KM (four-term form, MB = 3): the three weight tiles of a stage are three consecutive K STEPS of ONE weight block instead of
// one k step of three blocks -- for steps with so few tiles that a CTA gets single weight blocks (one to four tokens: 60
// to 165 three-block tiles for 148 SMs).  A stage of one 8 KB tile cannot keep a per-SM copy pipeline busy (a ring of
// 8 KB stages streams 3.3 TB/s over the GPU however many are in flight, 24 KB stages 7.1 TB/s).
// FIT (two-term form, MB = 2 or 3): a tile copies and multiplies, of a token block, what its rows need (16, 32 or 64 lines a term): 300 tokens of
// 128 experts 303.6 -> 287.6 us per step.  With four terms (8 or 16 lines) or single blocks it costs a tile's start more than it saves (16
// tokens 62.3 -> 63.9), and e4m3 tokens pay 5 % for the code alone.
template <typename TY, int MB, bool F4, bool KM = false, bool FIT = false>
__global__ void __launch_bounds__(MX_THREADS, 1)
gemm_mx_kernel(const GemmParams p, const MxParams q, const __grid_constant__ MxMaps w_maps) {
  static_assert(!KM || (F4 && MB == 3), "the k-step form is built for the four-term kernel with three tiles per stage");
  constexpr uint32_t W_TILE = F4 ? MX_W_TILE_TX : MX_W_TILE;       // bytes of a weight block in shared memory
  constexpr uint32_t X_ROW = F4 ? 64u : 128u;                      // bytes of a token row of a k step
  constexpr int NACC = KM ? 1 : MB;                                // accumulators (weight blocks) of a tile
  constexpr int SF_COLS = KM ? 24 : MX_SF_COLS;                    // scale columns of a stage: KM has three token chunks
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sbase = smem_u32(smem);
  const int warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;     // warp-uniform for the compiler
  const int STAGES = q.stages;
  // per stage: [MB weight tiles][token rows + 1024 B scale area (KM: three such chunks)][MB x 512 B weight scales]
  // where the k steps of a stage follow one another, S > 1: [S weight tiles][S such chunks][S x 512 B]
  auto off_x = [&](int S) { return (uint32_t)(S > 1 ? S : MB) * W_TILE; };
  auto off_ws = [&](int S) { return off_x(S) + (S > 1 ? (uint32_t)S * (uint32_t)q.chunk_bytes : (uint32_t)q.n_mma * X_ROW + 1024u); };
  const uint32_t SF_BASE = KM ? 512u - (uint32_t)(MX_MAX_STAGES > 5 ? 5 : MX_MAX_STAGES) * 24u : (uint32_t)MX_SF_BASE;
  const uint32_t ctl0 = sbase + (uint32_t)STAGES * (uint32_t)q.stage_bytes;
  auto BAR_FULL = [&](int s) { return ctl0 + 8u * (uint32_t)s; };
  auto BAR_EMPTY = [&](int s) { return ctl0 + 8u * (uint32_t)(MX_MAX_STAGES + s); };
  auto BAR_SF = [&](int s) { return ctl0 + 8u * (uint32_t)(2 * MX_MAX_STAGES + s); };      // scales are in tensor memory
  auto BAR_ACC_FULL = [&](int a) { return ctl0 + 8u * (uint32_t)(3 * MX_MAX_STAGES + a); };
  auto BAR_ACC_EMPTY = [&](int a) { return ctl0 + 8u * (uint32_t)(3 * MX_MAX_STAGES + 2 + a); };
  const uint32_t BAR_DRAIN = ctl0 + 8u * (uint32_t)(3 * MX_MAX_STAGES + 4);
  uint8_t* ctl_ptr = smem + (size_t)STAGES * (size_t)q.stage_bytes;
  volatile uint32_t* s_tmem = reinterpret_cast<volatile uint32_t*>(ctl_ptr + MX_CTL_BARS * 8);
  volatile int* s_abort = reinterpret_cast<volatile int*>(ctl_ptr + MX_CTL_BARS * 8 + 4);
  volatile int* s_cols = reinterpret_cast<volatile int*>(ctl_ptr + MX_CTL_BARS * 8 + 16);      // per stage
  Ctl ctl{s_abort, p.status};

  if (threadIdx.x == 0) {
    for (int s = 0; s < MX_MAX_STAGES; ++s) {
      mbar_init(BAR_FULL(s), 1);
      mbar_init(BAR_EMPTY(s), 1);
      mbar_init(BAR_SF(s), 4);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(BAR_ACC_FULL(a), 1);
      mbar_init(BAR_ACC_EMPTY(a), 4);
    }
    mbar_init(BAR_DRAIN, 1);
    *s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)s_tmem)),
                 "r"((uint32_t)TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xFFFFFFFFu, *s_tmem, 0);

  // (a scale loader: it waits longest for its first work)
  if (warp == MX_THREADS / 32 - 1) mx_hint_weights<NACC>(p, q, KM ? 3 : NACC == 3 ? 2 : 1, lane);
  pdl_begin();
  const int KT = q.KT, NB = q.NB;
  uint32_t useful_m = (uint32_t)q.grid_m;
  if (p.slice_sizes) useful_m = (uint32_t)__shfl_sync(0xFFFFFFFFu, p.block_offs[p.E], 0);
  const int acc_stride = NACC * q.n_mma;            // accumulator columns of one buffer
  MxSched sched(useful_m, NB, NACC);
  int64_t pid_m;
  int nb0, mb_live;
  // k steps of a stage of the current tile, as a constant of the role's loop (a loop for either form: with the choice inside, the
  // issuing warps took 2-5 us longer over a product of 50)
  auto with_steps = [&](auto&& loop) {
    if constexpr (KM) loop(std::integral_constant<int, 3>());
    else if (MB == 3 && sched.narrow) loop(std::integral_constant<int, 2>());
    else loop(std::integral_constant<int, 1>());
  };

  if (warp == 0) {
    // ================================= producer =======================================================
    uint32_t s = 0, ph = 1, issued = 0;
    bool ok = true;
    uint64_t policy;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
    auto weights = [&](uint32_t st, uint32_t ws, const CUtensorMap* w_map, int tile, uint32_t scales, uint32_t bar) {
      const uint8_t* from = p.w_scale + (int64_t)tile * MX_WS_TILE;
      if (KM || q.once) {
        elect_tile_3d_hint(st, w_map, 0, 0, tile, bar, policy);
        elect_bulk_g2s_hint(ws, from, scales, bar, policy);
      } else {
        elect_tile_3d(st, w_map, 0, 0, tile, bar);
        elect_bulk_g2s(ws, from, scales, bar);
      }
    };
    while (ok && sched.next(pid_m, nb0, mb_live)) {
      int e; int64_t row0; int rows;
      mx_map_block(p, q.tb, pid_m, e, row0, rows);
      // columns of the tile and bytes of a chunk: what its rows need
      int cols = q.n_mma;
      if (FIT) cols = 2 * chunk_lines(__shfl_sync(0xFFFFFFFFu, rows, 0));
      const uint32_t chunk = (uint32_t)q.chunk_bytes, live = FIT ? (uint32_t)cols * X_ROW + 512u : chunk;
      const uint8_t* xsrc = q.xq + pid_m * KT * chunk;
      int tile = __shfl_sync(0xFFFFFFFFu, e, 0) * KT * NB + nb0;             // weight tile of the stage's first k step
      with_steps([&](auto steps) {
        constexpr int S = decltype(steps)::value;
        const int stages = (KT + S - 1) / S;
        const CUtensorMap* w_map = &w_maps.m[S > 1 ? 0 : mb_live - 1];
        for (int kt = 0; kt < stages; ++kt, ++issued) {
          const uint32_t st = sbase + s * (uint32_t)q.stage_bytes, bar = BAR_FULL(s);
          ok = __all_sync(0xFFFFFFFFu, mbar_wait(BAR_EMPTY(s), ph, ctl, 601));
          if (!ok) break;
          if (FIT && kt == 0) {                        // (the arrival below publishes it)
            if (lane == 0) s_cols[s] = cols;
            __syncwarp();
          }
          const int k_live = S > 1 ? min(S, KT - S * kt) : 1;
          if constexpr (S > 1) {
            elect_expect_tx(bar, (uint32_t)k_live * ((uint32_t)(MX_W_TILE_TX + MX_WS_TILE) + live));
            for (int i = 0; i < k_live; ++i, tile += NB) {
              weights(st + (uint32_t)i * W_TILE, st + off_ws(S) + (uint32_t)i * MX_WS_TILE, w_map, tile, (uint32_t)MX_WS_TILE, bar);
            }
          } else {
            elect_expect_tx(bar, (uint32_t)(mb_live * (MX_W_TILE_TX + MX_WS_TILE)) + live);
            weights(st, st + off_ws(1), w_map, tile, (uint32_t)(mb_live * MX_WS_TILE), bar);
            tile += NB;
          }
          if (S == 1 || !FIT) {
            elect_bulk_g2s(st + off_x(S), xsrc, (uint32_t)k_live * live, bar);
            xsrc += (uint32_t)k_live * chunk;
          } else {
            for (int i = 0; i < k_live; ++i, xsrc += chunk) elect_bulk_g2s(st + off_x(S) + (uint32_t)i * chunk, xsrc, live, bar);
          }
          if (++s == (uint32_t)STAGES) { s = 0; ph ^= 1u; }
        }
      });
    }
    if (!ok && lane == 0) {
      // aborting: let the copies that were already issued land before the CTA leaves
      for (uint32_t j = issued > (uint32_t)STAGES ? issued - STAGES : 0; j < issued; ++j)
        for (uint32_t i = 0; i < (1u << 16) && !mbar_test(BAR_FULL(j % STAGES), (j / STAGES) & 1u); ++i) __nanosleep(64);
    }
    __syncwarp();
  } else if (warp == 1) {
    // ================================= MMA issuer =====================================================
    uint32_t idesc = F4 ? mx4_idesc(q.n_mma, 0) : mx_idesc(q.n_mma, 0);
    uint32_t s = 0, ph = 0, tc = 0;                    // stage and parity of the next k step
    bool ok = true, ready = false;                     // ready: the next step was complete when the last one was issued
    for (; ok && sched.next(pid_m, nb0, mb_live); ++tc) {
      const uint32_t ab = tc % (uint32_t)q.acc_bufs;
      ok = __all_sync(0xFFFFFFFFu, mbar_wait(BAR_ACC_EMPTY(ab), ((tc / (uint32_t)q.acc_bufs) & 1u) ^ 1u, ctl, 603));
      if (!ok) break;
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + ab * (uint32_t)acc_stride;
      with_steps([&](auto steps) {
        constexpr int S = decltype(steps)::value;
        constexpr int KK = F4 ? 2 : 4;
        constexpr uint32_t SFK = F4 ? (2u << 4) + (2u << 29) : (1u << 4) + (1u << 29);         // next scale byte (pair)
        const int stages = (KT + S - 1) / S;
        for (int kt = 0; kt < stages; ++kt) {
          // (the scale loaders have seen the stage's copies land)
          if (!__all_sync(0xFFFFFFFFu, ready)) ok = __all_sync(0xFFFFFFFFu, mbar_wait(BAR_SF(s), ph, ctl, 602));
          if (!ok) break;
          tc_fence_after();
          if (FIT && kt == 0) idesc = mx_idesc(__shfl_sync(0xFFFFFFFFu, s_cols[s], 0), 0);
          const uint32_t st = sbase + s * (uint32_t)q.stage_bytes;
          const uint32_t sf = tmem_base + SF_BASE + s * SF_COLS;
          const uint32_t a_lo = MX_DESC_LO | (st >> 4), b_lo = MX_DESC_LO | ((st + off_x(S)) >> 4);
          const uint32_t more = (uint32_t)(kt > 0);
          // k group outermost: consecutive MMAs go to different accumulators
          if constexpr (S > 1) {
            const uint32_t bstep = (uint32_t)q.chunk_bytes >> 4;
            const int k_live = min(S, KT - S * kt);
#pragma unroll
            for (int i = 0; i < S; ++i) {
              if (i < k_live) {
#pragma unroll
                for (int kk = 0; kk < KK; ++kk)
                  mma_mx<F4>(d_tmem, a_lo + i * (W_TILE >> 4) + kk * 2, b_lo + i * bstep + kk * 2, idesc + kk * SFK, sf + 4 * i, sf + 4 * S + 4 * i,
                             (i | kk) ? 1u : more);
              }
            }
          } else if (mb_live == MB) {
#pragma unroll
            for (int kk = 0; kk < KK; ++kk)
#pragma unroll
              for (int mb = 0; mb < MB; ++mb)
                mma_mx<F4>(d_tmem + (uint32_t)(mb * q.n_mma), a_lo + mb * (W_TILE >> 4) + kk * 2, b_lo + kk * 2, idesc + kk * SFK, sf + 4 * mb,
                           sf + 4 * MB, kk ? 1u : more);
          } else {
#pragma unroll
            for (int kk = 0; kk < KK; ++kk)
#pragma unroll
              for (int mb = 0; mb < MB; ++mb)
                if (mb < mb_live)
                  mma_mx<F4>(d_tmem + (uint32_t)(mb * q.n_mma), a_lo + mb * (W_TILE >> 4) + kk * 2, b_lo + kk * 2, idesc + kk * SFK, sf + 4 * mb,
                             sf + 4 * MB, kk ? 1u : more);
          }
          elect_commit(BAR_EMPTY(s));
          if (++s == (uint32_t)STAGES) { s = 0; ph ^= 1u; }
          ready = mbar_test(BAR_SF(s), ph);
        }
      });
      if (ok) elect_commit(BAR_ACC_FULL(ab));
    }
    // every MMA issued by this warp has retired before tensor memory is freed
    elect_commit(BAR_DRAIN);
    mbar_wait(BAR_DRAIN, 0, ctl, 605);
    __syncwarp();
  } else if (warp >= 6) {
    // ================================= scale loaders ==================================================
    // The scales of a stage go from shared to tensor memory through registers (tcgen05.st), one warp per lane quarter:
    // lane l of every quarter holds the 16 bytes of row l of each 512-byte scale block (the MB weight blocks, then the
    // tokens), i.e. the four columns the MMA reads for rows l, l + 32, l + 64, l + 96.  This keeps the copies out of
    // the in-order queue of the tensor pipe, where a tcgen05.cp ahead of every k step cost about a third of the step.
    const int qd = warp & 3;
    uint32_t it = 0;
    bool ok = true;
    while (ok && sched.next(pid_m, nb0, mb_live)) {
      with_steps([&](auto steps) {
        constexpr int S = decltype(steps)::value;
        const int stages = (KT + S - 1) / S;
        uint32_t scales_at = (uint32_t)q.n_mma * X_ROW;      // of a chunk's scales
        for (int kt = 0; kt < stages; ++kt, ++it) {
          const int s = it % STAGES;
          ok = __all_sync(0xFFFFFFFFu, mbar_wait(BAR_FULL(s), (it / STAGES) & 1u, ctl, 607));
          if (!ok) break;
          const uint32_t st = sbase + (uint32_t)s * (uint32_t)q.stage_bytes;
          const uint32_t taddr = tmem_base + ((uint32_t)(qd * 32) << 16) + SF_BASE + (uint32_t)(s * SF_COLS);
          if (FIT && kt == 0) scales_at = (uint32_t)s_cols[s] * X_ROW;
          // S > 1: the weight scales of the k steps, then the token scales of their chunks
          constexpr int LOADS = S > 1 ? 2 * S : MB + 1, NV = LOADS == 3 ? 4 : LOADS;
          const int live = S > 1 ? min(S, KT - S * kt) : mb_live;
          uint4 v[NV];
#pragma unroll
          for (int i = 0; i < NV; ++i) {
            const int j = S > 1 && i >= S ? i - S : i;
            uint32_t at = st + off_ws(S) + (uint32_t)j * MX_WS_TILE;
            if (S > 1 ? i >= S : i == MB) at = st + off_x(S) + (S > 1 ? (uint32_t)j * (uint32_t)q.chunk_bytes : 0u) + scales_at;
            v[i] = (i < LOADS && j < live) || (S == 1 && i == MB) ? lds128(at + (uint32_t)lane * 16u) : make_uint4(0, 0, 0, 0);
          }
          if constexpr (NV >= 4)
            asm volatile(
                "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
                "r"(v[0].x), "r"(v[0].y), "r"(v[0].z), "r"(v[0].w), "r"(v[1].x), "r"(v[1].y), "r"(v[1].z), "r"(v[1].w),
                "r"(v[2].x), "r"(v[2].y), "r"(v[2].z), "r"(v[2].w), "r"(v[3].x), "r"(v[3].y), "r"(v[3].z), "r"(v[3].w)
                : "memory");
          if constexpr (NV != 4) {
            constexpr int I = NV == 2 ? 0 : 4;
            asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr + 4u * I), "r"(v[I].x),
                         "r"(v[I].y), "r"(v[I].z), "r"(v[I].w), "r"(v[I + 1].x), "r"(v[I + 1].y), "r"(v[I + 1].z), "r"(v[I + 1].w)
                         : "memory");
          }
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(BAR_SF(s));
        }
      });
    }
  } else {
    // ================================= epilogue =======================================================
    // Accumulator [weight row = lane][token = column]: lane l of the warp that owns lane quarter qd holds output
    // column n = n0 + 128 mb + 32 qd + l.  Token parameters sit one token per lane and are broadcast by shuffle; for
    // SwiGLU the even lane holds the gate and the odd lane the linear half of a pair.
    const int qd = warp & 3;
    const bool swiglu = p.activation == MOE_ACT_SWIGLU;
    constexpr int TG = F4 ? 4 : 16;                    // tokens at a time: a four-term block has few
    const int half = qd >> 1;
    const TokStage tok{ctl0 + MX_CTL_BYTES + (uint32_t)(half * 3 * TOK_STAGE), 1 + half, (qd & 1) * 32 + lane};
    uint32_t tc = 0;
    bool ok = true;
    for (; ok && sched.next(pid_m, nb0, mb_live); ++tc) {
      int e; int64_t row0; int rows;
      mx_map_block(p, q.tb, pid_m, e, row0, rows);
      const uint32_t ab = tc % (uint32_t)q.acc_bufs;
      float bias_n[NACC];
#pragma unroll
      for (int mb = 0; mb < NACC; ++mb) {
        const int n = (nb0 + mb) * 128 + qd * 32 + lane;
        bias_n[mb] = (p.bias && n < p.N) ? load_bias(p.bias, p.bias_dtype, (int64_t)e * p.ld_bias + n) : 0.0f;
      }
      auto bias_of = [&](int mb) {                     // (selects: an index into registers would put them into memory)
        float b = bias_n[0];
#pragma unroll
        for (int i = 1; i < NACC; ++i) b = mb == i ? bias_n[i] : b;
        return b;
      };
      const int lines = FIT ? chunk_lines(rows) : q.tb;
      int off = 0, size = 0, first_block = 0;
      if constexpr (TOK_TERMS<TY> != 0) {
        off = p.slice_offs[e];
        size = p.slice_sizes[e];
        if (q.out.tb) first_block = q.out.block_offs[e];
      }
      ok = __all_sync(0xFFFFFFFFu, mbar_wait(BAR_ACC_FULL(ab), (tc / (uint32_t)q.acc_bufs) & 1u, ctl, 604));
      if constexpr (TOK_TERMS<TY> != 0) ok = tok.all(ok);
      if (!ok) break;
      tc_fence_after();
      for (int c0 = 0; c0 < rows; c0 += 16) {
        if constexpr (TOK_TERMS<TY> != 0) {
          // the rows of the tile's groups into their stages, then the groups of all of them to the threads, four lanes each: with the few
          // rows that a decode block has, one turn for the three blocks
          const int jmax = min(16, rows - c0);
#pragma unroll 1
          for (int mb = 0; mb < mb_live; ++mb) {
            const float bias = bias_of(mb);
            const uint32_t taddr = tmem_base + ((uint32_t)(qd * 32) << 16) + ab * (uint32_t)acc_stride + (uint32_t)(mb * q.n_mma + c0);
#pragma unroll 1
            for (int j0 = 0; j0 < jmax; j0 += TG) {
              uint32_t sum[TG];
              float y[TG / 2];
              mx_sums<F4>(taddr + (uint32_t)j0, q.split, lines, sum);
              swiglu_chunk(p, sum, bias, lane & 1, y);
              stage_tokens<TY>(tok.at + (uint32_t)(mb * TOK_STAGE), y, j0 + TG / 2 * (lane & 1), ((qd & 1) << 4) + (lane >> 1));
            }
          }
          tok.sync();
          const int l4 = tok.i & 3;
#pragma unroll 1
          for (int t0 = 0; t0 < jmax * mb_live; t0 += 16) {
            const int t = t0 + (tok.i >> 2);
            int mb = 0, token = t;
            for (int i = 1; i < NACC; ++i)             // (t / jmax)
              if (token >= jmax) { ++mb; token -= jmax; }
            uint8_t *tq = nullptr, *ts = nullptr;
            if (t < jmax * mb_live) token_addr(q.out, e, off, size, first_block, (int)(row0 - off) + c0 + token, tq, ts);
            else mb = token = 0;
            emit_group<TY>(q.out, staged_row<TY>(tok.at + (uint32_t)(mb * TOK_STAGE), token, l4), l4, token & 7, 2 * (nb0 + mb) + half, tq, ts,
                           nb0 + mb == NB - 1 && 2 * NB + half < 4 * q.out.KT);
          }
          tok.sync();                                  // the stages may be written again
        } else {
          // parameters of token c0 + lane (lanes 0..15)
          const int tj = c0 + (lane & 15);
          TY* dst_l = nullptr;
          float beta_l = 1.0f, gamma_l = 1.0f;
          if (tj < rows) {
            const int64_t m = row0 + tj;
            const int64_t d = p.scatter_indx ? (int64_t)p.scatter_indx[m] : m;
            if (d >= 0) dst_l = gemm_out_row<TY>(p, d);
            if (p.betas) beta_l = p.betas[m];
            if (p.gammas) gamma_l = p.gammas[m];
          }
          const int jmax = min(16, rows - c0);
          // rolled: unrolled over the blocks and sixteen tokens the code of a launch's first pass through here came from memory line by
          // line (fc2 of 64 tokens and 128 experts 48 us, so 43.6)
#pragma unroll 1
          for (int mb = 0; mb < mb_live; ++mb) {
            const int n = (nb0 + mb) * 128 + qd * 32 + lane;
            const float bias = bias_of(mb);
            const uint32_t taddr = tmem_base + ((uint32_t)(qd * 32) << 16) + ab * (uint32_t)acc_stride + (uint32_t)(mb * q.n_mma + c0);
#pragma unroll 1
            for (int j0 = 0; j0 < jmax; j0 += TG) {
              uint32_t sum[TG];
              mx_sums<F4>(taddr + (uint32_t)j0, q.split, lines, sum);
#pragma unroll
              for (int j = 0; j < TG; ++j) {
                if (j0 + j < jmax) {                              // warp-uniform
                  TY* yrow = (TY*)__shfl_sync(0xFFFFFFFFu, (unsigned long long)dst_l, j0 + j);
                  const float beta = __shfl_sync(0xFFFFFFFFu, beta_l, j0 + j);
                  const float gamma = __shfl_sync(0xFFFFFFFFu, gamma_l, j0 + j);
                  float a = __uint_as_float(sum[j]);
                  a += bias * beta;
                  if (p.has_out_alpha) a *= p.out_alpha;
                  if (swiglu) {
                    const float other = __shfl_xor_sync(0xFFFFFFFFu, a, 1);
                    if (!(lane & 1) && yrow != nullptr && n + 1 < p.N)
                      yrow[n >> 1] = from_f32<TY>(gemm_swiglu(a, other, p.act_alpha, p.act_limit, p.act_has_limit) * gamma);
                  } else if (yrow != nullptr && n < p.N) {
                    yrow[n] = from_f32<TY>(a * gamma);
                  }
                }
              }
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(BAR_ACC_EMPTY(ab));
    }
  }

  // ---- teardown ----------------------------------------------------------------------------------------
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)TMEM_COLS)
                 : "memory");
  }
}

// ---- host side -----------------------------------------------------------------------------------------------
struct MxPlan {
  int tb, n_mma, split, f4, km, mb, KT, NB, n_groups, stages, stage_bytes, acc_bufs;
  int64_t grid_m, chunk_bytes, ws_bytes;
};

int64_t blocks_bound(int64_t n_slices, int64_t n_rows, int64_t block) {
  if (n_rows <= n_slices) return n_rows;
  const int64_t a = n_rows + 1 - n_slices;
  return n_slices - 1 + (a + block - 1) / block;
}

MxPlan mx_plan(const MoeGemmArgs& a) {
  MxPlan pl;
  const bool bf16 = a.x_dtype == MOE_BF16;
  const bool pin_f4 = bf16 && a.kernel == MOE_GEMM_MX_F4, pin_f8 = a.kernel == MOE_GEMM_MX_F8;
  const int tb_max = bf16 ? (pin_f4 ? 32 : 64) : 128;
  int tb = 16;
  if (a.tile_m == 16 || a.tile_m == 32 || a.tile_m == 64 || a.tile_m == 128) {
    tb = a.tile_m;
  } else {
    // 16 rows up to 8 rows per expert on average, 32 beyond (64-row blocks were slower than two 32-row blocks at every size
    // measured, with bf16 and with fp8 tokens: 32 experts, 8 rows, fp8: 102 us with 32-row blocks, 125 with 64, 153 with 128)
    const int64_t per = a.slice_sizes ? (a.M + a.E - 1) / a.E : a.M;      // mean rows per expert
    const int tb_auto = tb_max < 32 ? tb_max : 32;
    while (tb < tb_auto && tb < 2 * per) tb *= 2;
  }
  if (tb > tb_max) tb = tb_max;
  pl.tb = tb;
  // bf16 tokens: four e2m1 terms for the smallest blocks (weight streaming decides there), else two e4m3 terms
  pl.f4 = (bf16 && !pin_f8 && (pin_f4 || tb == 16)) ? 1 : 0;
  pl.split = bf16 ? (pl.f4 ? 4 : 2) : 1;
  pl.n_mma = pl.split > 1 ? pl.split * tb : (tb < 32 ? 32 : tb);     // a scale chunk serves 32 columns at a time
  pl.KT = (int)cdiv64(a.K, 128);
  pl.NB = (int)cdiv64(a.N, 128);
  pl.grid_m = a.slice_sizes ? blocks_bound(a.E, a.M, tb) : cdiv64(a.M, tb);
  // several weight blocks per CTA tile share one token tile (fewer token bytes per weight byte); one block when there
  // would be too few tiles to fill the SMs.  Three of packed weights; two where a value takes a byte of shared memory, of which the ring holds five stages
  // where it takes three of three: what bounds those forms is the weights in flight per SM, 82 KB against 74, less the stage at work.  us per step at
  // boost clocks and (second pair) in a long run under the power limit: bf16, 300 tokens of 128 experts 252 -> 243, 279 -> 278; 500 tokens 348 -> 314, 374 ->
  // 358; 150 tokens of 32 experts of 4096 x 4096 218 -> 202, 230 -> 223; e4m3, 100 tokens of 32 experts 107 -> 97, 103 -> 97.
  // (Over 1400 products of 1 to 19 rows per expert two are 4 % ahead with bf16 tokens and 2 % with e4m3; where rounds fall badly three are, by up to 10 %: 16 experts of
  // 4096 x 2048, 16 biased rows 37.7, 34.9, e4m3 tokens of 128 experts of 2880 x 5760, 6 biased rows 148, 139.  What an expert has is not known here.)
  const int wide = pl.f4 ? 3 : 2;
  // (Three of a byte per value are built for the constraint that asks for them alone.)
  pl.mb = a.tile_n == 128 ? 1 : a.tile_n == 384 ? 3 : a.tile_n == 256 && !pl.f4 ? 2 : pl.grid_m * cdiv64(pl.NB, wide) >= (int64_t)moe_sm_count() ? wide : 1;
  // too few tiles for three blocks each, four-term form: single weight blocks, three k steps of one block per stage
  // (a stage of one 8 KB tile does not keep a copy pipeline busy)
  pl.km = (pl.f4 && tb == 16 && pl.mb == 1 && a.tile_n == 0 && pl.KT >= 3) ? 1 : 0;
  pl.n_groups = (int)cdiv64(pl.NB, pl.mb);
  pl.chunk_bytes = (int64_t)pl.n_mma * (pl.f4 ? 64 : 128) + 1024;
  const int ctl_bytes = MX_CTL_BYTES;
  if (pl.km) {
    pl.mb = 3;                                       // tiles of a stage; n_groups stays the number of weight blocks
    pl.stage_bytes = 3 * MX_W_TILE_TX + 3 * (int)pl.chunk_bytes + 2048;
    int st = (MX_SMEM_LIMIT - 1024 - ctl_bytes) / pl.stage_bytes;
    pl.stages = st > 5 ? 5 : st;
    pl.acc_bufs = 2;
  } else {
    pl.stage_bytes = pl.mb * (pl.f4 ? MX_W_TILE_TX : MX_W_TILE) + (int)pl.chunk_bytes + 2048;
    int st = (MX_SMEM_LIMIT - 1024 - ctl_bytes) / pl.stage_bytes;
    pl.stages = st > MX_MAX_STAGES ? MX_MAX_STAGES : st;
    pl.acc_bufs = (2 * pl.mb * pl.n_mma <= MX_SF_BASE) ? 2 : 1;
  }
  pl.ws_bytes = pl.grid_m * pl.KT * pl.chunk_bytes;
  return pl;
}

template <typename TY, int MB, bool F4, bool KM = false, bool FIT = false>
int launch_mx(const GemmParams& p, MxParams q, const MxPlan& pl, const MxMaps& w_map, int idle_sms, cudaStream_t st) {
  const int room = MX_SMEM_LIMIT - 1024 - MX_CTL_BYTES - MX_TOK_BYTES<TY>;
  if (q.stages * q.stage_bytes > room) q.stages = room / q.stage_bytes;
  const int smem = q.stages * q.stage_bytes + MX_CTL_BYTES + MX_TOK_BYTES<TY> + 1024;
  const int64_t items = pl.grid_m * (KM ? pl.n_groups : pl.NB);        // blocks: the last round's are dealt out one by one
  int sms = moe_sm_count() - idle_sms;
  if (sms < 1) sms = 1;
  const int grid = (int)(items < sms ? items : sms);
  MOE_CHECK_CUDA(cudaFuncSetAttribute(gemm_mx_kernel<TY, MB, F4, KM, FIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  MOE_CHECK_CUDA(launch_pdl(gemm_mx_kernel<TY, MB, F4, KM, FIT>, dim3(grid), dim3(MX_THREADS), (size_t)smem, st, p, q, w_map));
  MOE_CHECK_LAUNCH();
  return MOE_OK;
}

// TY: output rows, or the next product's tokens in the form this one's have
template <typename TY>
int launch_mx_ty(const GemmParams& p, const MxParams& q, const MxPlan& pl, const MxMaps& w_map, int idle_sms, cudaStream_t st) {
  if constexpr (TOK_TERMS<TY> == 0 || TOK_TERMS<TY> == 4) {
    if (pl.km) return launch_mx<TY, 3, true, true>(p, q, pl, w_map, idle_sms, st);
    if (pl.f4) return pl.mb == 3 ? launch_mx<TY, 3, true>(p, q, pl, w_map, idle_sms, st) : launch_mx<TY, 1, true>(p, q, pl, w_map, idle_sms, st);
  }
  if constexpr (TOK_TERMS<TY> == 4) return MOE_ERR_UNSUPPORTED;
  else {
    if constexpr (TOK_TERMS<TY> != 2)
      if (pl.mb == 2 && pl.split == 1) return launch_mx<TY, 2, false>(p, q, pl, w_map, idle_sms, st);
    if constexpr (TOK_TERMS<TY> != 1)
      if (pl.mb == 2 && pl.split == 2) return launch_mx<TY, 2, false, false, true>(p, q, pl, w_map, idle_sms, st);
    if (pl.mb != 3) return launch_mx<TY, 1, false>(p, q, pl, w_map, idle_sms, st);
    if constexpr (TOK_TERMS<TY> != 1)
      if (mx_fits(pl.split, pl.mb)) return launch_mx<TY, 3, false, false, true>(p, q, pl, w_map, idle_sms, st);
    if constexpr (TOK_TERMS<TY> != 2) return launch_mx<TY, 3, false>(p, q, pl, w_map, idle_sms, st);
    return MOE_ERR_UNSUPPORTED;
  }
}

}  // namespace

bool moe_gemm_mx_pair_wanted(const MoeGemmArgs& a);
int64_t moe_gemm_mx_pair_workspace(const MoeGemmArgs& a);

bool moe_gemm_mx_supported(const MoeGemmArgs& a, const char** why) {
  if (a.w_kind != MOE_W_MX4_B200MX) { *why = "weights are not in the block-scaled B200 layout"; return false; }
  if (a.x_dtype != MOE_BF16 && a.x_dtype != MOE_F8E4M3) { *why = "activations are neither bf16 nor e4m3"; return false; }
  if (a.y_dtype != MOE_BF16 && a.y_dtype != MOE_F32 && a.y_dtype != MOE_F8E4M3) { *why = "output is neither bf16, fp32 nor e4m3"; return false; }
  if ((uintptr_t)a.x % 16 != 0 || (a.ld_x * (a.x_dtype == MOE_BF16 ? 2 : 1)) % 16 != 0) {
    *why = "activation rows are not 16-byte aligned"; return false;
  }
  if ((uintptr_t)a.w % 32 != 0 || (uintptr_t)a.w_scale % 16 != 0) { *why = "weights are not 32-byte aligned"; return false; }
  if (a.K % 32 != 0) { *why = "K is not a multiple of 32"; return false; }
  if (a.x_scale && a.x_dtype != MOE_F8E4M3) { *why = "activation scales need e4m3 activations"; return false; }
  if (a.kernel == MOE_GEMM_MX_F4 && a.x_dtype != MOE_BF16) { *why = "the four-term form is for bf16 activations"; return false; }
  if ((int64_t)a.E * cdiv64(a.K, 128) * cdiv64(a.N, 128) >= 2147483647LL) { *why = "too many weight tiles"; return false; }
  *why = "";
  return true;
}

extern "C" __attribute__((visibility("default"))) size_t moe_gemm_mx_workspace_bytes(const MoeGemmArgs* a) {
  if (!a || a->M <= 0 || a->E <= 0) return 0;
  if (moe_gemm_mx_pair_wanted(*a)) return (size_t)moe_gemm_mx_pair_workspace(*a);
  return a->w_kind == MOE_W_MX4_B200MX ? (size_t)mx_plan(*a).ws_bytes : 0;
}

int moe_gemm_mx_terms(const MoeGemmArgs& a) { return mx_plan(a).split; }

bool moe_gemm_mx_token_out(const MoeGemmArgs& a, TokenOut& o) {
  const MxPlan pl = mx_plan(a);
  if (a.slice_sizes == nullptr || a.mx_workspace == nullptr || a.mx_workspace_bytes < pl.ws_bytes || (pl.split == 4 && pl.tb != 16)) return false;
  int log2_tb = 4;
  while ((1 << log2_tb) < pl.tb) ++log2_tb;
  o.q = o.s = (uint8_t*)a.mx_workspace;
  o.q_step = o.s_step = pl.chunk_bytes;
  o.block_bytes = pl.KT * pl.chunk_bytes;
  o.n_one = pl.n_mma; o.fit = mx_fits(pl.split, pl.mb);
  o.terms = pl.split; o.tb = pl.tb; o.KT = pl.KT;
  o.block_offs = a.block_offs_16 + (log2_tb - 4) * a.ld_block_offs;
  return true;
}

int moe_gemm_mx_launch(const GemmParams& p_in, const MoeGemmArgs& a, const TokenOut& out, bool packed, cudaStream_t st) {
  const MxPlan pl = mx_plan(a);
  if (pl.grid_m == 0) return MOE_OK;
  MOE_CHECK_ARG(a.mx_workspace != nullptr && a.mx_workspace_bytes >= pl.ws_bytes && (uintptr_t)a.mx_workspace % 1024 == 0,
                "moe_grouped_gemm: the block-scaled kernel needs mx_workspace of moe_gemm_mx_workspace_bytes() = %lld "
                "bytes, 1024-byte aligned (got %lld)", (long long)pl.ws_bytes, (long long)a.mx_workspace_bytes);
  MOE_CHECK_ARG(pl.stages >= 2, "moe_grouped_gemm: block-scaled tile does not fit shared memory");
  GemmParams p = p_in;
  if (a.slice_sizes) {
    int row = 0;
    while ((16 << row) < pl.tb) ++row;
    p.block_offs = a.block_offs_16 + row * a.ld_block_offs;
    p.block_sched = a.block_sched_16 + row * a.ld_block_sched;
  }
  PackParams pk;
  pk.x = a.x; pk.ld_x = a.ld_x; pk.rows_x = a.rows_x;
  pk.x_scale = a.x_scale; pk.ld_xs = a.ld_x_scale;
  pk.gather = a.gather_indx;
  pk.K = a.K; pk.KT = pl.KT; pk.tb = pl.tb; pk.n_mma = pl.n_mma; pk.fit = mx_fits(pl.split, pl.mb);
  pk.chunk_bytes = pl.chunk_bytes;
  pk.out = (uint8_t*)a.mx_workspace;
  const dim3 pgrid((unsigned)pl.grid_m, (unsigned)pl.KT);
  MOE_CHECK_ARG(pl.grid_m * pl.n_groups < 2147483647LL - 65536, "moe_grouped_gemm: too many token blocks");
  if (!packed) {
    if (a.x_positions && a.x_experts && a.x_k > 0 && a.slice_sizes && a.rows_x * a.x_k == a.M && cdiv64(a.rows_x * pl.KT, 8) < 2147483647LL) {
      const PackRows rows{a.x_positions, a.x_experts, a.x_k};
      auto pack = pl.f4 ? mx_pack_rows_kernel<4> : pl.split > 1 ? mx_pack_rows_kernel<2> : mx_pack_rows_kernel<1>;
      MOE_CHECK_CUDA(launch_pdl(pack, dim3((unsigned)cdiv64(a.rows_x * pl.KT, 8)), dim3(256), 0, st, p, pk, rows));
    } else {
      auto pack = pl.f4 ? mx_pack_x4_kernel : pl.split > 1 ? mx_pack_x_kernel<true> : mx_pack_x_kernel<false>;
      MOE_CHECK_CUDA(launch_pdl(pack, pgrid, dim3(256), 0, st, p, pk));
    }
    MOE_CHECK_LAUNCH();
  }

  MxParams q;
  q.out = out;
  q.xq = (const uint8_t*)a.mx_workspace; q.chunk_bytes = pl.chunk_bytes;
  q.n_mma = pl.n_mma; q.tb = pl.tb; q.split = pl.split;
  q.KT = pl.KT; q.NB = pl.NB; q.stages = pl.stages; q.stage_bytes = pl.stage_bytes; q.acc_bufs = pl.acc_bufs;
  q.grid_m = pl.grid_m;
  // Up to a third of a block of rows per expert, where few experts have several blocks.  What streams through L2 otherwise pushes out code, tokens
  // and rows: us per step of 128 experts, 1 token 34.6 -> 32.7, 4 tokens 56.3 -> 54.0, 64 tokens 161.9 -> 158.4, 300 tokens 285 -> 278 (252 -> 243 at boost
  // clocks), 16 tokens of 32 experts 73.1 -> 69.6; with half a block per expert (64 tokens, 32 experts) the other blocks of an expert would miss
  // what the first has read, 100.5 -> 103.5.
  q.once = 3 * a.M <= (int64_t)pl.tb * (a.slice_sizes ? a.E : 1);
  q.hint_m = (uint32_t)(a.slice_sizes && a.ld_block_sched < pl.grid_m ? a.ld_block_sched : pl.grid_m);
  MxMaps w_map;
  for (int nb = 1; nb <= 3; ++nb)
    if (int rc = make_w_map(a, pl.KT, pl.NB, pl.f4 != 0, nb <= pl.mb ? nb : pl.mb, &w_map.m[nb - 1])) return rc;
  const int idle = a.idle_sms > 0 ? a.idle_sms : 0;
  if (out.q) {
    if (out.terms == 4) return launch_mx_ty<Tok4>(p, q, pl, w_map, idle, st);
    return out.terms == 2 ? launch_mx_ty<Tok2>(p, q, pl, w_map, idle, st) : launch_mx_ty<Tok1>(p, q, pl, w_map, idle, st);
  }
  if (a.y_dtype == MOE_F8E4M3) return launch_mx_ty<__nv_fp8_e4m3>(p, q, pl, w_map, idle, st);
  if (a.y_dtype == MOE_BF16) return launch_mx_ty<__nv_bfloat16>(p, q, pl, w_map, idle, st);
  return launch_mx_ty<float>(p, q, pl, w_map, idle, st);
}
