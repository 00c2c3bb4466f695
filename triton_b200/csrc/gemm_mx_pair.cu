// Ragged grouped GEMM on the block-scaled tensor-core path for many rows per expert (prefill, mid-sized batches):
// e2m1 weights with their e8m0 scales x e4m3 tokens, tcgen05.mma.cta_group::2.kind::mxf8f6f4 on pairs of SMs.
//
// bf16 tokens enter as two e4m3 terms, hi = mxfp8(x) and lo = mxfp8(x - hi), each with its own e8m0 scale per 32 k (exact up
// to underflow: a bf16 value has 8 significant bits, each term holds 4); both terms accumulate into the same fp32 columns.
// e4m3 / MXFP8 tokens are one term.  Nothing is dequantised in software, and the MMA pipe does K = 32 per instruction in the
// time kind::f16 does K = 16 (measured: 4.4 PFLOP/s for N >= 128 on 148 SMs, so two terms run at 2.2 -- the bf16 rate).
//
// (Elements far below their group of 32's largest lose what lies below 2^-23 of it, as much as an fp32 sum rounds away.)
// A row with a value beyond e4m3's scales (infinite, or near the end of bf16's range) is computed by the pack kernel in fp32, and
// the GEMM kernel does not store it.  (The pack kernel's mark per row and its look-up cost about 1 us of 183 for fc1 + fc2 of 32
// experts, 300 tokens; the same recomputation called from this kernel's epilogue took 7, by the code the call made of the rest.)
//
// What bounds it.  Shared memory, 128 B per cycle and SM: every operand byte is written once and read once per MMA, and an
// e2m1 value takes a byte there.  A cluster of two CTAs computes (2 x 256 weight rows) x (up to 128 tokens of two terms, 192 of
// one): the weights are the M operand (every CTA loads its own 128 rows of each of the two 256-row blocks: 32 KB per 128 k,
// packed in global memory), the tokens the N operand (every CTA loads half of them).  128 tokens of two terms: 49 KB written and
// 97 KB read per step, 1140 cycles, against 1024 of MMA; as two tiles of 64 tokens the weights alone would be written and
// read twice.  Large prefill runs into the power limit first (1.5 GHz).  Tokens on N
// also make a ragged tail cost what it holds, in steps of 32 rows, where tokens on M padded every expert to a multiple of 128
// or 256 (31 % of the rows of a skewed 128-expert batch of 16384 tokens).  With few rows per expert it streams the packed weights at 3
// to 4 TB/s (128 experts of 2880 x 5760 and 2880 x 2880, eight rows each: 1.7 GB in 406 us): an MMA takes 45-59 cycles however few
// columns it has.
//
// A k step of a small tile is eight MMAs of 64 cycles, so what the issuing warp does around them counts: operands in uniform
// registers, the election inside the instruction's own asm block (a step took 1150 cycles with a leader flag kept in a register,
// 840 so), and a warp for either block, whose waits the other's MMAs cover (32 experts, 1200 tokens: 319 -> 305 us).
//
// The accumulators of a tile's 256-row blocks are regions of a ring in tensor memory, each handed to the epilogue and back by
// itself.  A warp whose block has a region goes on while the other block still waits for one, up to the stages of the operand
// ring ahead.  With two regions in all the pipe waited 10000 of 37000 cycles of a tile for the epilogue.
//
// Warps of a CTA: 0 producer, 1 and 2 MMA issue (even CTA; 1 owns tensor memory), 4-7 scale loaders (shared memory ->
// registers -> tensor memory; the token scales of all columns in both CTAs, the weight scales of the own rows), 8-19 epilogue.
// Every wait is bounded; both CTAs meet at a cluster barrier before tensor memory is freed.
#include "gemm_pair_common.cuh"
#include "token_out.cuh"

namespace {

constexpr int PP_SF_WARP0 = 4, PP_EPI_WARP0 = 8, PP_EPI_WARPS = 12;
// Registers: 640 threads start with 96 each (61440); the warpgroups of producer + MMA and of the scale loaders give some up
// for the epilogue's: 128 x (56 + 64) + 384 x 120 = 61440.
constexpr int REGS_ISSUE = 56, REGS_SF = 64, REGS_EPI = 120;
static_assert(128 * (REGS_ISSUE + REGS_SF) + PP_EPI_WARPS * 32 * REGS_EPI <= 96 * 640, "register split");
constexpr int PP_THREADS = (PP_EPI_WARP0 + PP_EPI_WARPS) * 32;

constexpr int PP_MAX_STAGES = 6, PP_MAX_REGIONS = 12;
constexpr int PP_NUM_BARS = 3 * PP_MAX_STAGES + 2 * PP_MAX_REGIONS + 1;
// shared memory behind the stages: [token tables x 2][barriers][tensor-memory base, abort flag][columns of the next tiles][prefix]
constexpr int PP_OFF_BAR = 2 * PAIR_TAB, PP_OFF_MISC = PP_OFF_BAR + (PP_NUM_BARS * 8 + 15) / 16 * 16, PP_OFF_COLS = PP_OFF_MISC + 16,
              PP_OFF_PREFIX = PP_OFF_COLS + 8 * 4, PP_CTL_BASE = (PP_OFF_PREFIX + PAIR_PREFIX_INTS * 4 + 15) / 16 * 16;
// ... and where the rows become the next product's tokens, a stage per two epilogue warps
template <typename TY> constexpr int PP_CTL = PP_CTL_BASE + (TOK_TERMS<TY> ? PP_EPI_WARPS / 2 * TOK_STAGE : 0);
constexpr int PP_SMEM = 227 * 1024;
// How tokens enter the MMA.  ONE: e4m3 rows, one term.  TWO: two terms, two MMAs into the same columns.  SIDE: the terms as
// neighbouring columns of one MMA (eight hi, eight lo, ...), added in the epilogue.  An MMA takes 45-59 cycles however few
// columns it has: with up to 96 tokens a tile SIDE issues half of them (32 tokens: 45 cycles per 32 k of a weight block
// against 118).
enum { PP_ONE = 1, PP_TWO = 2, PP_SIDE = 3 };
template <int FORM> constexpr int TERMS_OF = FORM == PP_ONE ? 1 : 2;
template <int FORM> constexpr int SF_COLS = FORM == PP_TWO ? 24 : 16;      // tensor-memory columns of scales per stage: 8 of two blocks, 8 per MMA of a k group

struct PairParams {
  const uint8_t* xq;            // [k step][padded row / 8][term][8 rows][128 B], 16-byte pieces swizzled with (row & 7)
  const uint8_t* xs;            // [k step][padded row / 8][term][8 rows][4 B]: e8m0 of the four 32-groups
  const uint32_t* done;         // [padded row], not zero: the pack kernel has written its outputs itself (two-term tokens)
  int64_t prows;                // padded rows: expert e's rows start at (slice_offs[e] & ~31) + 32 e
  int KT, NB;                   // 128-k steps, 128-row weight blocks
  int nmax;                     // token columns of a tile at most, a multiple of 32
  int upt;                      // weight blocks of 256 rows per tile: 1 or 2
  int stages, stage_bytes, regions, reg_cols;      // accumulator regions of reg_cols tensor-memory columns
  TokenOut out;
};

struct PairMaps { CUtensorMap w[2], s[2]; };        // weight tiles and their scales in boxes of one and two blocks

// line (128 bytes of values, 4 of scales) of a token's term
template <int TERMS> __device__ __forceinline__ int64_t token_line(int64_t kt, int64_t prows, int64_t prow, int term) {
  return TERMS * (kt * prows + (prow & ~(int64_t)7)) + term * 8 + (prow & 7);
}

// ============================================================================================================
// Pack kernel.  A block takes up to 16 rows of one expert (an entry of the 16-row block schedule).  bf16: a thread a group of
// 32 k.  e4m3: a warp a row at a time, a lane 16 consecutive k, four passes' loads in flight before the first is stored.
// HBM-bound: 2 + 2 bytes per bf16 element, 1 + 1 per e4m3 element (gathered rows are read through L2).
// ============================================================================================================
struct PairPackParams {
  const void* x; int64_t ld_x; int64_t rows_x;
  const uint8_t* x_scale; int64_t ld_xs;
  const int32_t* gather;
  int K, KT, NB, y_dtype;
  int64_t prows;
  uint8_t* xq; uint8_t* xs;
  uint32_t* done;
  const int32_t* positions; const int16_t* experts;      // [rows_x, k]: where the rows of x go (NULL: gather says)
  int k;
  TokenOut out;                  // the product's rows are the next one's tokens: those computed here go there too
};

__device__ __forceinline__ bool pack_block(const GemmParams& p, int64_t pid, int& e, int64_t& row0, int& rows, int64_t& prow0) {
  if (p.slice_sizes == nullptr) {
    e = 0;
    row0 = prow0 = pid * 16;
    rows = (int)min((int64_t)16, p.M - row0);
    return rows > 0;
  }
  const uint32_t ent = (uint32_t)p.block_sched[pid];
  if (ent == 0xFFFFFFFFu) return false;
  e = (int)(ent & 0xFFFFu);
  // An entry holds 16 bits of the block's place inside its expert.  The blocks of an expert are neighbours in the schedule, so
  // every entry of the same expert 65536 places (2^20 rows) further back is one more turn of the counter.
  int first = (int)(ent >> 16) * 16;
  for (int64_t back = pid - 65536; back >= 0 && (p.block_sched[back] & 0xFFFF) == e; back -= 65536) first += 65536 * 16;
  const int off = p.slice_offs[e];
  row0 = (int64_t)off + first;
  prow0 = padded_base(e, off) + first;
  rows = min(16, p.slice_sizes[e] - first);
  return rows > 0;
}

// One 32-group of a bf16 row as two terms.  PERMUTED: k inside eight in the order of the default weight tiles (0, 2, 4, 6, 1, 3, 5, 7).
struct Group2 { uint32_t h[8], l[8], sh, sl; };
template <bool PERMUTED>
__device__ __forceinline__ float quantise_group2(const uint4 (&raw)[4], Group2& q) {       // -> the group's maximum
  float v[32], m;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t w[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      v[8 * i + (PERMUTED ? j : 2 * j)] = __uint_as_float(w[j] << 16);
      v[8 * i + (PERMUTED ? 4 + j : 2 * j + 1)] = __uint_as_float(w[j] & 0xFFFF0000u);
    }
  }
  two_terms<32>(v, [](float own) { return own; }, q.h, q.l, q.sh, q.sl, m);
  return m;
}
// line, s: the row's line and scales at the k step of group g
__device__ __forceinline__ void store_group2(const Group2& q, int x7, int g, uint8_t* line, int lo_q, uint8_t* s, int lo_s) {
  const uint32_t odd = (uint32_t)x7 & 1u;                          // 16-byte pieces 2 g and 2 g + 1 of the line, xor x7
  uint8_t* dst = line + ((((uint32_t)(g & 3) << 1) ^ ((uint32_t)x7 & 6u)) << 4);
  const uint4 h0 = make_uint4(q.h[0], q.h[1], q.h[2], q.h[3]), h1 = make_uint4(q.h[4], q.h[5], q.h[6], q.h[7]);
  const uint4 l0 = make_uint4(q.l[0], q.l[1], q.l[2], q.l[3]), l1 = make_uint4(q.l[4], q.l[5], q.l[6], q.l[7]);
  st_v8(dst, odd ? h1 : h0, odd ? h0 : h1);
  st_v8(dst + lo_q, odd ? l1 : l0, odd ? l0 : l1);
  s[g & 3] = (uint8_t)q.sh;
  s[lo_s + (g & 3)] = (uint8_t)q.sl;
}
template <bool PERMUTED>
__device__ __forceinline__ float pack_group2(const uint4 (&raw)[4], int x7, int g, uint8_t* line, int lo_q, uint8_t* s, int lo_s) {
  Group2 q;
  const float m = quantise_group2<PERMUTED>(raw, q);
  store_group2(q, x7, g, line, lo_q, s, lo_s);
  return m;
}

// Magnitude from which on two e4m3 terms do not hold a token's value: infinities, and finite values that round to 2^128.
constexpr float BEYOND = 3.0e38f;

// Output of a row with such a value, in fp32 on the CUDA cores by the whole block, a thread per weight row: what the product of bf16
// values gives (an infinite token value times a weight is infinite, or NaN for a zero weight).  `groups`: bits of the groups of 32 k
// that decide it (those with an infinity or NaN, if there is an infinity), NULL for all.
constexpr int EXACT_WORDS = 64;
template <typename TY, bool TILED>
__device__ void exact_row(const GemmParams& p, const PairPackParams& a, int e, int64_t m, int64_t dst, const __nv_bfloat16* x,
                          const uint32_t* groups) {
  TY* y = gemm_out_row<TY>(p, dst);
  const int lane = threadIdx.x & 31;
  for (int n = threadIdx.x; n - lane < p.N; n += 256) {
    const int b = n >> 7, row = n & 127;
    float acc = 0.0f;
    for (int kg = 0; kg < p.K >> 5; ++kg) {                        // scale groups of 32 k
      if (groups && !((groups[kg >> 5] >> (kg & 31)) & 1u)) continue;
      const int kt = kg >> 2, g = kg & 3;
      const int64_t at = TILED ? ((int64_t)e * a.NB + b) * a.KT + kt : ((int64_t)e * a.KT + kt) * a.NB + b;
      const uint8_t* q = (const uint8_t*)p.w + at * 8192 + (TILED ? (g * 128 + row) * 16 : row * 64 + g * 16);
      const uint32_t sb = p.w_scale[at * 512 + (TILED ? row * 4 + g : (row & 31) * 16 + (row >> 5) * 4 + g)];
      const float s = __uint_as_float(sb ? (sb == 255u ? 0x7FC00000u : sb << 23) : 0x00400000u);
      const uint4 q4 = *reinterpret_cast<const uint4*>(q);
#pragma unroll
      for (int i = 0; i < 4; ++i) {                                // words of eight values
        uint32_t w = i == 0 ? q4.x : i == 1 ? q4.y : i == 2 ? q4.z : q4.w;
        if (TILED) {                                               // evens, then odds: back to pairs
          uint32_t pairs = 0;
          for (int j = 0; j < 4; ++j) pairs |= (((w >> (4 * j)) & 0xFu) | (((w >> (16 + 4 * j)) & 0xFu) << 4)) << (8 * j);
          w = pairs;
        }
        for (int j = 0; j < 4; ++j) {
          const float2 f = e2m1x2_to_f32x2((w >> (8 * j)) & 0xFFu);
          const int k = kg * 32 + 8 * i + 2 * j;
          acc = fmaf(__bfloat162float(x[k]), f.x * s, acc);
          acc = fmaf(__bfloat162float(x[k + 1]), f.y * s, acc);
        }
      }
    }
    if (p.bias && n < p.N) acc += load_bias(p.bias, p.bias_dtype, (int64_t)e * p.ld_bias + n) * (p.betas ? p.betas[m] : 1.0f);
    if (p.has_out_alpha) acc *= p.out_alpha;
    const float gamma = p.gammas ? p.gammas[m] : 1.0f, other = __shfl_xor_sync(0xFFFFFFFFu, acc, 1);
    if (p.activation == MOE_ACT_SWIGLU) {
      if (!(lane & 1) && n + 1 < p.N) y[n >> 1] = from_f32<TY>(gemm_swiglu(acc, other, p.act_alpha, p.act_limit, p.act_has_limit) * gamma);
    } else if (n < p.N) {
      y[n] = from_f32<TY>(acc * gamma);
    }
  }
}

// Such a row, position m of expert e; all threads of the block call
template <bool TILED>
__device__ __noinline__ void exact_position(const GemmParams& p, const PairPackParams& a, int e, int64_t m, const __nv_bfloat16* x) {
  __shared__ uint32_t s_groups[EXACT_WORDS];
  const int64_t d = p.scatter_indx ? (int64_t)p.scatter_indx[m] : m;
  if (d < 0) return;
  for (int i = threadIdx.x; i < EXACT_WORDS; i += 256) s_groups[i] = 0;
  __syncthreads();
  bool inf = false;
  for (int kg = threadIdx.x; kg < a.K >> 5; kg += 256) {
    bool odd = false;
    for (int k = kg * 32; k < kg * 32 + 32; ++k) {
      const float v = fabsf(__bfloat162float(x[k]));
      odd |= !(v < BEYOND);
      inf |= v > 3.4e38f;
    }
    if (odd && kg < 32 * EXACT_WORDS) atomicOr(&s_groups[kg >> 5], 1u << (kg & 31));
  }
  const uint32_t* groups = __syncthreads_or(inf) && a.K <= 1024 * EXACT_WORDS ? s_groups : nullptr;
  if (a.y_dtype == MOE_BF16) exact_row<__nv_bfloat16, TILED>(p, a, e, m, d, x, groups);
  else if (a.y_dtype == MOE_F32) exact_row<float, TILED>(p, a, e, m, d, x, groups);
  else exact_row<__nv_fp8_e4m3, TILED>(p, a, e, m, d, x, groups);
  __syncthreads();
  if (a.out.q) {
    const uint4* y = reinterpret_cast<const uint4*>((const __nv_bfloat16*)p.y + d * p.ld_y);
    uint8_t *q, *s;
    const int off = p.slice_offs[e], rr = (int)(m - off);
    token_addr(a.out, e, off, p.slice_sizes[e], a.out.tb ? a.out.block_offs[e] : 0, rr, q, s);
    int lo_q, lo_s;
    token_strides(a.out, s, lo_q, lo_s);
    s = (uint8_t*)((uintptr_t)s & ~(uintptr_t)3);
    for (int g = threadIdx.x; g < 4 * a.out.KT; g += 256) {
      uint4 raw[4] = {};
      if (g < p.N >> 6)
        for (int i = 0; i < 4; ++i) raw[i] = y[g * 4 + i];
      if (a.out.permuted) pack_group2<true>(raw, rr & 7, g, q + (g >> 2) * a.out.q_step, lo_q, s + (g >> 2) * a.out.s_step, lo_s);
      else pack_group2<false>(raw, rr & 7, g, q + (g >> 2) * a.out.q_step, lo_q, s + (g >> 2) * a.out.s_step, lo_s);
    }
  }
}

// The rows with such a value among a block's; all of its threads call.  -> their bits
template <bool TILED>
__device__ __noinline__ uint32_t exact_rows(const GemmParams& p, const PairPackParams& a, int e, int64_t row0, int rows) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t mine = 0, all = 0;
  for (int r = warp; r < rows; r += 8) {
    const int64_t src = p.gather_indx ? (int64_t)p.gather_indx[row0 + r] : row0 + r;
    if (src < 0 || src >= a.rows_x) continue;
    const __nv_bfloat16* x = (const __nv_bfloat16*)a.x + src * a.ld_x;
    bool is = false;
    for (int k = lane; k < a.K; k += 32) is |= fabsf(__bfloat162float(x[k])) >= BEYOND;
    if (__any_sync(0xFFFFFFFFu, is)) mine |= 1u << r;
  }
  for (int r = 0; r < rows; ++r) {
    if (!__syncthreads_or((mine >> r) & 1u)) continue;
    all |= 1u << r;
    const int64_t m = row0 + r;
    const __nv_bfloat16* x = (const __nv_bfloat16*)a.x + (p.gather_indx ? (int64_t)p.gather_indx[m] : m) * a.ld_x;
    exact_position<TILED>(p, a, e, m, x);
  }
  return all;
}

// TILED: k inside eight in the order of the default weight tiles (0, 2, 4, 6, 1, 3, 5, 7).  A thread takes a whole group of 32 k:
// no exchange between lanes, 64 bytes in, a 32-byte sector out per term.  With eight k per lane and four lanes to a group, 65536
// rows of 2880 took 153 us and 4800 rows 20.3, so 141 and 16.8.
// PARTS: blocks (1, 2 or 4) that share the groups of 16 rows, each with its bytes of the rows' words.  (A constant: divided by at run time, and with the
// registers of three blocks per SM for whole ones too, a product of 64 experts of 736 x 1440 took 0.8 us of 22 longer.)
template <bool TILED, int PARTS>
__global__ void __launch_bounds__(256, PARTS == 1 ? 1 : 3) mx_pair_pack2_kernel(const __grid_constant__ GemmParams p, const __grid_constant__ PairPackParams a) {
  pdl_begin();
  int e; int64_t row0, prow0; int rows;
  const int part = (int)(blockIdx.x % PARTS);
  if (!pack_block(p, blockIdx.x / PARTS, e, row0, rows, prow0)) return;
  const int kt0 = part * a.KT / PARTS, G = ((part + 1) * a.KT / PARTS - kt0) * 4;      // groups of this part's k steps
  bool beyond = false;
  for (int t = threadIdx.x; t < rows * G; t += 256) {
    const int r = t / G, g = kt0 * 4 + t - r * G;
    int64_t src = a.gather ? (int64_t)a.gather[row0 + r] : row0 + r;
    if (src >= a.rows_x) src = -1;
    uint4 raw[4] = {};
    if (src >= 0 && g * 32 < a.K) {                    // K % 32 == 0
      const uint4* x = reinterpret_cast<const uint4*>((const __nv_bfloat16*)a.x + src * a.ld_x + g * 32);
#pragma unroll
      for (int i = 0; i < 4; ++i) raw[i] = x[i];
    }
    const int64_t prow = prow0 + r, line = token_line<2>(g >> 2, a.prows, prow, 0);
    const float m = pack_group2<TILED>(raw, (int)prow & 7, g, a.xq + line * 128, 1024, a.xs + line * 4, 32);
    beyond |= !(m < BEYOND);                           // (what is packed of such a row is not used; a NaN makes its results NaN)
  }
  uint32_t done = 0;
  if (__syncthreads_or(beyond)) done = exact_rows<TILED>(p, a, e, row0, rows);
  if ((int)threadIdx.x < rows) {
    uint32_t* word = a.done + prow0 + threadIdx.x;
    const uint32_t bit = (done >> threadIdx.x) & 1u;
    if constexpr (PARTS == 1) *word = bit;
    else if constexpr (PARTS == 2) ((uint16_t*)word)[part] = (uint16_t)bit;
    else ((uint8_t*)word)[part] = (uint8_t)bit;
  }
}

template <bool TILED>
auto pack2_in_parts(int parts) {
  return parts == 4 ? mx_pair_pack2_kernel<TILED, 4> : parts == 2 ? mx_pair_pack2_kernel<TILED, 2> : mx_pair_pack2_kernel<TILED, 1>;
}

// The same with the rows of x in turn, given the positions of every one (positions, experts: k per row): a row that k experts take is read
// and quantised once and its lines are written k times.  16384 rows of 2880, four positions each: 137 us by position, 105 by row (390 MB out);
// the prefill step 3144 -> 3081 us, with 8192 e4m3 rows 910 -> 903.
constexpr int PACK_TOKENS = 8;
constexpr int PACK_MAX_K = 512;                        // positions of a row: PACK_TOKENS x k words of 8 bytes in the 48 KB that need no opt-in
// padded row of pick j of row t; -1 where the pick is not a row of one of the experts (dropped ones are -1)
__device__ __forceinline__ int64_t pick_prow(const GemmParams& p, const PairPackParams& a, int64_t t, int j, int& e, int64_t& m) {
  const int pick = a.experts[t * a.k + j];
  e = (unsigned)pick < (unsigned)p.E ? pick : 0;
  m = a.positions[t * a.k + j];
  const int off = p.slice_offs[e], rows = p.slice_sizes[e];
  return e == pick && m >= off && m < off + rows ? padded_base(e, off) + (m - off) : -1;
}
template <bool TILED>
__global__ void __launch_bounds__(256) mx_pair_pack2_rows_kernel(const __grid_constant__ GemmParams p, const __grid_constant__ PairPackParams a) {
  pdl_begin();
  extern __shared__ int64_t s_prow[];                  // [PACK_TOKENS][k]
  __shared__ uint32_t s_beyond;
  const int64_t t0 = (int64_t)blockIdx.x * PACK_TOKENS;
  const int n = (int)min((int64_t)PACK_TOKENS, a.rows_x - t0);
  if (threadIdx.x == 0) s_beyond = 0;
  for (int i = threadIdx.x; i < n * a.k; i += 256) {
    int e; int64_t m;
    s_prow[i] = pick_prow(p, a, t0 + i / a.k, i % a.k, e, m);
  }
  __syncthreads();
  const int G = a.KT * 4;
  for (int t = threadIdx.x; t < n * G; t += 256) {
    const int r = t / G, g = t - r * G;
    uint4 raw[4] = {};
    if (g * 32 < a.K) {                                // K % 32 == 0
      const uint4* x = reinterpret_cast<const uint4*>((const __nv_bfloat16*)a.x + (t0 + r) * a.ld_x + g * 32);
#pragma unroll
      for (int i = 0; i < 4; ++i) raw[i] = x[i];
    }
    Group2 q;
    if (!(quantise_group2<TILED>(raw, q) < BEYOND)) atomicOr(&s_beyond, 1u << r);
    for (int j = 0; j < a.k; ++j) {
      const int64_t prow = s_prow[r * a.k + j], line = token_line<2>(g >> 2, a.prows, prow, 0);
      if (prow < 0) continue;
      store_group2(q, (int)prow & 7, g, a.xq + line * 128, 1024, a.xs + line * 4, 32);
    }
  }
  __syncthreads();
  const uint32_t beyond = s_beyond;
  for (int i = threadIdx.x; i < n * a.k; i += 256)
    if (s_prow[i] >= 0) a.done[s_prow[i]] = (beyond >> (i / a.k)) & 1u;
  if (beyond)
    for (int i = 0; i < n * a.k; ++i)
      if (((beyond >> (i / a.k)) & 1u) && s_prow[i] >= 0) {
        int e; int64_t m;
        pick_prow(p, a, t0 + i / a.k, i % a.k, e, m);
        exact_position<TILED>(p, a, e, m, (const __nv_bfloat16*)a.x + (t0 + i / a.k) * a.ld_x);
        __syncthreads();
      }
}

__global__ void __launch_bounds__(256) mx_pair_pack1_rows_kernel(const __grid_constant__ GemmParams p, const __grid_constant__ PairPackParams a) {
  pdl_begin();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t t = (int64_t)blockIdx.x * PACK_TOKENS + warp;      // a warp a row
  if (t >= a.rows_x) return;
  const uint8_t* xrow = (const uint8_t*)a.x + t * a.ld_x;
  const int K128 = a.KT * 128;
  for (int kb = lane * 16; kb - lane * 16 < K128; kb += 2048) {
    uint4 raw[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) raw[u] = kb + 512 * u < a.K ? *reinterpret_cast<const uint4*>(xrow + kb + 512 * u) : make_uint4(0, 0, 0, 0);
    for (int j = 0; j < a.k; ++j) {
      int e; int64_t m;
      const int64_t prow = pick_prow(p, a, t, j, e, m);
      if (prow < 0) continue;
      const uint32_t x7 = (uint32_t)prow & 7u;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int k = kb + 512 * u;
        if (k < K128)
          *reinterpret_cast<uint4*>(a.xq + ((int64_t)(k >> 7) * a.prows + prow) * 128 + ((((uint32_t)(k & 127) >> 4) ^ x7) << 4)) = raw[u];
      }
    }
  }
  for (int i = lane; i < a.KT * a.k; i += 32) {
    const int kt = i / a.k;
    int e; int64_t m;
    const int64_t prow = pick_prow(p, a, t, i - kt * a.k, e, m);
    if (prow < 0) continue;
    uint32_t s = 0x7F7F7F7Fu;                                      // 1.0
    if (a.x_scale) {
      s = 0;
#pragma unroll
      for (int g = 0; g < 4; ++g) s |= (kt * 4 + g < (a.K >> 5) ? (uint32_t)a.x_scale[t * a.ld_xs + kt * 4 + g] : 127u) << (8 * g);
    }
    *reinterpret_cast<uint32_t*>(a.xs + ((int64_t)kt * a.prows + prow) * 4) = s;
  }
}

__global__ void __launch_bounds__(256) mx_pair_pack1_kernel(const __grid_constant__ GemmParams p, const __grid_constant__ PairPackParams a) {
  pdl_begin();
  int e; int64_t row0, prow0; int rows;
  if (!pack_block(p, blockIdx.x, e, row0, rows, prow0)) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int K128 = a.KT * 128;
  for (int r = warp; r < rows; r += 8) {
    int64_t src = a.gather ? (int64_t)a.gather[row0 + r] : row0 + r;
    if (src >= a.rows_x) src = -1;
    const uint8_t* xrow = (const uint8_t*)a.x + (src >= 0 ? src : 0) * a.ld_x;
    const int64_t prow = prow0 + r;
    const uint32_t x7 = (uint32_t)prow & 7u;
    for (int kb = lane * 16; kb - lane * 16 < K128; kb += 2048) {
      uint4 raw[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int k = kb + 512 * u;                                // K % 32 == 0: 16 values are in or out together
        raw[u] = (src >= 0 && k < a.K) ? *reinterpret_cast<const uint4*>(xrow + k) : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int k = kb + 512 * u;
        if (k < K128)
          *reinterpret_cast<uint4*>(a.xq + ((int64_t)(k >> 7) * a.prows + prow) * 128 + ((((uint32_t)(k & 127) >> 4) ^ x7) << 4)) = raw[u];
      }
    }
    for (int kt = lane; kt < a.KT; kt += 32) {
      uint32_t s = 0x7F7F7F7Fu;                                    // 1.0
      if (a.x_scale && src >= 0) {
        s = 0;
#pragma unroll
        for (int g = 0; g < 4; ++g)
          s |= (kt * 4 + g < (a.K >> 5) ? (uint32_t)a.x_scale[src * a.ld_xs + kt * 4 + g] : 127u) << (8 * g);
      }
      *reinterpret_cast<uint32_t*>(a.xs + ((int64_t)kt * a.prows + prow) * 4) = s;
    }
  }
}

// ============================================================================================================
// The GEMM kernel
// ============================================================================================================
// A_HI, B_HI: high words of the descriptors (swizzle, distance of 8-row groups)
template <uint32_t A_HI, uint32_t B_HI>
__device__ __forceinline__ void mma_mxf8f6f4_pair(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t sfa,
                                                  uint32_t sfb, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 da, db;\n\t"
      "mov.b64 da, {%1, %7};\n\t"
      "mov.b64 db, {%2, %8};\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "elect.sync _|q, 0xFFFFFFFF;\n\t"
      "@q tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale.scale_vec::1X [%0], da, db, %3, [%4], [%5], p;\n\t}" ::"r"(d_tmem),
      "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(sfa), "r"(sfb), "r"(accumulate), "n"(A_HI), "n"(B_HI)
      : "memory");
}
// Weights in the default tiles ([group of 32 k][128 rows][16 B], see layout.cu).  The TMA unit reads 64 bytes = four rows of
// one group per 128-byte line and swizzles 16-byte pieces with the line (address bits 4-6 ^= bits 7-9).  Read as rows of 32
// bytes with the 32-byte swizzle (bit 4 ^= bit 7) those lines are one K = 32 operand of 128 rows in which row r sits at
// r ^ ((r >> 3) & 3): the other two swizzled bits are row bits.  The order of k inside eight (even, then odd) is taken up by the
// token pack kernel.  So the tiles of the bf16 kernels feed the block-scaled MMA as they are stored.
constexpr uint32_t DESC_HI_SW32 = (256u >> 4) | (1u << 14) | (6u << 29);      // 8-row groups 256 B apart, 32-byte swizzle
__device__ __forceinline__ int tiled_row(int pos) { return pos ^ ((pos >> 3) & 3); }       // its own inverse
// A = e2m1 (code 5), B = e4m3 (code 0), both K-major, e8m0 scales, M = 256 over the two CTAs; sf: byte of the scale words
__device__ __forceinline__ uint32_t pair_idesc(int n, uint32_t sf) {
  return (sf << 4) | (5u << 7) | ((uint32_t)(n >> 3) << 17) | (1u << 23) | (2u << 27) | (sf << 29);
}

// TILED: weights in the default tiles [E][n_tile][k_tile], else in the block-scaled ones [E][k_tile][n_block]
// ONCE: weights are read about once, and are the first to leave L2.  (A constant: as a choice inside the producer's loop, or as a second loop, it made the
// others 0.5 to 1.4 % slower.)
template <typename TY, int FORM, bool TILED, bool ONCE>
__global__ void __launch_bounds__(PP_THREADS, 1)
gemm_mx_pair_kernel(const GemmParams p, const PairParams a, const __grid_constant__ PairMaps maps) {
  constexpr int TERMS = TERMS_OF<FORM>, MMAS = FORM == PP_TWO ? 2 : 1;
  constexpr uint32_t B_HI = FORM == PP_TWO ? (2048u >> 4) | (DESC_HI & 0xFFFFC000u) : DESC_HI;      // TWO: 8 hi rows, 8 lo rows, ...
  constexpr uint32_t A_HI = TILED ? DESC_HI_SW32 : DESC_HI, A_KK = TILED ? 4096 >> 4 : 2;      // next 32 k of A: 16-byte units
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sbase = smem_u32(smem);
  const int warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;     // warp-uniform for the compiler
  const uint32_t rank = cluster_ctarank();
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
  const int STAGES = a.stages, UPT = a.upt;
  // stage: [UPT x 16 KB weights, byte per element][TERMS x nmax / 2 token rows x 128 B][weight scales][token scales of all columns:
  // TERMS x 256 words]
  const uint32_t OFF_X = (uint32_t)UPT * (128 * 128), OFF_WS = OFF_X + TERMS * (uint32_t)a.nmax * 64u, OFF_XS = OFF_WS + 1024u;
  const uint32_t SF_BASE = (uint32_t)(TMEM_COLS - STAGES * SF_COLS<FORM>);
  uint8_t* ctl_ptr = smem + (size_t)STAGES * a.stage_bytes;
  const uint32_t ctl0 = smem_u32(ctl_ptr), bar0 = ctl0 + PP_OFF_BAR;
  auto BAR_FULL = [&](int s) { return bar0 + 8u * (uint32_t)s; };                       // own copies have landed
  auto BAR_EMPTY = [&](int s) { return bar0 + 8u * (uint32_t)(PP_MAX_STAGES + s); };
  auto BAR_SF = [&](int s) { return bar0 + 8u * (uint32_t)(2 * PP_MAX_STAGES + s); };    // even CTA: scales (and operands) of both CTAs
  auto BAR_ACC_FULL = [&](int r) { return bar0 + 8u * (uint32_t)(3 * PP_MAX_STAGES + r); };
  auto BAR_ACC_EMPTY = [&](int r) { return bar0 + 8u * (uint32_t)(3 * PP_MAX_STAGES + PP_MAX_REGIONS + r); };   // even CTA
  const uint32_t BAR_DRAIN = bar0 + 8u * (uint32_t)(PP_NUM_BARS - 1);
  volatile uint32_t* s_tmem = reinterpret_cast<volatile uint32_t*>(ctl_ptr + PP_OFF_MISC);
  volatile int* s_abort = reinterpret_cast<volatile int*>(ctl_ptr + PP_OFF_MISC + 4);
  volatile int* s_cols = reinterpret_cast<volatile int*>(ctl_ptr + PP_OFF_COLS);
  int32_t* s_prefix = reinterpret_cast<int32_t*>(ctl_ptr + PP_OFF_PREFIX);
  Ctl ctl{s_abort, p.status};

  if (threadIdx.x == 0) {
    for (int s = 0; s < PP_MAX_STAGES; ++s) {
      mbar_init(BAR_FULL(s), 1);
      mbar_init(BAR_EMPTY(s), 2);                      // both MMA warps
      mbar_init(BAR_SF(s), 8);                         // four scale warps in each CTA
    }
    for (int r = 0; r < PP_MAX_REGIONS; ++r) {
      mbar_init(BAR_ACC_FULL(r), 1);
      mbar_init(BAR_ACC_EMPTY(r), 2 * PP_EPI_WARPS);
    }
    mbar_init(BAR_DRAIN, 2);
    *s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ctl0 + PP_OFF_MISC), "r"((uint32_t)TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  const int KT = a.KT, NB = a.NB;
  const int MB = (NB + 1) >> 1, MT = (MB + UPT - 1) / UPT;      // 256-row weight blocks, tiles of UPT of them
  // The blocks of a tile: CTA r takes the neighbouring blocks 4 t + 2 r and + 1 (one copy each stage), a block of the MMA is one
  // block of either CTA; with at most two blocks left (or UPT = 1), block + r.  -> own first block, own blocks, MMA blocks.
  struct Blocks { int first, own, units; };
  auto blocks_of = [&](int tile) {
    const int b0 = (tile % MT) * UPT * 2, left = NB - b0;
    Blocks b;
    const bool wide = UPT == 2 && left > 2;
    b.first = b0 + (wide ? 2 : 1) * (int)rank;
    b.own = wide ? min(2, max(0, NB - b.first)) : (int)((int)rank < left);
    b.units = wide ? 2 : 1;
    return b;
  };
  if (warp == 3) {
    // Ahead of the wait for the kernel before (whose CTA on this SM may have left long before its last one does): L2 is asked for the weights
    // of the first tile's first stages (8 experts of 512 x 2048, 256 tokens: 30.5 -> 29.0 us per step).
    const int e = pair_hint_expert(p, a.nmax, pair / MT, lane);
    const Blocks b = blocks_of(pair);
    if (e >= 0) {
      for (int i = lane; i < (TILED ? b.own : STAGES); i += 32) {
        const int64_t tile = TILED ? (int64_t)(e * NB + b.first + i) * KT : (int64_t)(e * KT + i) * NB + b.first;
        const uint32_t n = (uint32_t)(TILED ? STAGES : b.own);
        if (n == 0) break;
        l2_hint((const uint8_t*)p.w + tile * 8192, n * 8192u);
        l2_hint(p.w_scale + tile * 512, n * 512u);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                                  // the other CTA's barriers exist before anyone signals them
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xFFFFFFFFu, *s_tmem, 0);
  pdl_begin();
  if (warp == PP_SF_WARP0) pair_prefix(p, s_prefix, a.nmax, lane);      // tile prefix over experts
  __syncthreads();
  const int n_tiles = __shfl_sync(0xFFFFFFFFu, s_prefix[p.slice_sizes ? p.E : 1], 0) * MT;

  if (warp < PP_SF_WARP0) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_ISSUE));
  if (warp == 0) {
    // ================================= producer =======================================================
    uint32_t s = 0, ph = 1, issued = 0;
    uint64_t policy = 0;
    if constexpr (ONCE) asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
    bool ok = true;
    PTile nxt;                                         // the next tile is looked up while this one streams
    if (pair < n_tiles) nxt = map_ptile(p, s_prefix, pair / MT);
    for (int tile = pair; tile < n_tiles && ok; tile += n_pairs) {
      const int e = __shfl_sync(0xFFFFFFFFu, nxt.e, 0), cols = __shfl_sync(0xFFFFFFFFu, nxt.cols, 0);
      const int prow0 = __shfl_sync(0xFFFFFFFFu, (int)padded_base(nxt.e, nxt.off) + nxt.first, 0);
      const Blocks b = blocks_of(tile);
      const uint32_t bx = (uint32_t)(TERMS * cols) * 64u, bs = (uint32_t)(TERMS * cols) * 4u;        // own half of the rows, all scales
      const uint32_t tx = (uint32_t)b.own * (128 * 64 + 512) + bx + bs;
      const CUtensorMap* wm = &maps.w[b.own == 2];
      const CUtensorMap* sm = &maps.s[b.own == 2];
      const uint8_t* xq = a.xq + TERMS * ((int64_t)prow0 * 128) + rank * bx;
      const uint8_t* xs = a.xs + TERMS * ((int64_t)prow0 * 4);
      const int64_t q_step = TERMS * a.prows * 128, s_step = TERMS * a.prows * 4;
      int c2 = TILED ? 0 : b.first, c3 = TILED ? e * NB + b.first : e * KT;
      for (int kt = 0; kt < KT; ++kt, ++issued) {
        ok = __all_sync(0xFFFFFFFFu, mbar_wait(BAR_EMPTY(s), ph, ctl, 611));
        if (!ok) break;
        const uint32_t st = sbase + s * (uint32_t)a.stage_bytes, bar = BAR_FULL(s);
        elect_expect_tx(bar, tx);
        if (b.own > 0) {
          if constexpr (ONCE) {
            elect_tile_4d_hint(st, wm, 0, 0, c2, c3, bar, policy);
            elect_tile_3d_hint(st + OFF_WS, sm, 0, c2, c3, bar, policy);
          } else {
            elect_tile_4d(st, wm, 0, 0, c2, c3, bar);
            elect_tile_3d(st + OFF_WS, sm, 0, c2, c3, bar);
          }
        }
        elect_bulk_g2s(st + OFF_X, xq, bx, bar);
        elect_bulk_g2s(st + OFF_XS, xs, bs, bar);
        xq += q_step; xs += s_step;
        if (TILED) ++c2; else ++c3;
        if (++s == (uint32_t)STAGES) { s = 0; ph ^= 1u; }
        if (kt == 0 && tile + n_pairs < n_tiles) nxt = map_ptile(p, s_prefix, (tile + n_pairs) / MT);
      }
    }
    if (!ok && lane == 0) {
      // aborting: let the copies that were already issued land before the CTA leaves
      for (uint32_t j = issued > (uint32_t)STAGES ? issued - STAGES : 0; j < issued; ++j)
        for (uint32_t i = 0; i < (1u << 16) && !mbar_test(BAR_FULL(j % STAGES), (j / STAGES) & 1u); ++i) __nanosleep(64);
    }
    __syncwarp();
  } else if (warp <= 2) {
    // ================================= MMA issuers (even CTA) =========================================
    // One warp per block of the tile: what a warp does between its k steps is covered by the other's MMAs, and a block whose
    // region is free starts while the other still waits for the epilogue, up to the stages of the ring ahead.
    if (rank == 0) {
      const int u = warp - 1, k_whole = p.K >> 7;      // steps of 128 k; the last may hold less
      uint32_t s = 0, ph = 0;                          // stage and parity of the next k step
      uint32_t tc = 0, blk = 0;                        // tiles and blocks of this CTA so far: block b is use b / regions of region b % regions
      bool ok = true;
      for (int tile = pair; tile < n_tiles && ok; tile += n_pairs, ++tc) {
        const int units = blocks_of(tile).units;
        const bool mine = u < units;
        // (The ring has at most as many stages as a tile k steps: when one warp starts a tile the other is past its wait for a
        // region of the tile before, so a region's barrier is never two uses behind.)
        const uint32_t use = (blk + (uint32_t)u) / (uint32_t)a.regions, reg = blk + (uint32_t)u - use * (uint32_t)a.regions;
        const uint32_t d = tmem_base + reg * (uint32_t)a.reg_cols;
        blk += (uint32_t)units;
        uint32_t id0 = 0;
        for (int kt = 0; kt < KT; ++kt) {
          ok = __all_sync(0xFFFFFFFFu, mbar_wait(BAR_SF(s), ph, ctl, 612));
          if (!ok) break;
          if (mine) {
            if (kt == 0) {
              id0 = pair_idesc(__shfl_sync(0xFFFFFFFFu, s_cols[tc & 7u], 0) * (FORM == PP_SIDE ? 2 : 1), 0);     // left by the scale loader
              ok = __all_sync(0xFFFFFFFFu, mbar_wait(BAR_ACC_EMPTY(reg), (use & 1u) ^ 1u, ctl, 613));
              if (!ok) break;
            }
            tc_fence_after();
            const uint32_t st = sbase + s * (uint32_t)a.stage_bytes;
            const uint32_t sf = tmem_base + SF_BASE + s * SF_COLS<FORM>;
            const uint32_t a_lo = DESC_LO | ((st + (uint32_t)u * (128 * 128)) >> 4);
            const uint32_t b_lo = DESC_LO | ((st + OFF_X) >> 4);
            const int kk_live = kt < k_whole ? 4 : (p.K - kt * 128 + 31) >> 5;
            auto mma = [&](int kk, int c) {
              mma_mxf8f6f4_pair<A_HI, B_HI>(d, a_lo + kk * A_KK, b_lo + c * (1024 >> 4) + kk * 2, id0 + ((uint32_t)kk << 4) + ((uint32_t)kk << 29),
                                            sf + 4 * u, sf + 8 + 8 * c, (kk | c) ? 1u : (uint32_t)(kt > 0));
            };
            // (a step that is whole has no test between its instructions: they must issue in less than the 45-64 cycles that
            // one of them runs)
            if (kk_live == 4) {
#pragma unroll
              for (int kk = 0; kk < 4; ++kk)
#pragma unroll
                for (int c = 0; c < MMAS; ++c) mma(kk, c);
            } else {
#pragma unroll
              for (int kk = 0; kk < 4; ++kk)
                if (kk < kk_live) {
#pragma unroll
                  for (int c = 0; c < MMAS; ++c) mma(kk, c);
                }
            }
          }
          elect_commit_pair(BAR_EMPTY(s));
          if (++s == (uint32_t)STAGES) { s = 0; ph ^= 1u; }
        }
        if (ok && mine) elect_commit_pair(BAR_ACC_FULL(reg));
      }
      // every MMA issued by these warps has retired before tensor memory is freed
      elect_commit_pair_local(BAR_DRAIN);
      mbar_wait(BAR_DRAIN, 0, ctl, 614);
    }
    __syncwarp();
  } else if (warp < PP_SF_WARP0) {
    // (fills the warpgroup)
  } else if (warp < PP_EPI_WARP0) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_SF));
    // ================================= scale loaders ==================================================
    // lane l of every lane quarter holds rows l, l + 32, ... of each block of scales: four columns per weight block, one per
    // 32 tokens and term (words are one row's four k groups, rows in order).
    const int qd = warp & 3;
    uint32_t s = 0, ph = 0, tc = 0;
    bool ok = true;
    PTile t, nxt;
    if (pair < n_tiles) nxt = map_ptile(p, s_prefix, pair / MT);
    for (int tile = pair; tile < n_tiles && ok; tile += n_pairs, ++tc) {
      t = nxt;
      if (warp == PP_SF_WARP0 && lane == 0) s_cols[tc & 7u] = t.cols;     // read by the MMA warp after the first SF wait
      for (int kt = 0; kt < KT; ++kt) {
        ok = __all_sync(0xFFFFFFFFu, mbar_wait(BAR_FULL(s), ph, ctl, 615));
        if (!ok) break;
        const uint32_t st = sbase + s * (uint32_t)a.stage_bytes;
        const uint32_t taddr = tmem_base + ((uint32_t)(qd * 32) << 16) + SF_BASE + s * SF_COLS<FORM>;
        uint4 w0, w1;
        if constexpr (TILED) {                         // [row][4 groups], rows in the order the operand has them
          const uint32_t ws = st + OFF_WS + (uint32_t)tiled_row(lane) * 4u;
          w0 = make_uint4(lds32(ws), lds32(ws + 128u), lds32(ws + 256u), lds32(ws + 384u));
          w1 = make_uint4(lds32(ws + 512u), lds32(ws + 640u), lds32(ws + 768u), lds32(ws + 896u));
        } else {
          w0 = lds128(st + OFF_WS + (uint32_t)lane * 16u);
          w1 = lds128(st + OFF_WS + 512u + (uint32_t)lane * 16u);
        }
        uint32_t x[MMAS][8];
        const int n_cols = FORM == PP_SIDE ? 2 * t.cols : t.cols;
#pragma unroll
        for (int c = 0; c < MMAS; ++c)
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int n = 32 * i + lane;               // column; TWO: eight hi words, eight lo words, ...
            x[c][i] = 0;
            if (32 * i < n_cols) x[c][i] = lds32(st + OFF_XS + (uint32_t)(FORM == PP_TWO ? (n >> 3) * 64 + c * 32 + (n & 7) * 4 : n * 4));
          }
        asm volatile(
            "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
            "r"(w0.x), "r"(w0.y), "r"(w0.z), "r"(w0.w), "r"(w1.x), "r"(w1.y), "r"(w1.z), "r"(w1.w), "r"(x[0][0]), "r"(x[0][1]),
            "r"(x[0][2]), "r"(x[0][3]), "r"(x[0][4]), "r"(x[0][5]), "r"(x[0][6]), "r"(x[0][7])
            : "memory");
        if constexpr (FORM == PP_TWO)
          asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr + 16u), "r"(x[1][0]),
                       "r"(x[1][1]), "r"(x[1][2]), "r"(x[1][3]), "r"(x[1][4]), "r"(x[1][5]), "r"(x[1][6]), "r"(x[1][7])
                       : "memory");
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(BAR_SF(s), 0);
        if (++s == (uint32_t)STAGES) { s = 0; ph ^= 1u; }
        if (kt == 0 && tile + n_pairs < n_tiles) nxt = map_ptile(p, s_prefix, (tile + n_pairs) / MT);
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS_EPI));
    // ================================= epilogue =======================================================
    // The warps of a lane quarter take the 16-token chunks of a unit in turn.
    const int ew = warp - PP_EPI_WARP0, qd = warp & 3, grp = ew >> 2;
    const int tid = threadIdx.x - PP_EPI_WARP0 * 32;
    const int own = TILED ? tiled_row(lane) : lane;    // weight row of this lane inside its quarter
    const int odd = own & 1;
    const uint32_t sel = odd ? 0x3276u : 0x5410u;
    const bool swiglu = p.activation == MOE_ACT_SWIGLU;
    const bool vec = p.ld_y % 2 == 0 && (uintptr_t)p.y % (2 * sizeof(TY)) == 0;
    uint32_t tc = 0;
    uint32_t acc_ph = 0, reg = 0;                      // parity to wait for, per region; region of the next block
    // (two warps to a group of 32 outputs, see emit_tokens)
    const int half = qd >> 1, tok_pair = grp * 2 + half;
    const TokStage tok{ctl0 + PP_CTL_BASE + (uint32_t)(tok_pair * TOK_STAGE), 2 + tok_pair, (qd & 1) * 32 + lane};
    // 16 tokens of block b, from the raw sums
    auto emit = [&](const PairOut& out, const uint32_t (&sums)[16], uint32_t tab, int c, int block) {
      if constexpr (TOK_TERMS<TY> != 0) {
        if (block >= NB) return;                       // (both warps of the pair)
        float y[8];
        swiglu_chunk(p, sums, out.bias, odd, y);
        stage_tokens<TY>(tok.at, y, 8 * odd, ((qd & 1) << 4) + (own >> 1));
        tok.sync();
        const int token = tok.i >> 2, l4 = tok.i & 3;
        const StagedRow row = staged_row<TY>(tok.at, token, l4);
        tok.sync();                                    // the stage may be written again
        const uint32_t at = tab + (uint32_t)(c + token) * 8u;
        const uint2 q = lds64(at), s = lds64(at + 2048u);
        emit_group<TY>(a.out, row, l4, token & 7, 2 * block + half, (uint8_t*)(((uint64_t)q.y << 32) | q.x),
                       (uint8_t*)(((uint64_t)s.y << 32) | s.x), block == NB - 1 && 2 * NB + half < 4 * a.out.KT);
      } else {
        pair_emit<TY>(p, out, sums, tab, c);
      }
    };
    bool ok = true;
    for (int tile = pair; tile < n_tiles && ok; tile += n_pairs, ++tc) {
      const PTile t = map_ptile(p, s_prefix, tile / MT);
      const Blocks b = blocks_of(tile);
      const uint32_t tab = ctl0 + (tc & 1u) * PAIR_TAB;
      if (tid < t.cols) {
        bool stored = tid < t.rows;                    // not by the pack kernel
        if (TERMS == 2 && stored && a.done) stored = !a.done[padded_base(t.e, t.off) + t.first + tid];
        if constexpr (TOK_TERMS<TY> != 0) {            // line and scales of the row as the next product's token, in place of row and weights
          uint8_t *q = nullptr, *s = nullptr;
          if (stored) token_addr(a.out, t.e, t.off, p.slice_sizes[t.e], a.out.tb ? a.out.block_offs[t.e] : 0, t.first + tid, q, s);
          asm volatile("st.shared.u64 [%0], %1;" ::"r"(tab + (uint32_t)tid * 8u), "l"(q) : "memory");
          asm volatile("st.shared.u64 [%0], %1;" ::"r"(tab + 2048u + (uint32_t)tid * 8u), "l"(s) : "memory");
        } else {
          pair_table_entry<TY>(p, t, tid, stored, tab);
        }
      }
      float bias_m[2];
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int n = (b.first + m) * 128 + qd * 32 + own;
        bias_m[m] = (p.bias && n < p.N) ? load_bias(p.bias, p.bias_dtype, (int64_t)t.e * p.ld_bias + n) : 0.0f;
      }
      asm volatile("bar.sync 1, %0;" ::"n"(PP_EPI_WARPS * 32) : "memory");
#pragma unroll 1
      for (int u = 0; u < b.units; ++u) {
        const int ne = (b.first + u) * 128 + qd * 32 + (own & ~1);      // first of the lane pair's two columns
        const bool first = ne < p.N, both = ne + 1 < p.N;
        const PairOut out{ne, first, both, __all_sync(0xFFFFFFFFu, both && (swiglu || vec)) != 0, odd, sel, u ? bias_m[1] : bias_m[0]};
        ok = __all_sync(0xFFFFFFFFu, mbar_wait(BAR_ACC_FULL(reg), (acc_ph >> reg) & 1u, ctl, 616));
        if constexpr (TOK_TERMS<TY> != 0) ok = tok.all(ok);
        if (!ok) break;
        acc_ph ^= 1u << reg;
        tc_fence_after();
        const uint32_t taddr = tmem_base + ((uint32_t)(qd * 32) << 16) + reg * (uint32_t)a.reg_cols;
        // The warp's share of the region (up to four chunks at a time) goes to registers and the region back to the MMA warp
        // before any of it is worked on: drained chunk by chunk, the tensor pipe waited 3000-4600 cycles for the first region of
        // every tile.
        constexpr int STEP = 4 * PP_EPI_WARPS;         // columns from one chunk of a warp to its next
        constexpr int BATCH = FORM == PP_SIDE ? 2 : 4;
#pragma unroll 1
        for (int c0 = grp * 16; c0 < t.rows || c0 == grp * 16; c0 += BATCH * STEP) {
          constexpr int W = FORM == PP_SIDE ? 32 : 16;
          uint32_t raw[BATCH][W];
#pragma unroll
          for (int i = 0; i < BATCH; ++i)
            if (c0 + STEP * i < t.rows) {
              if constexpr (FORM == PP_SIDE) tmem_ld32(taddr + (uint32_t)(2 * (c0 + STEP * i)), raw[i]);
              else tmem_ld16(taddr + (uint32_t)(c0 + STEP * i), raw[i]);
            }
          tmem_ld_wait();
          if (c0 + BATCH * STEP >= t.rows) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(BAR_ACC_EMPTY(reg), 0);
          }
#pragma unroll
          for (int i = 0; i < BATCH; ++i)
            if (c0 + STEP * i < t.rows) {
              if constexpr (FORM == PP_SIDE) {
                uint32_t v[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                  const int at = (j >> 3) * 16 + (j & 7);
                  v[j] = __float_as_uint(__uint_as_float(raw[i][at]) + __uint_as_float(raw[i][at + 8]));
                }
                emit(out, v, tab, c0 + STEP * i, b.first + u);
              } else {
                emit(out, raw[i], tab, c0 + STEP * i, b.first + u);
              }
            }
        }
        if (++reg == (uint32_t)a.regions) reg = 0;
      }
    }
    // aborting: a warp that is a tile ahead may be at the table barrier
    if (!ok) asm volatile("bar.arrive 1, %0;" ::"n"(PP_EPI_WARPS * 32) : "memory");
  }

  // ---- teardown ----------------------------------------------------------------------------------------
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                                  // neither CTA's memories go away while the other still works
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)TMEM_COLS) : "memory");
  }
}

// ---- host side -----------------------------------------------------------------------------------------------
struct PairPlan {
  int KT, NB, terms;
  int64_t prows, xs_off, done_off, ws_bytes;
};

PairPlan pair_plan(const MoeGemmArgs& a) {
  PairPlan pl;
  pl.KT = (int)cdiv64(a.K, 128);
  pl.NB = (int)cdiv64(a.N, 128);
  pl.terms = a.x_dtype == MOE_BF16 ? 2 : 1;
  const int64_t E = a.slice_sizes ? a.E : 1;
  pl.prows = cdiv64(a.M, 32) * 32 + 32 * (E + 1);
  pl.xs_off = pl.terms * pl.KT * pl.prows * 128;
  pl.done_off = pl.xs_off + pl.terms * pl.KT * pl.prows * 4;
  pl.ws_bytes = pl.done_off + pl.prows * 4;
  return pl;
}

// Token columns and weight blocks of a tile, and the form of two-term tokens.  fc1 + fc2, us:
// - SIDE with 96 columns of tokens below 56 rows per expert, TWO with 128 from there on (32 experts of 2880 x 5760: 50 rows 176
//   and 180, 80 rows 219 and 197, 150 rows 305 and 293, 300 rows 489 and 457; 128 experts, 512 rows: 3157 and 2978).  SIDE with 64
//   columns reads the weight operand more often and is 0-20 % slower from 32 rows on; TWO with 192 has no third region to go on in
//   while a tile is drained (150 rows: 336, 512 rows: 3349).
// - One weight block per tile where twice the tiles still run at a time (8 experts of 512 x 2048, 16 rows: 19 -> 17); beyond, a
//   tile of two blocks reads the tokens once for both (32 experts, 64 rows: 91 against 105).
struct PairShape { int nmax, upt, form; };
// mean rows per expert: what the caller expects, else the bound on the rows over the experts
int64_t mean_rows(const MoeGemmArgs& a) {
  const int64_t mean = a.M / (a.slice_sizes ? a.E : 1);
  return a.rows_per_expert > 0 && a.rows_per_expert < mean ? a.rows_per_expert : mean;
}

PairShape pair_shape(const MoeGemmArgs& a, int terms) {
  const int64_t experts = a.slice_sizes ? a.E : 1, per = mean_rows(a);
  PairShape s;
  s.form = terms == 1 ? PP_ONE : (per < 56 ? PP_SIDE : PP_TWO);
  s.nmax = s.form == PP_SIDE ? 96 : s.form == PP_TWO ? 128 : 192;
  const int64_t active = experts < a.M ? experts : a.M;
  s.upt = active * (per / s.nmax + 1) * cdiv64(a.N, 256) <= moe_sm_count() / 2 ? 1 : 2;
  return s;
}

template <typename TY, int FORM, bool TILED, bool ONCE = false>
int launch_mx_pair(const GemmParams& p, PairParams q, const PairShape& shape, const MoeGemmArgs& args, const PairMaps& maps,
                   cudaStream_t st) {
  auto kernel = gemm_mx_pair_kernel<TY, FORM, TILED, ONCE>;
  q.nmax = shape.nmax; q.upt = shape.upt;
  q.reg_cols = q.nmax * (FORM == PP_SIDE ? 2 : 1);
  q.stage_bytes = q.upt * 128 * 128 + TERMS_OF<FORM> * (q.nmax * 64 + 1024) + 1024;
  q.stages = (PP_SMEM - 1024 - PP_CTL<TY>) / q.stage_bytes;
  if (q.stages > PP_MAX_STAGES) q.stages = PP_MAX_STAGES;
  while ((TMEM_COLS - q.stages * SF_COLS<FORM>) / q.reg_cols < 2) --q.stages;
  if (q.stages > q.KT) q.stages = q.KT;               // see the MMA warps
  q.regions = (TMEM_COLS - q.stages * SF_COLS<FORM>) / q.reg_cols;
  if (q.regions > PP_MAX_REGIONS) q.regions = PP_MAX_REGIONS;
  MOE_CHECK_ARG(q.stages >= 1, "moe_grouped_gemm: block-scaled pair tile does not fit shared memory");
  // every expert has at most ceil(rows / nmax) token tiles
  const int64_t experts = args.slice_sizes ? (args.E < args.M ? args.E : args.M) : 0;
  const int64_t tiles = (experts + cdiv64(args.M, q.nmax)) * cdiv64(cdiv64(q.NB, 2), q.upt);
  const int idle_sms = args.idle_sms > 0 ? args.idle_sms : 0;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(PP_THREADS, 1, 1);
  cfg.dynamicSmemBytes = PP_SMEM;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at; cfg.numAttrs = 1;                    // (the occupancy query has no use for the second)
  // per device: opt in to the shared-memory size once, and ask how many pairs can be resident at a time
  static std::mutex mu;
  static int max_pairs[64] = {0};
  int dev = 0;
  MOE_CHECK_CUDA(cudaGetDevice(&dev));
  MOE_CHECK_ARG(dev < 64, "moe_grouped_gemm: device index %d out of range", dev);
  int resident;
  {
    std::lock_guard<std::mutex> lk(mu);
    if (max_pairs[dev] == 0) {
      MOE_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PP_SMEM));
      cfg.gridDim = dim3(2 * (unsigned)(moe_sm_count() / 2), 1, 1);
      int n = 0;
      MOE_CHECK_CUDA(cudaOccupancyMaxActiveClusters(&n, kernel, &cfg));
      max_pairs[dev] = n > 0 ? n : -1;
    }
    resident = max_pairs[dev];
  }
  if (resident <= 0) {
    moe_set_error("moe_grouped_gemm: no pair of SMs can hold the cluster kernel on this device");
    return MOE_ERR_UNSUPPORTED;
  }
  int64_t pairs = resident - (idle_sms + 1) / 2;
  if (pairs < 1) pairs = 1;
  if (tiles < pairs) pairs = tiles;
  cfg.gridDim = dim3((unsigned)(2 * pairs), 1, 1);
  cfg.numAttrs = 2;
  moe_count_launch();
  MOE_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kernel, p, q, maps));
  return MOE_OK;
}

// TY: output rows, or the next product's tokens
template <typename TY>
int launch_mx_pair_ty(const GemmParams& p, const PairParams& q, const MoeGemmArgs& a, const PairMaps& m, cudaStream_t st) {
  const PairShape shape = pair_shape(a, a.x_dtype == MOE_BF16 ? 2 : 1);
  if constexpr (sizeof(TY) > 1) {
    // Weights read about once: up to an eighth of a tile of rows per expert (with a fifth and biased routing the other tiles of an expert would miss
    // what the first has read, 336 us -> 350).  us per step of the operators: 16 tokens of 32 experts 108.2 -> 100.8, 64 tokens of 128 experts 200 -> 194,
    // 200 tokens of 128 experts of 1440 120 -> 110.  (The block-scaled copy leaves so few rows to the decode kernel.)
    const int64_t experts = a.slice_sizes ? a.E : 1;
    if (a.w_kind == MOE_W_MX4_B200 && shape.form == PP_SIDE && 8 * a.M <= shape.nmax * experts)
      return launch_mx_pair<TY, PP_SIDE, true, true>(p, q, shape, a, m, st);
    if (a.w_kind == MOE_W_MX4_B200)
      return shape.form == PP_SIDE ? launch_mx_pair<TY, PP_SIDE, true>(p, q, shape, a, m, st) : launch_mx_pair<TY, PP_TWO, true>(p, q, shape, a, m, st);
  }
  // (a product hands its rows on in the form its own tokens have)
  if constexpr (TOK_TERMS<TY> != 1) {
    if (shape.form == PP_SIDE) return launch_mx_pair<TY, PP_SIDE, false>(p, q, shape, a, m, st);
    if (shape.form == PP_TWO) return launch_mx_pair<TY, PP_TWO, false>(p, q, shape, a, m, st);
  }
  if constexpr (TOK_TERMS<TY> != 2) return launch_mx_pair<TY, PP_ONE, false>(p, q, shape, a, m, st);
  return MOE_ERR_UNSUPPORTED;
}

}  // namespace

// Where the pair form is the faster one (us, fc1 + fc2 unless said; balanced routing unless said).  `load` is what one pass over the
// weights of the experts in use costs, in elements.
// Default tiles (against the bf16 tensor-core kernel, above ten or so rows also against the streaming one), kernel "mx" asks
// for it: the pack pass and the cluster launch want 2^24 elements and 2^28 products a token row to be repaid, and a product
// over fewer than 2560 weight rows stays ahead up to 512 rows per expert only.
//   32 experts of 2880 x 5760:  8 rows 141 (streaming: 235), 64 rows 170 (272), 150 rows 289 (379), 1024 rows 1515 (1564)
//   64 experts of 1024 x 1536:  4 rows 55 (75), 16 rows 53 (86), 64 rows 69 (82), 256 rows 144 (146)
//   16 experts of 1440 x 1472:  64 rows 38 (43), 256 rows 61 (53), logits biased by N(0, 1) per expert 62 (79), 1024 rows 151 (135)
// Wide SwiGLU products over few k are bound by this kernel's epilogue and stay with the bf16 kernel from 512 rows on (512 x 4096, 8
// experts of 1024 rows: 72 here, 57 there; 16 experts 132 and 109; without the activation 64 and 61, 114 and 116).
// (Both kernels lose up to a third of a wave, so no line in these sizes is right everywhere: over 500 products of 48 to 1024 rows
// this one is 2 % from the better kernel on average, most of it at 100-400 balanced rows of K <= 1024.)
// Block-scaled tiles (against the decode forms of gemm_mx.cu), tile_m = 256 asks for it.  bf16 tokens from 20 rows per expert on, e4m3 tokens from 16.
// What an expert has decides the time, not the mean: under logits biased by N(0, 1) per expert some experts have several blocks of the decode form.  The
// lines were drawn before the decode form's tiles of two blocks, with which it is ahead of this one to some 25 rows where the product's tiles here
// are between one and eight rounds of the pairs (a last round partly filled costs a good part of the whole then).  bf16 products stay here all the same: a token
// with an infinity gives infinities here, and large finite values there.  For e4m3 tokens the line has not been moved.  Whole layer steps,
// four picks (decode form, this one; even, then biased):
//   bf16   128 experts of 2880 x 5760:  20 rows 429, 452; 377, 357.  24 rows 449, 437; 436, 391
//          32 experts of the same:  20 rows 109, 131; 123, 129.  25 rows 118, 134; 133, 131.  30 rows 135, 138; 141, 136.  40 rows 172, 143; 164, 149
//          64 experts of 1440 x 2880:  20 rows 86, 96; 81, 88.  25 rows 84, 95; 94, 94.  32 rows 101, 98; 102, 97
//          a product of 64 experts of 736 x 1440:  20 rows 26, 23; 29, 23.  24 rows 28, 24; 34, 25
//   e4m3   128 experts of 2880 x 5760:  16 rows 359, 397; 307, 287.  20 rows 361, 396; 338, 295.  24 rows 376, 406; 377, 314
//          32 experts of the same:  16 rows 102, 129; 100, 121.  25 rows 110, 131; 122, 127.  32 rows 130, 133; 135, 132
//          64 experts of 1440 x 2880:  16 rows 77, 91; 75, 80.  25 rows 79, 91; 87, 89
// Small ones (products with their token packs) once the decode kernel's tiles of 32 rows x 128 weight rows (half a block lost per expert) are more than a wave, up to
// which it takes one tile's time: a product of 32 experts of 512 x 512, 16 rows 10 there, 11 here, 64 rows 21 and 13; 8 experts of
// 512 x 2048, 16 rows 9 and 11, 80 rows 20 and 13; of 2048 x 512, 96 rows 17 and 21.
bool moe_gemm_mx_pair_wanted(const MoeGemmArgs& a) {
  if (a.slice_sizes && a.E > MAX_PREFIX_EXPERTS) return false;
  if (a.M >= (1ll << 31) - (1 << 20) || a.kernel == MOE_GEMM_MX_F4 || a.tile_n != 0) return false;
  const int64_t experts = a.slice_sizes ? a.E : 1, per = mean_rows(a);
  const int64_t load = (experts < a.M ? experts : a.M) * a.N * a.K;
  if (a.w_kind == MOE_W_MX4_B200) {
    // default tiles, bf16 tokens
    if (a.x_dtype != MOE_BF16 || (a.y_dtype != MOE_BF16 && a.y_dtype != MOE_F32) || (uintptr_t)a.w % 32 != 0 ||
        (uintptr_t)a.w_scale % 16 != 0 || (uintptr_t)a.x % 16 != 0 || a.ld_x % 8 != 0 ||
        (int64_t)a.E * cdiv64(a.K, 128) * cdiv64(a.N, 128) >= 2147483647LL)
      return false;
    if (a.kernel == MOE_GEMM_MX) return true;
    if (a.kernel != MOE_GEMM_AUTO || a.tile_m != 0) return false;
    const bool wide = a.N >= 2560 && !(a.activation == MOE_ACT_SWIGLU && a.K < 1024);
    return load >= (1 << 24) && (per > 0 ? per : 1) * load >= (1 << 28) && (wide || per < 512);
  }
  if (a.tile_m == 256) return true;
  if (a.tile_m != 0 || a.kernel == MOE_GEMM_MX_F8) return false;
  if (a.x_dtype != MOE_BF16) return per >= 16;
  if (load >= (1 << 24)) return per >= 20;
  return experts * (per + 16) / 32 * cdiv64(a.N, 128) > moe_sm_count();
}

int64_t moe_gemm_mx_pair_workspace(const MoeGemmArgs& a) { return pair_plan(a).ws_bytes; }

bool moe_gemm_mx_pair_token_out(const MoeGemmArgs& a, TokenOut& o) {
  const PairPlan pl = pair_plan(a);
  if (a.mx_workspace == nullptr || a.mx_workspace_bytes < pl.ws_bytes) return false;
  o.q = (uint8_t*)a.mx_workspace; o.s = o.q + pl.xs_off;
  o.q_step = pl.terms * pl.prows * 128; o.s_step = pl.terms * pl.prows * 4;
  o.terms = pl.terms; o.permuted = a.w_kind == MOE_W_MX4_B200; o.KT = pl.KT;
  return true;
}

int moe_gemm_mx_pair_launch(const GemmParams& p_in, const MoeGemmArgs& a, const TokenOut& out, bool packed, cudaStream_t st) {
  const PairPlan pl = pair_plan(a);
  MOE_CHECK_ARG(a.mx_workspace != nullptr && a.mx_workspace_bytes >= pl.ws_bytes && (uintptr_t)a.mx_workspace % 1024 == 0,
                "moe_grouped_gemm: the block-scaled kernel needs mx_workspace of moe_gemm_mx_workspace_bytes() = %lld "
                "bytes, 1024-byte aligned (got %lld)", (long long)pl.ws_bytes, (long long)a.mx_workspace_bytes);
  GemmParams p = p_in;
  int64_t blocks16;
  if (a.slice_sizes) {
    p.block_offs = a.block_offs_16;
    p.block_sched = a.block_sched_16;
    blocks16 = a.M <= a.E ? a.M : a.E - 1 + cdiv64(a.M + 1 - a.E, 16);
  } else {
    blocks16 = cdiv64(a.M, 16);
  }
  PairPackParams pk;
  pk.x = a.x; pk.ld_x = a.ld_x; pk.rows_x = a.rows_x;
  pk.x_scale = a.x_scale; pk.ld_xs = a.ld_x_scale;
  pk.gather = a.gather_indx;
  pk.K = a.K; pk.KT = pl.KT; pk.NB = pl.NB; pk.y_dtype = a.y_dtype; pk.prows = pl.prows;
  pk.xq = (uint8_t*)a.mx_workspace; pk.xs = pk.xq + pl.xs_off; pk.done = (uint32_t*)(pk.xq + pl.done_off);
  const bool tiled = a.w_kind == MOE_W_MX4_B200;
  pk.out = out;
  pk.positions = nullptr; pk.experts = nullptr; pk.k = 0;
  if (!packed) {
    // by rows of x where every one of them has its k positions, several (and no more than a block has shared memory for), and their blocks
    // fill the SMs (256 rows, two positions each: 27.6 us per layer step by position, 28.1 by row)
    if (a.x_positions && a.x_experts && a.x_k > 1 && a.x_k <= PACK_MAX_K && a.slice_sizes && a.rows_x * a.x_k == a.M &&
        a.rows_x >= (int64_t)PACK_TOKENS * moe_sm_count()) {
      pk.positions = a.x_positions; pk.experts = a.x_experts; pk.k = a.x_k;
      auto pack = pl.terms == 1 ? mx_pair_pack1_rows_kernel : tiled ? mx_pair_pack2_rows_kernel<true> : mx_pair_pack2_rows_kernel<false>;
      MOE_CHECK_CUDA(launch_pdl(pack, dim3((unsigned)cdiv64(a.rows_x, PACK_TOKENS)), dim3(256),
                                pl.terms == 1 ? 0 : (size_t)PACK_TOKENS * a.x_k * sizeof(int64_t), st, p, pk));
    } else {
      // Blocks of 16 rows in parts of a turn or two of their threads, where whole ones are less than the three that an SM holds (512 deep, four k
      // steps: 29.4 us whole, 30.1 in four).  us of a product of 1024 columns with its pass, whole and in parts: 32 experts, 2880 deep, 1024 rows (95 blocks) 34.9, 23.9;
      // 2400 (182) 40.0, 31.9; 4800 (331) 54.9, 51.6; 9600 (631) 78.4, 79.1; 16000 (1031) 113, 116; 64000 432, 478; 1440 deep, 4800 rows 34.3, 34.2; 7200 (481) 38.1,
      // 39.8; 32000 118, 124; 128 experts, 1440 deep, 2400 rows (278) 44.4, 42.1; 4800 (427) 48.2, 49.3.
      const int parts = pl.terms == 1 || 2 * blocks16 > 5 * (int64_t)moe_sm_count() ? 1 : pl.KT >= 16 ? 4 : pl.KT >= 8 ? 2 : 1;
      auto pack = pl.terms == 1 ? mx_pair_pack1_kernel : tiled ? pack2_in_parts<true>(parts) : pack2_in_parts<false>(parts);
      MOE_CHECK_CUDA(launch_pdl(pack, dim3((unsigned)(blocks16 * parts)), dim3(256), 0, st, p, pk));
    }
    MOE_CHECK_LAUNCH();
  }
  PairParams q;
  q.out = out;
  q.xq = pk.xq; q.xs = pk.xs; q.done = packed ? nullptr : pk.done; q.prows = pl.prows; q.KT = pl.KT; q.NB = pl.NB;
  PairMaps maps;
  for (int n = 1; n <= 2; ++n) {
    // values as the TMA unit expands them (a row of a box: 64 bytes -> 128), scales as words; blocks along the slowest dimension
    // (default tiles) or the one before (block-scaled tiles)
    const cuuint64_t d2 = tiled ? pl.KT : pl.NB, d3 = (cuuint64_t)a.E * (tiled ? pl.NB : pl.KT);
    const cuuint32_t b2 = tiled ? 1 : n, b3 = tiled ? n : 1;
    const cuuint64_t wd[4] = {128, 128, d2, d3}, wst[3] = {64, 8192, 8192 * d2};
    const cuuint32_t wb[4] = {128, 128, b2, b3};
    if (int rc = encode_map(&maps.w[n - 1], CU_TENSOR_MAP_DATA_TYPE_16U4_ALIGN16B, 4, a.w, wd, wst, wb, CU_TENSOR_MAP_SWIZZLE_128B,
                            "packed e2m1 weights"))
      return rc;
    const cuuint64_t sd[3] = {128, d2, d3}, sst[2] = {512, 512 * d2};
    const cuuint32_t sb[3] = {128, b2, b3};
    if (int rc = encode_map(&maps.s[n - 1], CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, a.w_scale, sd, sst, sb, CU_TENSOR_MAP_SWIZZLE_NONE, "weight scales"))
      return rc;
  }
  if (out.q) return out.terms == 1 ? launch_mx_pair_ty<Tok1>(p, q, a, maps, st) : launch_mx_pair_ty<Tok2>(p, q, a, maps, st);
  if (a.y_dtype == MOE_BF16) return launch_mx_pair_ty<__nv_bfloat16>(p, q, a, maps, st);
  if (a.y_dtype == MOE_F32) return launch_mx_pair_ty<float>(p, q, a, maps, st);
  MOE_CHECK_ARG(!tiled, "moe_grouped_gemm: e4m3 output needs weights in the block-scaled layout");
  return launch_mx_pair_ty<__nv_fp8_e4m3>(p, q, a, maps, st);
}
