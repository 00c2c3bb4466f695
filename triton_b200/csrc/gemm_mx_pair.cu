// Ragged grouped GEMM on the block-scaled tensor-core path for many rows per expert (prefill, mid-sized batches):
// e2m1 weights with their e8m0 scales x e4m3 tokens, tcgen05.mma.cta_group::2.kind::mxf8f6f4 on pairs of SMs.
//
// bf16 tokens enter as two e4m3 terms, hi = mxfp8(x) and lo = mxfp8(x - hi), each with its own e8m0 scale per 32 k (exact up
// to underflow: a bf16 value has 8 significant bits, each term holds 4); both terms accumulate into the same fp32 columns.
// e4m3 / MXFP8 tokens are one term.  Nothing is dequantised in software, and the MMA pipe does K = 32 per instruction in the
// time kind::f16 does K = 16 (measured: 4.4 PFLOP/s for N >= 128 on 148 SMs, so two terms run at 2.2 -- the bf16 rate).
//
// What bounds it.  An SM takes in at most about 26 B per cycle from L2, and the MMA of a 128-k step is 64 cycles per 128
// token columns, weight block and K = 32: the tile has to be large.  A cluster of two CTAs computes (2 x 256 weight rows) x
// (up to 224 tokens; 192 with two terms): the weights are the M operand (every CTA loads its own 128 rows of each of the
// two 256-row blocks, packed in global memory: 16 KB per step), the tokens the N operand (every CTA loads half of them:
// 14 or 24 KB), 26-34 B per MMA cycle.  Tokens on N also make a ragged tail cost what it holds, in steps of 32 rows, where
// tokens on M padded every expert to a multiple of 128 or 256 (31 % of the rows of a skewed 128-expert batch of 16384
// tokens).
//
// A tile's accumulator is two units (its 256-row weight blocks), and each is handed to the epilogue and back by itself: the
// next tile starts on the unit that is drained while the other still is (the MMA warp lets a unit lag by at most the stages
// of the ring).  One accumulator of 448 columns drained as a whole would leave the tensor pipe idle for the time of an
// epilogue on every tile; two buffers of it do not fit tensor memory.  (Four units, halves of the columns each, drain in
// finer steps but read the weight operand twice: 59 cycles for an MMA of 96 columns against 96 for one of 192.)
//
// Warps of a CTA: 0 producer (one thread), 1 MMA issue (even CTA) and tensor-memory owner, 4-7 scale loaders (shared memory ->
// registers -> tensor memory; the token scales of all columns in both CTAs, the weight scales of the own rows), 8-19 epilogue.
// Every wait is bounded; both CTAs meet at a cluster barrier before tensor memory is freed.
#include "gemm_mx_common.cuh"
#include "gemm_pair_common.cuh"

namespace {

constexpr int PP_SF_WARP0 = 4, PP_EPI_WARP0 = 8, PP_EPI_WARPS = 12;
// Registers: 640 threads start with 96 each (61440); the warpgroups of producer + MMA and of the scale loaders give some up
// for the epilogue's: 128 x (56 + 64) + 384 x 120 = 61440.
constexpr int REGS_ISSUE = 56, REGS_SF = 64, REGS_EPI = 120;
static_assert(128 * (REGS_ISSUE + REGS_SF) + PP_EPI_WARPS * 32 * REGS_EPI <= 96 * 640, "register split");
constexpr int PP_THREADS = (PP_EPI_WARP0 + PP_EPI_WARPS) * 32;

template <int TERMS> struct PCfg {
  static constexpr int NMAX = TERMS == 1 ? 224 : 192;        // token columns of a tile
  static constexpr int STAGES = TERMS == 1 ? 4 : 3;
  static constexpr int X_TERM = NMAX / 2 * 128;              // bytes of a CTA's half of the tokens, one term
  static constexpr int OFF_X = 2 * 128 * 128;                // two weight blocks, byte per element
  static constexpr int OFF_WS = OFF_X + TERMS * X_TERM;      // their scales
  static constexpr int OFF_XS = OFF_WS + 1024;               // token scales of all columns (256 words per term)
  static constexpr int STAGE = OFF_XS + TERMS * 1024;
  static constexpr int SF_BASE = 2 * NMAX, SF_COLS = 8 + 8 * TERMS;
  static constexpr int TAB = 256 * 16;                       // token table of a tile: row address [256], gamma [256], beta [256]
  static constexpr int OFF_TAB = STAGES * STAGE;             // two of them
  static constexpr int OFF_BAR = OFF_TAB + 2 * TAB;
  static constexpr int NUM_BARS = 3 * STAGES + 4 + 1;
  static constexpr int EPI_CHUNKS = (NMAX / 16 + 2) / 3;      //  16-token chunks of a unit per epilogue warp (three warps share a lane quarter)
  static constexpr int OFF_MISC = OFF_BAR + NUM_BARS * 8 + (NUM_BARS % 2) * 8;
  static constexpr int OFF_COLS = OFF_MISC + 16;             // columns of the next tiles, for the MMA warp
  static constexpr int OFF_PREFIX = OFF_COLS + 8 * 4;        // int32 tile prefix over experts, their row counts and offsets
  static constexpr int ALLOC = OFF_PREFIX + (3 * MAX_PREFIX_EXPERTS + 1) * 4 + 1024;
  static_assert(STAGE % 1024 == 0 && X_TERM % 1024 == 0, "operand tiles start on swizzle atoms");
  static_assert(SF_BASE + STAGES * SF_COLS <= TMEM_COLS && ALLOC <= 232448, "budgets");
};

struct PairParams {
  const uint8_t* xq;            // [term][k step][padded row][128 B], 16-byte pieces swizzled with (row & 7)
  const uint8_t* xs;            // [term][k step][padded row][4 B]: e8m0 of the four 32-groups
  int64_t prows;                // padded rows: expert e's rows start at (slice_offs[e] & ~31) + 32 e
  int KT, NB;                   // 128-k steps, 128-row weight blocks
};

// first padded row of an expert: a multiple of 32, and never before the end of the previous expert's last group of 32
__device__ __forceinline__ int64_t padded_base(int e, int off) { return (int64_t)(off & ~31) + 32 * (int64_t)e; }

// ============================================================================================================
// Pack kernel.  A block takes up to 16 rows of one expert (an entry of the 16-row block schedule), a warp a row at a
// time, a lane 8 (bf16) or 16 (e4m3) consecutive k; four passes' loads are in flight before the first is converted.
// HBM-bound: 2 + 2 bytes per bf16 element, 1 + 1 per e4m3 element (gathered rows are read through L2).
// ============================================================================================================
struct PairPackParams {
  const void* x; int64_t ld_x; int64_t rows_x;
  const uint8_t* x_scale; int64_t ld_xs;
  const int32_t* gather;
  int K, KT;
  int64_t prows;
  uint8_t* xq; uint8_t* xs;
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
  const int first = (int)(ent >> 16) * 16, off = p.slice_offs[e];
  row0 = (int64_t)off + first;
  prow0 = padded_base(e, off) + first;
  rows = min(16, p.slice_sizes[e] - first);
  return rows > 0;
}

__device__ __forceinline__ float amax4(float a) {          // maximum over the four lanes of a 32-group
  a = fmaxf(a, __shfl_xor_sync(0xFFFFFFFFu, a, 1));
  return fmaxf(a, __shfl_xor_sync(0xFFFFFFFFu, a, 2));
}

__global__ void __launch_bounds__(256) mx_pair_pack2_kernel(const GemmParams p, const PairPackParams a) {
  int e; int64_t row0, prow0; int rows;
  if (!pack_block(p, blockIdx.x, e, row0, rows, prow0)) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t q_term = (int64_t)a.KT * a.prows * 128, s_term = (int64_t)a.KT * a.prows * 4;
  const int K128 = a.KT * 128;
  for (int r = warp; r < rows; r += 8) {
    int64_t src = a.gather ? (int64_t)a.gather[row0 + r] : row0 + r;
    if (src >= a.rows_x) src = -1;
    const __nv_bfloat16* xrow = (const __nv_bfloat16*)a.x + (src >= 0 ? src : 0) * a.ld_x;
    const int64_t prow = prow0 + r;
    const uint32_t x7 = (uint32_t)prow & 7u;
    for (int kb = lane * 8; kb - lane * 8 < K128; kb += 1024) {
      uint4 raw[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int k = kb + 256 * u;
        raw[u] = (src >= 0 && k < a.K) ? *reinterpret_cast<const uint4*>(xrow + k) : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int k = kb + 256 * u;
        if (k - lane * 8 >= K128) break;                           // warp-uniform
        const uint32_t w[4] = {raw[u].x, raw[u].y, raw[u].z, raw[u].w};
        float v[8];
        float m = 0.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          v[2 * i] = __uint_as_float(w[i] << 16);
          v[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
          m = fmaxf(m, fmaxf(fabsf(v[2 * i]), fabsf(v[2 * i + 1])));
        }
        m = amax4(m);
        if (!(m < 3.0e38f)) m = 3.0e38f;                           // Inf / NaN in the group: keep the scale finite
        uint32_t sh; float s_hi, i_hi;
        mx8_scale(m, sh, s_hi, i_hi);
        uint32_t h[4], l[4];
        float rm = 0.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          h[i] = f32x2_to_e4m3x2(v[2 * i] * i_hi, v[2 * i + 1] * i_hi);
          const float2 f = e4m3x2_to_f32x2(h[i]);
          v[2 * i] -= f.x * s_hi;
          v[2 * i + 1] -= f.y * s_hi;
          rm = fmaxf(rm, fmaxf(fabsf(v[2 * i]), fabsf(v[2 * i + 1])));
        }
        rm = amax4(rm);
        if (!(rm < 3.0e38f)) rm = 0.0f;
        uint32_t sl; float s_lo, i_lo;
        mx8_scale(rm, sl, s_lo, i_lo);
#pragma unroll
        for (int i = 0; i < 4; ++i) l[i] = f32x2_to_e4m3x2(v[2 * i] * i_lo, v[2 * i + 1] * i_lo);
        if (k < K128) {
          const int64_t line = (int64_t)(k >> 7) * a.prows + prow;
          uint8_t* dst = a.xq + line * 128 + ((((uint32_t)(k & 127) >> 4) ^ x7) << 4) + (k & 8);
          *reinterpret_cast<uint2*>(dst) = make_uint2(h[0] | (h[1] << 16), h[2] | (h[3] << 16));
          *reinterpret_cast<uint2*>(dst + q_term) = make_uint2(l[0] | (l[1] << 16), l[2] | (l[3] << 16));
          if ((lane & 3) == 0) {
            uint8_t* sd = a.xs + line * 4 + ((k >> 5) & 3);
            sd[0] = (uint8_t)sh;
            sd[s_term] = (uint8_t)sl;
          }
        }
      }
    }
  }
}

__global__ void __launch_bounds__(256) mx_pair_pack1_kernel(const GemmParams p, const PairPackParams a) {
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
// The whole MMA warp runs the issue loop and one lane's predicate guards the instruction.  The operands of tcgen05.mma live in
// uniform registers: computed by a single thread of a divergent branch, each takes a move from a vector register first, and
// an MMA cost 170-190 cycles to issue.  Of a shared-memory descriptor only the low word varies (start address, 16-byte units).
constexpr uint32_t DESC_LO = 1u << 16;                               // leading byte offset (unused for swizzled K-major)
constexpr uint32_t DESC_HI = (1024u >> 4) | (1u << 14) | (2u << 29); // 8-row groups 1024 B apart, sm_100, 128-byte swizzle
__device__ __forceinline__ void mma_mxf8f6f4_pair(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t sfa,
                                                  uint32_t sfb, uint32_t accumulate, uint32_t leader) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 da, db;\n\t"
      "mov.b64 da, {%1, %8};\n\t"
      "mov.b64 db, {%2, %8};\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "setp.ne.b32 q, %7, 0;\n\t"
      "@q tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale.scale_vec::1X [%0], da, db, %3, [%4], [%5], p;\n\t}" ::"r"(d_tmem),
      "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(sfa), "r"(sfb), "r"(accumulate), "r"(leader), "n"(DESC_HI)
      : "memory");
}
// A = e2m1 (code 5), B = e4m3 (code 0), both K-major, e8m0 scales, M = 256 over the two CTAs; sf: byte of the scale words
__device__ __forceinline__ uint32_t pair_idesc(int n, uint32_t sf) {
  return (sf << 4) | (5u << 7) | ((uint32_t)(n >> 3) << 17) | (1u << 23) | (2u << 27) | (sf << 29);
}

// Token tile tt: rows of one expert, in groups of 32 dealt evenly over the expert's tiles (a tail of a few rows does not
// become a tile of its own).
struct PTile { int e, rows, cols; int64_t row0, prow0; };
template <int NMAX> __device__ __forceinline__ PTile map_ptile(const GemmParams& p, const int32_t* prefix, int tt) {
  PTile t;
  int lo = 0, hi = p.slice_sizes ? p.E : 1;                          // largest e with prefix[e] <= tt
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (prefix[mid] <= tt) lo = mid; else hi = mid;
  }
  const int size = prefix[MAX_PREFIX_EXPERTS + 1 + lo], off = prefix[2 * MAX_PREFIX_EXPERTS + 1 + lo];
  const int nt = prefix[lo + 1] - prefix[lo], j = tt - prefix[lo];
  const int64_t q = (size + 31) >> 5;
  const int u0 = (int)(j * q / nt), u1 = (int)((j + 1) * q / nt);
  t.e = lo;
  t.row0 = (int64_t)off + 32 * u0;
  t.prow0 = padded_base(lo, off) + 32 * u0;
  t.cols = 32 * (u1 - u0);
  t.rows = min(t.cols, size - 32 * u0);
  return t;
}

// two fp32 operations in one instruction
__device__ __forceinline__ void add_f32x2(float& o0, float& o1, float a0, float a1, float b0, float b1) {
  asm("{\n\t.reg .b64 a, b, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tadd.rn.f32x2 d, a, b;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(o0), "=f"(o1) : "f"(a0), "f"(a1), "f"(b0), "f"(b1));
}
__device__ __forceinline__ void mul_f32x2(float& o0, float& o1, float a0, float a1, float b0, float b1) {
  asm("{\n\t.reg .b64 a, b, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmul.rn.f32x2 d, a, b;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(o0), "=f"(o1) : "f"(a0), "f"(a1), "f"(b0), "f"(b1));
}

template <typename TY, int TERMS>
__global__ void __launch_bounds__(PP_THREADS, 1)
gemm_mx_pair_kernel(const GemmParams p, const PairParams a, const __grid_constant__ CUtensorMap w_map) {
  using C = PCfg<TERMS>;
  constexpr int STAGES = C::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sbase = smem_u32(smem);
  const int warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;     // warp-uniform for the compiler
  const uint32_t rank = cluster_ctarank();
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
  const uint32_t bar0 = sbase + C::OFF_BAR;
  auto BAR_FULL = [&](int s) { return bar0 + 8u * (uint32_t)s; };                       // own copies have landed
  auto BAR_EMPTY = [&](int s) { return bar0 + 8u * (uint32_t)(STAGES + s); };
  auto BAR_SF = [&](int s) { return bar0 + 8u * (uint32_t)(2 * STAGES + s); };           // even CTA: scales (and operands) of both CTAs
  auto BAR_ACC_FULL = [&](int u) { return bar0 + 8u * (uint32_t)(3 * STAGES + u); };
  auto BAR_ACC_EMPTY = [&](int u) { return bar0 + 8u * (uint32_t)(3 * STAGES + 2 + u); };   // even CTA
  const uint32_t BAR_DRAIN = bar0 + 8u * (uint32_t)(3 * STAGES + 4);
  volatile uint32_t* s_tmem = reinterpret_cast<volatile uint32_t*>(smem + C::OFF_MISC);
  volatile int* s_abort = reinterpret_cast<volatile int*>(smem + C::OFF_MISC + 4);
  volatile int* s_cols = reinterpret_cast<volatile int*>(smem + C::OFF_COLS);
  int32_t* s_prefix = reinterpret_cast<int32_t*>(smem + C::OFF_PREFIX);
  Ctl ctl{s_abort, p.status};

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(BAR_FULL(s), 1);
      mbar_init(BAR_EMPTY(s), 1);
      mbar_init(BAR_SF(s), 8);                         // four scale warps in each CTA
    }
    for (int u = 0; u < 2; ++u) {
      mbar_init(BAR_ACC_FULL(u), 1);
      mbar_init(BAR_ACC_EMPTY(u), 2 * PP_EPI_WARPS);
    }
    mbar_init(BAR_DRAIN, 1);
    *s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sbase + C::OFF_MISC), "r"((uint32_t)TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  if (warp == PP_SF_WARP0) {                           // tile prefix over experts
    const int n = p.slice_sizes ? p.E : 1;
    int run = 0;
    for (int e0 = 0; e0 < n; e0 += 32) {
      const int e = e0 + lane;
      const int size = e < n ? max(p.slice_sizes ? p.slice_sizes[e] : (int)p.M, 0) : 0;
      int v = (size + C::NMAX - 1) / C::NMAX;
      if (e < n) {
        s_prefix[MAX_PREFIX_EXPERTS + 1 + e] = size;
        s_prefix[2 * MAX_PREFIX_EXPERTS + 1 + e] = p.slice_sizes ? p.slice_offs[e] : 0;
      }
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if (lane >= o) v += t;
      }
      if (e < n) s_prefix[e + 1] = run + v;
      run += __shfl_sync(0xFFFFFFFFu, v, 31);
    }
    if (lane == 0) s_prefix[0] = 0;
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                                  // the other CTA's barriers exist before anyone signals them
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xFFFFFFFFu, *s_tmem, 0);

  const int KT = a.KT, NB = a.NB;
  const int MB = (NB + 1) >> 1, MT = (MB + 1) >> 1;     // 256-row weight blocks, tiles of two of them
  const int n_tiles = __shfl_sync(0xFFFFFFFFu, s_prefix[p.slice_sizes ? p.E : 1], 0) * MT;

  if (warp < PP_SF_WARP0) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_ISSUE));
  if (warp == 0) {
    // ================================= producer =======================================================
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      PTile t, nxt;                                    // the next tile is looked up while this one streams
      if (pair < n_tiles) nxt = map_ptile<C::NMAX>(p, s_prefix, pair / MT);
      for (int tile = pair; tile < n_tiles && ok; tile += n_pairs) {
        t = nxt;
        const int blk0 = (tile % MT) * 4 + (int)rank;                 // own block of the first 256-row block; the second's is + 2
        const int n_w = (blk0 < NB) + (blk0 + 2 < NB);                // (an absent block's stage keeps stale data)
        const uint32_t bx = (uint32_t)t.cols * 64u, bs = (uint32_t)t.cols * 4u;       // own half of the rows, all scales
        const uint32_t tx = (uint32_t)n_w * (128 * 64 + 512) + TERMS * (bx + bs);
        for (int kt = 0; kt < KT; ++kt, ++it) {
          const int s = it % STAGES;
          ok = mbar_wait(BAR_EMPTY(s), ((it / STAGES) & 1u) ^ 1u, ctl, 611);
          if (!ok) break;
          const uint32_t st = sbase + (uint32_t)s * C::STAGE;
          mbar_expect_tx(BAR_FULL(s), tx);
          const int64_t wt = ((int64_t)t.e * KT + kt) * NB + blk0;
#pragma unroll
          for (int m = 0; m < 2; ++m)
            if (m < n_w) {
              tma_tile_3d(st + m * 128 * 128, &w_map, 0, 0, (int)(wt + 2 * m), BAR_FULL(s));
              bulk_g2s(st + C::OFF_WS + m * 512, p.w_scale + (wt + 2 * m) * 512, 512u, BAR_FULL(s));
            }
#pragma unroll
          for (int c = 0; c < TERMS; ++c) {
            const int64_t line = ((int64_t)c * KT + kt) * a.prows + t.prow0;
            bulk_g2s(st + C::OFF_X + c * C::X_TERM, a.xq + line * 128 + rank * bx, bx, BAR_FULL(s));
            bulk_g2s(st + C::OFF_XS + c * 1024, a.xs + line * 4, bs, BAR_FULL(s));
          }
          if (kt == 0 && tile + n_pairs < n_tiles) nxt = map_ptile<C::NMAX>(p, s_prefix, (tile + n_pairs) / MT);
        }
      }
      if (!ok) {
        // aborting: let the copies that were already issued land before the CTA leaves
        const uint32_t lo = it > (uint32_t)STAGES ? it - STAGES : 0;
        for (uint32_t j = lo; j < it; ++j)
          for (uint32_t i = 0; i < (1u << 16) && !mbar_test(BAR_FULL(j % STAGES), (j / STAGES) & 1u); ++i) __nanosleep(64);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ================================= MMA issuer (even CTA) ==========================================
    if (rank == 0) {
      const uint32_t leader = elect_one();
      const int k_whole = p.K >> 7;                    // steps of 128 k; the last may hold less
      uint32_t s = 0, ph = 0;                          // stage and parity of the next k step
      uint32_t acc_ph = 3u;                          // parity to wait for, per unit
      uint32_t tc = 0;
      bool ok = true;
      for (int tile = pair; tile < n_tiles && ok; tile += n_pairs, ++tc) {
        ok = __all_sync(0xFFFFFFFFu, mbar_wait_cluster(BAR_SF(s), ph, ctl, 612));         // first k step; the scale loader left the columns
        if (!ok) break;
        const uint32_t id0 = pair_idesc(__shfl_sync(0xFFFFFFFFu, s_cols[tc & 7u], 0), 0);
        const uint32_t live = (tile % MT) * 2 + 1 < MB ? 3u : 1u;      // units of the tile: 256-row weight blocks
        auto issue = [&](int u, int k, uint32_t s) {   // k step `k` of unit u, operands in stage s
          const uint32_t st = sbase + s * C::STAGE;
          const uint32_t sf = tmem_base + C::SF_BASE + s * C::SF_COLS;
          const uint32_t a_lo = DESC_LO | ((st + (uint32_t)u * (128 * 128)) >> 4);
          const uint32_t b_lo = DESC_LO | ((st + C::OFF_X) >> 4);
          const uint32_t d = tmem_base + (uint32_t)(u * C::NMAX);
          // (a step that is whole has no test between its instructions: they must issue in less than the 45-64 cycles that
          // one of them runs)
          if (k < k_whole) {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
#pragma unroll
              for (int c = 0; c < TERMS; ++c)
                mma_mxf8f6f4_pair(d, a_lo + kk * 2, b_lo + c * (C::X_TERM >> 4) + kk * 2, id0 + ((uint32_t)kk << 4) + ((uint32_t)kk << 29),
                                  sf + 4 * u, sf + 8 + 8 * c, (kk | c) ? 1u : (uint32_t)(k > 0), leader);
          } else {
            const int kk_live = (p.K - k * 128 + 31) >> 5;
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              if (kk < kk_live) {
#pragma unroll
                for (int c = 0; c < TERMS; ++c)
                  mma_mxf8f6f4_pair(d, a_lo + kk * 2, b_lo + c * (C::X_TERM >> 4) + kk * 2, id0 + ((uint32_t)kk << 4) + ((uint32_t)kk << 29),
                                    sf + 4 * u, sf + 8 + 8 * c, (k | kk | c) ? 1u : 0u, leader);
              }
          }
        };
        // ---- ramp: units join as the epilogue hands them back; those that have joined run ahead by up to the ring ------
        uint32_t joined = 0;
        int kt = 0, base = 0;                          // next k step of the joined units, of the others
        uint32_t s_base = s;
        while (ok && (joined != live || kt == 0)) {
          if (kt - base < STAGES && kt < KT) {
            ok = __all_sync(0xFFFFFFFFu, mbar_wait_cluster(BAR_SF(s), ph, ctl, 612));
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int u = 0; u < 2; ++u)
              if ((joined >> u) & 1u) issue(u, kt, s);
            ++kt;
            if (++s == STAGES) { s = 0; ph ^= 1u; }
          }
          const bool full = kt - base >= STAGES || kt >= KT;           // nothing to do for the joined units: wait for the next one
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            if (!((live >> u) & 1u) || ((joined >> u) & 1u)) continue;
            const uint32_t par = (acc_ph >> u) & 1u;
            bool got;
            if (full || joined == 0) got = ok = __all_sync(0xFFFFFFFFu, mbar_wait_cluster(BAR_ACC_EMPTY(u), par, ctl, 613));
            else got = __all_sync(0xFFFFFFFFu, mbar_test(BAR_ACC_EMPTY(u), par));                  // (try_wait would sleep)
            if (!got) break;
            tc_fence_after();
            joined |= 1u << u;
            acc_ph ^= 1u << u;
            uint32_t sk = s_base;
            for (int k = base; k < kt; ++k) {                          // catch up with the others
              issue(u, k, sk);
              if (joined == live) mma_commit_pair(BAR_EMPTY(sk), leader);
              if (++sk == STAGES) sk = 0;
            }
            if (full) break;
          }
        }
        // ---- steady state ---------------------------------------------------------------------------------------
        const bool all_in_ramp = kt == KT;
        for (; ok && kt < KT; ++kt) {
          ok = __all_sync(0xFFFFFFFFu, mbar_wait_cluster(BAR_SF(s), ph, ctl, 612));
          if (!ok) break;
          tc_fence_after();
#pragma unroll
          for (int u = 0; u < 2; ++u)
            if ((live >> u) & 1u) {
              issue(u, kt, s);
              if (kt == KT - 1) mma_commit_pair(BAR_ACC_FULL(u), leader);
            }
          mma_commit_pair(BAR_EMPTY(s), leader);
          if (++s == STAGES) { s = 0; ph ^= 1u; }
        }
        if (ok && all_in_ramp)
#pragma unroll
          for (int u = 0; u < 2; ++u)
            if ((live >> u) & 1u) mma_commit_pair(BAR_ACC_FULL(u), leader);
      }
      // every MMA issued by this warp has retired before tensor memory is freed
      mma_commit_pair_local(BAR_DRAIN, leader);
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
    uint32_t it = 0, tc = 0;
    bool ok = true;
    PTile t, nxt;
    if (pair < n_tiles) nxt = map_ptile<C::NMAX>(p, s_prefix, pair / MT);
    for (int tile = pair; tile < n_tiles && ok; tile += n_pairs, ++tc) {
      t = nxt;
      if (warp == PP_SF_WARP0 && lane == 0) s_cols[tc & 7u] = t.cols;     // read by the MMA warp after the first SF wait
      for (int kt = 0; kt < KT; ++kt, ++it) {
        const int s = it % STAGES;
        ok = __all_sync(0xFFFFFFFFu, mbar_wait(BAR_FULL(s), (it / STAGES) & 1u, ctl, 615));
        if (!ok) break;
        const uint32_t st = sbase + (uint32_t)s * C::STAGE;
        const uint32_t taddr = tmem_base + ((uint32_t)(qd * 32) << 16) + (uint32_t)(C::SF_BASE + s * C::SF_COLS);
        const uint4 w0 = lds128(st + C::OFF_WS + (uint32_t)lane * 16u), w1 = lds128(st + C::OFF_WS + 512u + (uint32_t)lane * 16u);
        uint32_t x[TERMS][8];
#pragma unroll
        for (int c = 0; c < TERMS; ++c)
#pragma unroll
          for (int i = 0; i < 8; ++i) x[c][i] = lds32(st + C::OFF_XS + (uint32_t)(c * 1024 + (32 * i + lane) * 4));
        asm volatile(
            "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
            "r"(w0.x), "r"(w0.y), "r"(w0.z), "r"(w0.w), "r"(w1.x), "r"(w1.y), "r"(w1.z), "r"(w1.w), "r"(x[0][0]), "r"(x[0][1]),
            "r"(x[0][2]), "r"(x[0][3]), "r"(x[0][4]), "r"(x[0][5]), "r"(x[0][6]), "r"(x[0][7])
            : "memory");
        if constexpr (TERMS == 2)
          asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr + 16u), "r"(x[1][0]),
                       "r"(x[1][1]), "r"(x[1][2]), "r"(x[1][3]), "r"(x[1][4]), "r"(x[1][5]), "r"(x[1][6]), "r"(x[1][7])
                       : "memory");
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(BAR_SF(s), 0);
        if (kt == 0 && tile + n_pairs < n_tiles) nxt = map_ptile<C::NMAX>(p, s_prefix, (tile + n_pairs) / MT);
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS_EPI));
    // ================================= epilogue =======================================================
    // Accumulator [weight row = lane][token = column].  The warps of a lane quarter take the 16-token chunks of a unit in turn.
    // Neighbouring lanes hold neighbouring outputs of a row (or gate and linear): they swap halves of a chunk, after which the
    // even lane has both values of tokens 0-7 and the odd lane those of tokens 8-15.  Row addresses and routing weights come
    // from a table in shared memory, filled once per tile.
    const int ew = warp - PP_EPI_WARP0, qd = warp & 3, grp = ew >> 2;
    const int tid = threadIdx.x - PP_EPI_WARP0 * 32;
    const int odd = lane & 1;
    const uint32_t sel = odd ? 0x3276u : 0x5410u;
    const bool swiglu = p.activation == MOE_ACT_SWIGLU;
    const bool vec = p.ld_y % 2 == 0 && (uintptr_t)p.y % (2 * sizeof(TY)) == 0;
    uint32_t tc = 0;
    uint32_t acc_ph = 0;                               // parity to wait for, per unit
    bool ok = true;
    for (int tile = pair; tile < n_tiles && ok; tile += n_pairs, ++tc) {
      const PTile t = map_ptile<C::NMAX>(p, s_prefix, tile / MT);
      const int mt = tile % MT;
      const uint32_t tab = sbase + C::OFF_TAB + (tc & 1u) * C::TAB;
      if (tid < t.cols) {                                         // at most 224 of the 256 or more threads
        unsigned long long row = 0;
        float beta = 1.0f, gamma = 1.0f;
        if (tid < t.rows) {
          const int64_t m = t.row0 + tid;
          const int64_t d = p.scatter_indx ? (int64_t)p.scatter_indx[m] : m;
          if (d >= 0) row = (unsigned long long)gemm_out_row<TY>(p, d);
          if (p.betas) beta = p.betas[m];
          if (p.gammas) gamma = p.gammas[m];
        }
        asm volatile("st.shared.u64 [%0], %1;" ::"r"(tab + (uint32_t)tid * 8u), "l"(row) : "memory");
        asm volatile("st.shared.f32 [%0], %1;" ::"r"(tab + 2048u + (uint32_t)tid * 4u), "f"(gamma) : "memory");
        asm volatile("st.shared.f32 [%0], %1;" ::"r"(tab + 3072u + (uint32_t)tid * 4u), "f"(beta) : "memory");
      }
      float bias_m[2];
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int n = ((mt * 2 + m) * 2 + (int)rank) * 128 + qd * 32 + lane;     // own weight row
        bias_m[m] = (p.bias && n < p.N) ? load_bias(p.bias, p.bias_dtype, (int64_t)t.e * p.ld_bias + n) : 0.0f;
      }
      asm volatile("bar.sync 1, %0;" ::"n"(PP_EPI_WARPS * 32) : "memory");
#pragma unroll 1
      for (int u = 0; u < 2; ++u) {
        if (mt * 2 + u >= MB) break;
        const int ne = ((mt * 2 + u) * 2 + (int)rank) * 128 + qd * 32 + (lane & ~1);      // first of the lane pair's two columns
        const bool first = ne < p.N, both = ne + 1 < p.N;
        const float bias_n = u ? bias_m[1] : bias_m[0];
        ok = __all_sync(0xFFFFFFFFu, mbar_wait(BAR_ACC_FULL(u), (acc_ph >> u) & 1u, ctl, 616));
        if (!ok) break;
        acc_ph ^= 1u << u;
        tc_fence_after();
        const uint32_t taddr = tmem_base + ((uint32_t)(qd * 32) << 16) + (uint32_t)(u * C::NMAX);
        // No branch inside a chunk but the stores' own predicates: exchanges, table loads and arithmetic of its tokens
        // overlap (token by token behind a branch each, a chunk took 1700 cycles).
        const bool fast = __all_sync(0xFFFFFFFFu, both && (swiglu || vec));
        auto emit = [&](const uint32_t (&raw)[16], int c) {
          const uint32_t tb = tab + (uint32_t)(c) * 8u, tg = tab + 2048u + (uint32_t)(c) * 4u;
          float v[16];
#pragma unroll
          for (int j = 0; j < 16; j += 2) add_f32x2(v[j], v[j + 1], __uint_as_float(raw[j]), __uint_as_float(raw[j + 1]), bias_n, bias_n);
          if (p.betas) {
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(raw[j]) + bias_n * __uint_as_float(lds32(tg + 1024u + (uint32_t)j * 4u));
          }
          if (p.has_out_alpha) {
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] *= p.out_alpha;
          }
          unsigned long long row[8];                                   // output rows of this lane's eight tokens
#pragma unroll
          for (int j = 0; j < 8; j += 2) {
            const uint4 e = lds128(tb + (uint32_t)(j + 8 * odd) * 8u);
            row[j] = ((unsigned long long)e.y << 32) | e.x;
            row[j + 1] = ((unsigned long long)e.w << 32) | e.z;
          }
          if (!swiglu && sizeof(TY) == 2 && fast) {
            // weights applied and rounded before the exchange: one shuffle and one byte permute per pair of outputs
#pragma unroll
            for (int j = 0; j < 16; j += 4) {
              const uint4 g = lds128(tg + (uint32_t)j * 4u);
              mul_f32x2(v[j], v[j + 1], v[j], v[j + 1], __uint_as_float(g.x), __uint_as_float(g.y));
              mul_f32x2(v[j + 2], v[j + 3], v[j + 2], v[j + 3], __uint_as_float(g.z), __uint_as_float(g.w));
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              TY h[2] = {from_f32<TY>(v[j]), from_f32<TY>(v[8 + j])};
              const uint32_t own = *reinterpret_cast<const uint32_t*>(h);
              const uint32_t out = __byte_perm(own, __shfl_xor_sync(0xFFFFFFFFu, own, 1), sel);
              if (row[j]) *reinterpret_cast<uint32_t*>((TY*)row[j] + ne) = out;
            }
            return;
          }
          float v0[8], v1[8], g[8];
#pragma unroll
          for (int j = 0; j < 8; j += 4) {
            const uint4 e = lds128(tg + (uint32_t)(j + 8 * odd) * 4u);
            g[j] = __uint_as_float(e.x); g[j + 1] = __uint_as_float(e.y); g[j + 2] = __uint_as_float(e.z); g[j + 3] = __uint_as_float(e.w);
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float recv = __shfl_xor_sync(0xFFFFFFFFu, odd ? v[j] : v[8 + j], 1);
            v0[j] = odd ? recv : v[j];
            v1[j] = odd ? v[8 + j] : recv;
          }
          if (swiglu) {
#pragma unroll
            for (int j = 0; j < 8; ++j) v0[j] = gemm_swiglu(v0[j], v1[j], p.act_alpha, p.act_limit, p.act_has_limit) * g[j];
#pragma unroll
            for (int j = 0; j < 8; ++j)
              if (row[j] && both) ((TY*)row[j])[ne >> 1] = from_f32<TY>(v0[j]);
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              if (row[j] && first) ((TY*)row[j])[ne] = from_f32<TY>(v0[j] * g[j]);
              if (row[j] && both) ((TY*)row[j])[ne + 1] = from_f32<TY>(v1[j] * g[j]);
            }
          }
        };
        if constexpr (TERMS == 2) {
          // The warp's whole share of the unit goes to registers and the unit back to the MMA warp before any of it is worked
          // on: drained chunk by chunk, the tensor pipe waited 3000-4600 cycles for the first unit of every tile.  (The wider
          // one-term tile does not fit the registers that way.)
          uint32_t raw[C::EPI_CHUNKS][16];
#pragma unroll
          for (int i = 0; i < C::EPI_CHUNKS; ++i) {
            const int c = (grp + i * (PP_EPI_WARPS / 4)) * 16;
            if (c < t.rows) tmem_ld16(taddr + (uint32_t)c, raw[i]);
          }
          tmem_ld_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(BAR_ACC_EMPTY(u), 0);
#pragma unroll
          for (int i = 0; i < C::EPI_CHUNKS; ++i) {
            const int c = (grp + i * (PP_EPI_WARPS / 4)) * 16;
            if (c < t.rows) emit(raw[i], c);
          }
        } else {
          uint32_t raw[16];
#pragma unroll 1
          for (int c = grp * 16; c < t.rows; c += 4 * PP_EPI_WARPS) {
            tmem_ld16(taddr + (uint32_t)c, raw);
            tmem_ld_wait();
            emit(raw, c);
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(BAR_ACC_EMPTY(u), 0);
        }
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
  int64_t prows, xs_off, ws_bytes;
};

PairPlan pair_plan(const MoeGemmArgs& a) {
  PairPlan pl;
  pl.KT = (int)cdiv64(a.K, 128);
  pl.NB = (int)cdiv64(a.N, 128);
  pl.terms = a.x_dtype == MOE_BF16 ? 2 : 1;
  const int64_t E = a.slice_sizes ? a.E : 1;
  pl.prows = cdiv64(a.M, 32) * 32 + 32 * (E + 1);
  pl.xs_off = pl.terms * pl.KT * pl.prows * 128;
  pl.ws_bytes = pl.xs_off + pl.terms * pl.KT * pl.prows * 4;
  return pl;
}

template <typename TY, int TERMS>
int launch_mx_pair(const GemmParams& p, const PairParams& q, int64_t tiles, const CUtensorMap& w_map, int idle_sms, cudaStream_t st) {
  auto kernel = gemm_mx_pair_kernel<TY, TERMS>;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(PP_THREADS, 1, 1);
  cfg.dynamicSmemBytes = PCfg<TERMS>::ALLOC;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  cfg.attrs = at; cfg.numAttrs = 1;
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
      MOE_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PCfg<TERMS>::ALLOC));
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
  moe_count_launch();
  MOE_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kernel, p, q, w_map));
  return MOE_OK;
}

template <typename TY>
int launch_mx_pair_terms(const GemmParams& p, const PairParams& q, int terms, int64_t tiles, const CUtensorMap& m, int idle, cudaStream_t st) {
  return terms == 2 ? launch_mx_pair<TY, 2>(p, q, tiles, m, idle, st) : launch_mx_pair<TY, 1>(p, q, tiles, m, idle, st);
}

}  // namespace

// The pair form against the decode forms of gemm_mx.cu, by mean rows per expert (fc1 + fc2).  bf16 tokens, from 40 on: 32
// experts of 2880 x 5760, 32 rows 172 us there and 189 here, 48 rows 219 and 216; 128 experts, 32 rows 530 and 486; narrow
// products repay the larger tiles later (8 experts of 512 x 2048, 64 rows: 41 and 48).  e4m3 tokens, one term, from 16 on
// (32 experts, 8 rows: 102 and 114; 64 rows: 320 and 167).  tile_m = 256 asks for it.
bool moe_gemm_mx_pair_wanted(const MoeGemmArgs& a) {
  if (a.slice_sizes && a.E > MAX_PREFIX_EXPERTS) return false;
  if (a.M >= (1ll << 31) - (1 << 20) || a.kernel == MOE_GEMM_MX_F4 || a.tile_n != 0) return false;
  if (a.tile_m == 256) return true;
  if (a.tile_m != 0 || a.kernel == MOE_GEMM_MX_F8) return false;
  const int64_t per = a.slice_sizes ? a.M / a.E : a.M;
  if (a.x_dtype != MOE_BF16) return per >= 16;
  return per >= (a.N >= 1280 ? 40 : 96);
}

int64_t moe_gemm_mx_pair_workspace(const MoeGemmArgs& a) { return pair_plan(a).ws_bytes; }

int moe_gemm_mx_pair_launch(const GemmParams& p_in, const MoeGemmArgs& a, cudaStream_t st) {
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
  pk.K = a.K; pk.KT = pl.KT; pk.prows = pl.prows;
  pk.xq = (uint8_t*)a.mx_workspace; pk.xs = pk.xq + pl.xs_off;
  if (pl.terms == 2) mx_pair_pack2_kernel<<<(unsigned)blocks16, 256, 0, st>>>(p, pk);
  else mx_pair_pack1_kernel<<<(unsigned)blocks16, 256, 0, st>>>(p, pk);
  MOE_CHECK_LAUNCH();
  PairParams q;
  q.xq = pk.xq; q.xs = pk.xs; q.prows = pl.prows; q.KT = pl.KT; q.NB = pl.NB;
  CUtensorMap w_map;
  if (int rc = make_w_map(a, pl.KT, pl.NB, false, 1, &w_map)) return rc;
  // every expert has at most ceil(rows / 192) token tiles
  const int64_t tiles = ((a.slice_sizes ? a.E : 0) + cdiv64(a.M, PCfg<2>::NMAX)) * cdiv64(pl.NB, 4);
  const int idle = a.idle_sms > 0 ? a.idle_sms : 0;
  if (a.y_dtype == MOE_F8E4M3) return launch_mx_pair_terms<__nv_fp8_e4m3>(p, q, pl.terms, tiles, w_map, idle, st);
  if (a.y_dtype == MOE_BF16) return launch_mx_pair_terms<__nv_bfloat16>(p, q, pl.terms, tiles, w_map, idle, st);
  return launch_mx_pair_terms<float>(p, q, pl.terms, tiles, w_map, idle, st);
}
