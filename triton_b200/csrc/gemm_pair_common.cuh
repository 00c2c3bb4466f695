// Pieces of the kernels that run on a cluster of two CTAs (tcgen05 cta_group::2): barriers of the other CTA, commits that
// signal both.
#pragma once
#include "gemm_tc_common.cuh"

namespace {

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Arrive on the barrier at the same shared-memory offset in CTA `cta` of the cluster.  Default (CTA-scope release)
// semantics: a cluster-scope release costs about a thousand cycles per arrival while copies are in flight, and what
// the arrival publishes here is either a go-ahead for the tensor core of the SM that already holds the data (stage
// full) or the end of tensor-memory reads that were fenced by tcgen05.fence (accumulator drained).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar, uint32_t cta) {
  asm volatile(
      "{\n\t.reg .b32 ra;\n\t"
      "mapa.shared::cluster.u32 ra, %0, %1;\n\t"
      "mbarrier.arrive.shared::cluster.b64 _, [ra];\n\t}" ::"r"(bar),
      "r"(cta)
      : "memory");
}
// arrive on the barrier at this offset in both CTAs of the pair once every MMA issued so far has completed
__device__ __forceinline__ void mma_commit_pair(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
      "h"((uint16_t)3)
      : "memory");
}
__device__ __forceinline__ void mma_commit_pair_local(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// the same for a warp that runs its issue loop as a whole
__device__ __forceinline__ void elect_commit_pair(uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\telect.sync _|q, 0xFFFFFFFF;\n\t"
      "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}" ::"r"(bar),
      "h"((uint16_t)3)
      : "memory");
}
__device__ __forceinline__ void elect_commit_pair_local(uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\telect.sync _|q, 0xFFFFFFFF;\n\t"
      "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar)
      : "memory");
}

// ---- token tiles -------------------------------------------------------------------------------------------------
// prefix (shared memory): [E + 1] tiles of the experts before, [E] rows at MAX_PREFIX_EXPERTS + 1, [E] first rows after them
constexpr int PAIR_PREFIX_INTS = 3 * MAX_PREFIX_EXPERTS + 1;
__device__ __forceinline__ void pair_prefix(const GemmParams& p, int32_t* s_prefix, int nmax, int lane) {       // one warp
  const int n = p.slice_sizes ? p.E : 1;
  int run = 0;
  for (int e0 = 0; e0 < n; e0 += 128) {
    int sizes[4], offs[4];                             // loads of 128 experts side by side
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int e = e0 + 32 * i + lane;
      sizes[i] = e < n ? max(p.slice_sizes ? p.slice_sizes[e] : (int)p.M, 0) : 0;
      offs[i] = e < n && p.slice_sizes ? p.slice_offs[e] : 0;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int e = e0 + 32 * i + lane;
      int v = (sizes[i] + nmax - 1) / nmax;
      if (e < n) {
        s_prefix[MAX_PREFIX_EXPERTS + 1 + e] = sizes[i];
        s_prefix[2 * MAX_PREFIX_EXPERTS + 1 + e] = offs[i];
      }
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if (lane >= o) v += t;
      }
      if (e < n) s_prefix[e + 1] = run + v;
      run += __shfl_sync(0xFFFFFFFFu, v, 31);
    }
  }
  if (lane == 0) s_prefix[0] = 0;
}
// The expert that token tile tt belongs to by what ld_hint reads, -1: none (one warp).
__device__ __forceinline__ int pair_hint_expert(const GemmParams& p, int nmax, int tt, int lane) {
  const int n = p.slice_sizes ? p.E : 1;
  int run = 0;
  for (int e0 = 0; e0 < n; e0 += 32) {
    const int e = e0 + lane;
    const int size = e < n ? max(p.slice_sizes ? ld_hint(p.slice_sizes + e) : (int)p.M, 0) : 0;
    int v = size / nmax + (size % nmax != 0);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xFFFFFFFFu, v, o);
      if (lane >= o) v += t;
    }
    const unsigned past = __ballot_sync(0xFFFFFFFFu, e < n && run + v > tt);
    if (past) return e0 + __ffs(past) - 1;
    run += __shfl_sync(0xFFFFFFFFu, v, 31);
  }
  return -1;
}

// Token tile tt: rows of one expert, in groups of 32 dealt evenly over the expert's tiles (a tail of a few rows does not
// become a tile of its own).
struct PTile { int e, rows, cols; int64_t row0; int off, first; };      // first: row of the expert the tile starts with
__device__ __forceinline__ PTile map_ptile(const GemmParams& p, const int32_t* prefix, int tt) {
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
  t.off = off;
  t.first = 32 * u0;
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

// ---- epilogue ------------------------------------------------------------------------------------------------------
// Accumulator [weight row = lane][token = column].  Neighbouring lanes hold neighbouring outputs of a row (or gate and linear):
// they swap halves of a 16-token chunk, after which the even lane has both values of tokens 0-7 and the odd lane those of
// tokens 8-15.  Row addresses and routing weights come from a table in shared memory, filled once per tile:
// row address [256], gamma [256], beta [256].
constexpr int PAIR_TAB = 256 * 16;
template <typename TY> __device__ __forceinline__ void pair_table_entry(const GemmParams& p, const PTile& t, int tid, bool stored, uint32_t tab) {
  unsigned long long row = 0;
  float beta = 1.0f, gamma = 1.0f;
  if (stored) {
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

struct PairOut {
  int ne;                        // first of the lane pair's two columns
  bool first, both, fast;        // they exist; every pair of the warp may be stored as one word
  int odd;
  uint32_t sel;                  // byte permute that puts own and received halves in order
  float bias;                    // of the lane's own column
};

// No branch inside a chunk but the stores' own predicates: exchanges, table loads and arithmetic of its tokens overlap (token
// by token behind a branch each, a chunk took 1700 cycles).
template <typename TY>
__device__ __forceinline__ void pair_emit(const GemmParams& p, const PairOut& o, const uint32_t (&raw)[16], uint32_t tab, int c) {
  const bool swiglu = p.activation == MOE_ACT_SWIGLU;
  const uint32_t tb = tab + (uint32_t)(c) * 8u, tg = tab + 2048u + (uint32_t)(c) * 4u;
  float v[16];
#pragma unroll
  for (int j = 0; j < 16; j += 2) add_f32x2(v[j], v[j + 1], __uint_as_float(raw[j]), __uint_as_float(raw[j + 1]), o.bias, o.bias);
  if (p.betas) {
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(raw[j]) + o.bias * __uint_as_float(lds32(tg + 1024u + (uint32_t)j * 4u));
  }
  if (p.has_out_alpha) {
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] *= p.out_alpha;
  }
  unsigned long long row[8];                                   // output rows of this lane's eight tokens
#pragma unroll
  for (int j = 0; j < 8; j += 2) {
    const uint4 e = lds128(tb + (uint32_t)(j + 8 * o.odd) * 8u);
    row[j] = ((unsigned long long)e.y << 32) | e.x;
    row[j + 1] = ((unsigned long long)e.w << 32) | e.z;
  }
  if (!swiglu && sizeof(TY) == 2 && o.fast) {
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
      const uint32_t two = __byte_perm(own, __shfl_xor_sync(0xFFFFFFFFu, own, 1), o.sel);
      if (row[j]) *reinterpret_cast<uint32_t*>((TY*)row[j] + o.ne) = two;
    }
    return;
  }
  float v0[8], v1[8], g[8];
#pragma unroll
  for (int j = 0; j < 8; j += 4) {
    const uint4 e = lds128(tg + (uint32_t)(j + 8 * o.odd) * 4u);
    g[j] = __uint_as_float(e.x); g[j + 1] = __uint_as_float(e.y); g[j + 2] = __uint_as_float(e.z); g[j + 3] = __uint_as_float(e.w);
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float recv = __shfl_xor_sync(0xFFFFFFFFu, o.odd ? v[j] : v[8 + j], 1);
    v0[j] = o.odd ? recv : v[j];
    v1[j] = o.odd ? v[8 + j] : recv;
  }
  if (swiglu) {
#pragma unroll
    for (int j = 0; j < 8; ++j) v0[j] = gemm_swiglu(v0[j], v1[j], p.act_alpha, p.act_limit, p.act_has_limit) * g[j];
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (row[j] && o.both) ((TY*)row[j])[o.ne >> 1] = from_f32<TY>(v0[j]);
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (row[j] && o.first) ((TY*)row[j])[o.ne] = from_f32<TY>(v0[j] * g[j]);
      if (row[j] && o.both) ((TY*)row[j])[o.ne + 1] = from_f32<TY>(v1[j] * g[j]);
    }
  }
}

}  // namespace
