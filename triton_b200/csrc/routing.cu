// Routing kernels for sm_100a: top-k (+softmax) + expert bitmatrix, the expert histogram with the
// stable expert-major sort of the (token, slot) entries, and the ragged-segment metadata.
//
// Semantics follow triton_kernels topk_details/_topk_forward.py:15-150, tensor_details/bitmatrix.py:43-150
// and tensor_details/ragged_tensor.py:128-210, 310-381; the kernels themselves are organised
// differently (four lanes per token row for the top-k, a warp for other k; a counting sort, in one launch for up to 32768 entries, else
// in three passes, instead of per-block bitonic sorts; one launch each for the ragged metadata and its remap; the
// whole step in one to three launches).
#include "common.cuh"
#include "topk_select.cuh"

namespace {

constexpr int kWarpsPerBlock = 8;
constexpr int kMaxTopK = 64;

// order-preserving map float -> uint32 (larger float <=> larger key)
__device__ __forceinline__ uint32_t float_key(float f) {
  uint32_t b = __float_as_uint(f);
  return b ^ ((b & 0x80000000u) ? 0xFFFFFFFFu : 0x80000000u);
}
__device__ __forceinline__ float key_float(uint32_t k) {
  uint32_t b = k ^ ((k & 0x80000000u) ? 0x80000000u : 0xFFFFFFFFu);
  return __uint_as_float(b);
}

__device__ __forceinline__ unsigned long long warp_max_u64(unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    unsigned long long other = __shfl_xor_sync(0xFFFFFFFFu, v, o);
    v = other > v ? other : v;
  }
  return v;
}

// One warp per token row.  Selection i picks the largest packed key (value key << 32 | ~index) that is
// smaller than the key picked by selection i-1, so equal values resolve to the smaller expert index and
// the k results come out sorted by (value desc, index asc).  The row is re-read from L1 for each pick.
template <typename T>
__global__ void __launch_bounds__(kWarpsPerBlock * 32) topk_kernel(
    const T* __restrict__ logits, int64_t ld_logits, int64_t T_rows, int E, int k, int apply_softmax,
    T* __restrict__ vals, int64_t ld_vals, int16_t* __restrict__ indx, int64_t ld_indx,
    uint32_t* __restrict__ bitmatrix, int64_t bm_stride_row, int64_t bm_stride_word,
    const int32_t* __restrict__ n_rows_dev, int use_provided_indx) {
  __shared__ float s_val[kWarpsPerBlock][kMaxTopK];
  __shared__ int s_idx[kWarpsPerBlock][kMaxTopK];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * kWarpsPerBlock + warp;
  const int64_t n_rows = n_rows_dev ? (int64_t)*n_rows_dev : T_rows;
  if (row >= T_rows || row >= n_rows) return;
  const T* x = logits + row * ld_logits;

  if (use_provided_indx) {
    for (int j = lane; j < k; j += 32) {
      int e = indx[row * ld_indx + j];
      s_idx[warp][j] = e;
      s_val[warp][j] = to_f32<T>(x[e]);
    }
  } else {
    // rows of up to 256 experts are read once and kept as packed keys in registers
    constexpr int kRegKeys = 8;
    unsigned long long keys[kRegKeys];
    const bool in_regs = E <= 32 * kRegKeys;
    if (in_regs) {
#pragma unroll
      for (int u = 0; u < kRegKeys; ++u) {
        const int e = lane + 32 * u;
        keys[u] = e < E ? (((unsigned long long)float_key(to_f32<T>(x[e])) << 32) | (uint32_t)(~(uint32_t)e)) : 0ull;
      }
    }
    unsigned long long prev = ~0ull;
    for (int j = 0; j < k; ++j) {
      unsigned long long best = 0ull;
      if (in_regs) {
#pragma unroll
        for (int u = 0; u < kRegKeys; ++u)
          if (keys[u] < prev && keys[u] > best) best = keys[u];
      } else {
        for (int e = lane; e < E; e += 32) {
          unsigned long long key = ((unsigned long long)float_key(to_f32<T>(x[e])) << 32) | (uint32_t)(~(uint32_t)e);
          if (key < prev && key > best) best = key;
        }
      }
      best = warp_max_u64(best);
      prev = best;
      if (lane == 0) {
        s_idx[warp][j] = (int)(~(uint32_t)(best & 0xFFFFFFFFull));
        s_val[warp][j] = key_float((uint32_t)(best >> 32));
      }
    }
  }
  __syncwarp();

  if (apply_softmax) {
    float mx = -INFINITY;
    for (int j = 0; j < k; ++j) mx = fmaxf(mx, s_val[warp][j]);
    float sum = 0.0f;
    for (int j = 0; j < k; ++j) sum += expf(s_val[warp][j] - mx);
    for (int j = lane; j < k; j += 32) vals[row * ld_vals + j] = from_f32<T>(__fdiv_rn(expf(s_val[warp][j] - mx), sum));
  } else {
    for (int j = lane; j < k; j += 32) vals[row * ld_vals + j] = from_f32<T>(s_val[warp][j]);
  }
  if (!use_provided_indx)
    for (int j = lane; j < k; j += 32) indx[row * ld_indx + j] = (int16_t)s_idx[warp][j];

  const int words = (E + 31) >> 5;
  for (int w = lane; w < words; w += 32) {
    uint32_t bits = 0;
    for (int j = 0; j < k; ++j) {
      int e = s_idx[warp][j];
      if ((e >> 5) == w) bits |= 1u << (e & 31);
    }
    bitmatrix[row * bm_stride_row + (int64_t)w * bm_stride_word] = bits;
  }
}

// Four lanes per token row (k in {1, 2, 4, 8, 16}, every row valid, no provided indices; `parts` lanes for small batches).
// Lane `part` of a row's four walks the chunks of four experts c = part, part + 4, ... with best-k lists in registers (two
// lists side by side for k <= 4: independent insertion chains), the four lanes' lists meet by shuffles, lane 0 writes values
// and indices and the four lanes share the bitmatrix words.  With HIST the block (256 rows) also counts its picks per expert into
// partial[block][e], the first pass of the expert sort.  The warp-per-row kernel above spends its time in k rounds of
// 64-bit warp reductions per row: 19.6 us for 16384 x 128 logits against about 5 us here.
template <typename T, int K>
__device__ __forceinline__ TopK<K> quad_select(const T* x, int E, int part, int parts = 4) {
  constexpr int NL = K <= 4 ? 2 : 1;
  TopK<K> sub[NL];
  float v[NL][4];
  auto load = [&](int c0, float (&to)[NL][4]) {
#pragma unroll
    for (int u = 0; u < NL; ++u)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int e = (c0 + parts * u) * 4 + i;
        to[u][i] = e < E ? to_f32<T>(x[e]) : 0.0f;
      }
  };
  load(part, v);
  for (int c0 = part; c0 * 4 < E; c0 += parts * NL) {
    float next[NL][4];                             // in flight while this chunk is inserted
    load(c0 + parts * NL, next);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int u = 0; u < NL; ++u) {               // the lists alternate; each takes its experts in ascending order
        const int e = (c0 + parts * u) * 4 + i;
        if (e < E) sub[u].push(v[u][i], e);
      }
#pragma unroll
    for (int u = 0; u < NL; ++u)
#pragma unroll
      for (int i = 0; i < 4; ++i) v[u][i] = next[u][i];
  }
  TopK<K> tk = sub[0];
#pragma unroll
  for (int u = 1; u < NL; ++u) tk.merge(sub[u].key, sub[u].idx);
  tk.merge_lanes(parts);
  return tk;
}

// values (softmax over the picks), indices, bitmatrix words of one row; `hist` (shared memory, may be NULL) counts the picks,
// s_pick and s_val (shared memory, may be NULL) keep the row's picks and values for the block
template <typename T, int K>
__device__ __forceinline__ void quad_store(const TopK<K>& tk, int part, int64_t row, int E, int apply_softmax, T* __restrict__ vals,
                                           int64_t ld_vals, int16_t* __restrict__ indx, int64_t ld_indx,
                                           uint32_t* __restrict__ bitmatrix, int64_t bm_stride_row, int64_t bm_stride_word,
                                           int32_t* hist, int parts = 4, int16_t* s_pick = nullptr, float* s_val = nullptr) {
  if (part == 0) {
    float v[K];
#pragma unroll
    for (int i = 0; i < K; ++i) v[i] = sel_key_float(tk.key[i]);
    if (apply_softmax) {
      float mx = -INFINITY;
#pragma unroll
      for (int i = 0; i < K; ++i) mx = fmaxf(mx, v[i]);
      float sum = 0.0f;
#pragma unroll
      for (int i = 0; i < K; ++i) sum += expf(v[i] - mx);
#pragma unroll
      for (int i = 0; i < K; ++i) v[i] = __fdiv_rn(expf(v[i] - mx), sum);
    }
#pragma unroll
    for (int i = 0; i < K; ++i) {
      vals[row * ld_vals + i] = from_f32<T>(v[i]);
      indx[row * ld_indx + i] = (int16_t)tk.idx[i];
      if (hist) atomicAdd(&hist[tk.idx[i]], 1);
      if (s_pick) {
        s_pick[i] = (int16_t)tk.idx[i];
        s_val[i] = to_f32<T>(from_f32<T>(v[i]));
      }
    }
  }
  const int words = (E + 31) >> 5;
  for (int w = part; w < words; w += parts) {
    uint32_t bits = 0;
#pragma unroll
    for (int i = 0; i < K; ++i)
      if ((tk.idx[i] >> 5) == w) bits |= 1u << (tk.idx[i] & 31);
    bitmatrix[row * bm_stride_row + (int64_t)w * bm_stride_word] = bits;
  }
}

template <typename T, int K, bool HIST>
__global__ void __launch_bounds__(HIST ? 1024 : 256) topk_quad_kernel(
    const T* logits, int64_t ld_logits, int64_t T_rows, int E, int apply_softmax, T* vals, int64_t ld_vals, int16_t* indx,
    int64_t ld_indx, uint32_t* bitmatrix, int64_t bm_stride_row, int64_t bm_stride_word, int32_t* partial) {
  extern __shared__ int32_t s_hist[];                     // [E] with HIST
  pdl_begin();
  if constexpr (HIST) {
    for (int e = threadIdx.x; e < E; e += blockDim.x) s_hist[e] = 0;
    __syncthreads();
  }
  const int part = threadIdx.x & 3;
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 2) + (threadIdx.x >> 2);
  const bool live = row < T_rows;
  const T* x = logits + (live ? row : 0) * ld_logits;      // rows past the end walk row 0 and store nothing
  const TopK<K> tk = quad_select<T, K>(x, E, part);
  if (live)
    quad_store<T, K>(tk, part, row, E, apply_softmax, vals, ld_vals, indx, ld_indx, bitmatrix, bm_stride_row, bm_stride_word,
                     HIST ? s_hist : nullptr);
  if constexpr (HIST) {
    __syncthreads();
    for (int e = threadIdx.x; e < E; e += blockDim.x) partial[(int64_t)blockIdx.x * E + e] = s_hist[e];
  }
}

// ---------------------------------------------------------------------------------------------------
// Expert histogram + stable expert-major sort.  Flat entry i = token * k + slot, expert c = indx[i]
// (negative, or token >= n_rows: dropped).  row_sorted[i] = col_offs[c] + #{j < i : indx[j] == c},
// col_sorted = inverse permutation; both -1 padded.  Three passes (up to 32768 entries of 256 experts: bm_wide_kernel below):
//   pass 1: per block of kTokPerBlock tokens, a shared-memory histogram -> partial[blk][e]; both index arrays
//           pre-filled with -1.
//   pass 2: exclusive scan of partial[.][e] over blocks, totals -> col_sum, their exclusive scan -> col_offs.
//   pass 3: rank inside the block: each warp owns 32 consecutive tokens and ranks them in order with
//           warp match, on top of the counts of the warps before it.
constexpr int kTokPerBlock = 256;

__device__ __forceinline__ int entry_expert(const int16_t* indx, int64_t ld_indx, int k, int64_t token, int slot,
                                            int64_t n_rows, int E) {
  if (token >= n_rows) return -1;
  int c = indx[token * ld_indx + slot];
  return (c < 0 || c >= E) ? -1 : c;
}

__global__ void __launch_bounds__(256) bm_hist_kernel(const int16_t* indx, int64_t ld_indx, int64_t T_rows,
                                                      int E, int k, const int32_t* n_rows_dev,
                                                      int32_t* partial, int32_t* col_sorted, int32_t* row_sorted) {
  pdl_begin();
  extern __shared__ int32_t s_cnt[];
  const int64_t n_rows = n_rows_dev ? min((int64_t)*n_rows_dev, T_rows) : T_rows;
  for (int e = threadIdx.x; e < E; e += blockDim.x) s_cnt[e] = 0;
  __syncthreads();
  const int64_t tok0 = (int64_t)blockIdx.x * kTokPerBlock;
  const int64_t n_ent = (int64_t)kTokPerBlock * k;
  // four loads in flight (one at a time: 6.1 us for 4100 tokens, so 3.7)
  for (uint32_t j0 = threadIdx.x; j0 < n_ent; j0 += 4 * blockDim.x) {
    int c[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint32_t j = j0 + u * blockDim.x;
      const int64_t token = tok0 + j / (uint32_t)k;
      c[u] = j < n_ent && token < T_rows ? entry_expert(indx, ld_indx, k, token, (int)(j % (uint32_t)k), n_rows, E) : -1;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint32_t j = j0 + u * blockDim.x;
      if (j < n_ent && tok0 + j / (uint32_t)k < T_rows) {
        col_sorted[tok0 * k + j] = -1;
        row_sorted[tok0 * k + j] = -1;
      }
      if (c[u] >= 0) atomicAdd(&s_cnt[c[u]], 1);
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    partial[(int64_t)blockIdx.x * E + e] = s_cnt[e];
  }
}

// block-wide exclusive scan of `n` ints (in place allowed), returns nothing; one block only.
__device__ void block_exclusive_scan(const int32_t* in, int32_t* out, int n, int32_t* s_warp /*[33]*/) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  int carry = 0;
  for (int base = 0; base < n; base += blockDim.x) {
    int i = base + threadIdx.x;
    int v = (i < n) ? in[i] : 0;
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
      if (lane >= o) inc += t;
    }
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    if (warp == 0) {
      int w = (lane < nwarps) ? s_warp[lane] : 0;
      int winc = w;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(0xFFFFFFFFu, winc, o);
        if (lane >= o) winc += t;
      }
      s_warp[lane] = winc - w;          // exclusive warp offsets
      if (lane == 31) s_warp[32] = winc;  // chunk total
    }
    __syncthreads();
    if (i < n) out[i] = carry + s_warp[warp] + inc - v;
    carry += s_warp[32];
    __syncthreads();
  }
}

// One block: exclusive scan of partial[.][e] over the blocks of tokens, by S segments of blocks per expert (1024 experts at a time),
// the expert totals (col_sum) and their exclusive scan (col_offs).  Totals added up by atomics in the pass before would want a cleared
// array, a launch of its own.
__global__ void __launch_bounds__(1024) bm_scan_kernel(int32_t* partial, int64_t n_blocks, int E, int32_t* col_sum, int32_t* col_offs) {
  pdl_begin();
  __shared__ int32_t s_seg[1024];
  __shared__ int32_t s_warp[33];
  int Ep = 1;
  while (Ep < E && Ep < 1024) Ep <<= 1;
  const int S = 1024 / Ep, seg = threadIdx.x / Ep;
  const int64_t per = (n_blocks + S - 1) / S;
  const int64_t b_lo = min((int64_t)seg * per, n_blocks), b_hi = min(b_lo + per, n_blocks);
  for (int e0 = 0; e0 < E; e0 += Ep) {
    const int e = e0 + (int)(threadIdx.x % Ep);
    // sixteen loads in flight per thread: the walk is a chain of L2 round trips otherwise
    auto walk = [&](int run, bool store) {
      if (e < E)
        for (int64_t b0 = b_lo; b0 < b_hi; b0 += 16) {
          int v[16];
#pragma unroll
          for (int u = 0; u < 16; ++u) v[u] = b0 + u < b_hi ? partial[(b0 + u) * E + e] : 0;
#pragma unroll
          for (int u = 0; u < 16; ++u) {
            if (store && b0 + u < b_hi) partial[(b0 + u) * E + e] = run;
            run += v[u];
          }
        }
      return run;
    };
    s_seg[threadIdx.x] = walk(0, false);
    __syncthreads();
    int run = 0, total = 0;
    for (int i = 0; i < S; ++i) {
      const int v = s_seg[i * Ep + (int)(threadIdx.x % Ep)];
      if (i < seg) run += v;
      total += v;
    }
    walk(run, true);
    if (seg == 0 && e < E) col_sum[e] = total;
    __syncthreads();
  }
  block_exclusive_scan(col_sum, col_offs, E, s_warp);
}

// What the layer wants per expert-sorted position beside the permutation: token row and routing weight (token NULL: nothing).
struct PerPosition {
  int32_t* token = nullptr;
  float* weight = nullptr;
  const float* vals = nullptr;
  int64_t ld_vals = 0;
};

// Positions of the entries of one block of blockDim.x tokens starting at token `tok_base`: `base[e]` is where the
// block's entries of expert e start (expert offset + entries of earlier blocks); s_cnt holds [warps][E] counters.
__device__ __forceinline__ void rank_block(const int16_t* indx, int64_t ld_indx, int64_t T_rows, int E, int k,
                                           int64_t n_rows, const int32_t* base_a, const int32_t* base_b, int64_t tok_base,
                                           int32_t* __restrict__ col_sorted, int32_t* __restrict__ row_sorted, int32_t* s_cnt,
                                           const PerPosition& out = PerPosition()) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  int32_t* my = s_cnt + (int64_t)warp * E;
  for (int i = threadIdx.x; i < nwarps * E; i += blockDim.x) s_cnt[i] = 0;
  __syncthreads();
  const int64_t tok0 = tok_base + warp * 32;
  const int n_ent = 32 * k;
  // count the entries of this warp's 32 tokens
  for (int j = lane; j < n_ent; j += 32) {
    int c = entry_expert(indx, ld_indx, k, tok0 + j / k, j % k, n_rows, E);
    if (c >= 0) atomicAdd(&my[c], 1);
  }
  __syncthreads();
  // turn the per-warp counts into starting offsets: base + counts of the warps before this one
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    int run = (base_a ? base_a[e] : 0) + base_b[e];
    for (int w = 0; w < nwarps; ++w) {
      int v = s_cnt[w * E + e];
      s_cnt[w * E + e] = run;
      run += v;
    }
  }
  __syncthreads();
  // rank in order, 32 entries at a time
  for (int j0 = 0; j0 < n_ent; j0 += 32) {
    const int j = j0 + lane;
    const int64_t token = tok0 + j / k;
    const int slot = j % k;
    int c = (j < n_ent && token < T_rows) ? entry_expert(indx, ld_indx, k, token, slot, n_rows, E) : -1;
    const unsigned peers = __match_any_sync(0xFFFFFFFFu, c);
    const int before = __popc(peers & ((1u << lane) - 1u));
    int base = 0;
    if (c >= 0) base = my[c];
    __syncwarp();
    if (c >= 0 && before == 0) my[c] = base + __popc(peers);
    __syncwarp();
    if (c >= 0) {
      const int pos = base + before;
      const int64_t flat = token * k + slot;
      row_sorted[flat] = pos;
      col_sorted[pos] = (int32_t)flat;
      if (out.token) {
        out.token[pos] = (int32_t)token;
        if (out.weight) out.weight[pos] = out.vals[token * out.ld_vals + slot];
      }
    }
  }
}

__global__ void __launch_bounds__(256) bm_rank_kernel(const int16_t* indx, int64_t ld_indx, int64_t T_rows, int E, int k,
                                                      const int32_t* n_rows_dev, const int32_t* partial,
                                                      const int32_t* col_offs, int32_t* col_sorted, int32_t* row_sorted,
                                                      const PerPosition out) {
  extern __shared__ int32_t s_cnt[];  // [warps][E]; a block covers blockDim.x tokens, the blocks of `partial`
  pdl_begin();
  const int64_t n_rows = n_rows_dev ? min((int64_t)*n_rows_dev, T_rows) : T_rows;
  rank_block(indx, ld_indx, T_rows, E, k, n_rows, partial + (int64_t)blockIdx.x * E, col_offs, (int64_t)blockIdx.x * blockDim.x,
             col_sorted, row_sorted, s_cnt, out);
}

constexpr int kRouteCluster = 8;
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ int ld_cluster(const int32_t* shared, uint32_t rank) {      // the same variable of another block
  uint32_t at = (uint32_t)__cvta_generic_to_shared(shared), v;
  asm volatile("{\n\t.reg .b32 ra;\n\tmapa.shared::cluster.u32 ra, %1, %2;\n\tld.shared::cluster.u32 %0, [ra];\n\t}" : "=r"(v) : "r"(at), "r"(rank) : "memory");
  return (int)v;
}


// The sort of up to 32768 entries in one launch of blocks that do not wait on one another: a block ranks 1024 entries, one to a thread, and
// counts all of them for itself, those ahead of its own apart (two counters per expert, in four copies against threads that
// meet on one).  Every chain is short: a read of at most 64 KB from L2, its counts, a scan of the experts, a prefix over the warps.  As one cluster of eight
// blocks with an eighth of the entries each the counts took two cluster barriers and three rounds of a warp's matches.  Behind the router, before and now: 1 token
// 16.6 -> 16.0 us, 4100 tokens of 128 experts, k = 4, 29.2 -> 26.7, k = 8 35.1 -> 29.7, 8192 tokens 32.9 -> 31.9.
constexpr int kSortWideEntries = 32768, kSortWideBlock = 1024, kSortWideCopies = 4;
__global__ void __launch_bounds__(kSortWideBlock) bm_wide_kernel(const int16_t* indx, int64_t ld_indx, int T_rows, int E, int k, const int32_t* n_rows_dev,
                                                                 int32_t* col_sum, int32_t* col_sorted, int32_t* row_sorted) {
  // [copies][2][E] counts, [E] sizes, [E] offsets, [E] entries of the blocks before, [32][E] first positions of a warp's entries
  extern __shared__ int32_t s_mem[];
  __shared__ int32_t s_warp[33];
  pdl_begin();
  const int n = T_rows * k, first = (int)blockIdx.x * kSortWideBlock, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_rows = n_rows_dev ? min(max(*n_rows_dev, 0), T_rows) : T_rows, live = n_rows * k;      // entries that count
  int32_t* s_size = s_mem + 2 * kSortWideCopies * E;
  int32_t* s_offs = s_size + E;
  int32_t* s_before = s_offs + E;
  int32_t* s_cnt = s_before + E;
  for (int i = threadIdx.x; i < 2 * kSortWideCopies * E; i += kSortWideBlock) s_mem[i] = 0;
  for (int i = threadIdx.x; i < 32 * E; i += kSortWideBlock) s_cnt[i] = 0;
  const int j = first + (int)threadIdx.x;
  const int c = j < live ? entry_expert(indx, ld_indx, k, j / k, j % k, n_rows, E) : -1;
  __syncthreads();
  int32_t* copy = s_mem + (warp & (kSortWideCopies - 1)) * 2 * E;
  int done = 0;                                      // entries counted eight at a time: rows without a gap, on a 16-byte boundary
  if (ld_indx == k && (uintptr_t)indx % 16 == 0) {
    done = live & ~7;
    for (int i = (int)threadIdx.x * 8; i < done; i += kSortWideBlock * 8) {
      const uint4 v = *reinterpret_cast<const uint4*>(indx + i);
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
      int32_t* at = copy + (i >= first ? E : 0);     // (`first` is a multiple of eight)
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int e = (int16_t)(w[u >> 1] >> (16 * (u & 1)));
        if (e >= 0 && e < E) atomicAdd(at + e, 1);
      }
    }
  }
  for (int i = done + (int)threadIdx.x; i < live; i += kSortWideBlock) {
    const int e = entry_expert(indx, ld_indx, k, i / k, i % k, n_rows, E);
    if (e >= 0) atomicAdd(copy + (i >= first ? E : 0) + e, 1);
  }
  const unsigned peers = __match_any_sync(0xFFFFFFFFu, c);
  const int rank = __popc(peers & ((1u << lane) - 1u));
  if (c >= 0 && rank == 0) s_cnt[warp * E + c] = __popc(peers);
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += kSortWideBlock) {
    int before = 0, total = 0;
#pragma unroll
    for (int i = 0; i < kSortWideCopies; ++i) {
      before += s_mem[2 * i * E + e];
      total += s_mem[(2 * i + 1) * E + e];
    }
    total += before;
    s_size[e] = total;
    s_before[e] = before;
    if (blockIdx.x == 0) col_sum[e] = total;
  }
  __syncthreads();
  block_exclusive_scan(s_size, s_offs, E, s_warp);
  const int kept = s_offs[E - 1] + s_size[E - 1];
  for (int e = threadIdx.x; e < E; e += kSortWideBlock) {
    int run = s_offs[e] + s_before[e];
#pragma unroll
    for (int w0 = 0; w0 < 32; w0 += 8) {
      int v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = s_cnt[(w0 + u) * E + e];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        s_cnt[(w0 + u) * E + e] = run;
        run += v[u];
      }
    }
  }
  if (j < n && j >= kept) col_sorted[j] = -1;        // positions past the last entry that counts
  __syncthreads();
  const int at = c >= 0 ? s_cnt[warp * E + c] + rank : -1;
  if (j < n) row_sorted[j] = at;
  if (c >= 0) col_sorted[at] = j;
}

// ---------------------------------------------------------------------------------------------------
// Ragged metadata.  blockIdx.x = 0: slice_offs (block size 1); 1..4: block sizes 16,32,64,128.
// Every block scans its own offsets into shared memory; blockIdx.y == 0 writes them out; all blocks of
// a row fill their chunk of the schedule by binary search: sched[p] = ((p - offs[e]) << 16) | e.
constexpr int kSchedChunk = 4096;

__global__ void __launch_bounds__(1024) ragged_kernel(const int32_t* __restrict__ slice_sizes, int E,
                                                      int32_t* __restrict__ slice_offs, int32_t* __restrict__ block_offs,
                                                      int64_t ld_block_offs, int32_t* __restrict__ block_sched,
                                                      int64_t ld_sched, int64_t n_sched) {
  extern __shared__ int32_t s_offs[];  // [E + 1] then scratch [E + 1]
  __shared__ int32_t s_warp[33];
  const int row = blockIdx.x;                     // 0 = slice_offs
  const int log2bs = row == 0 ? 0 : row + 3;
  int32_t* s_nb = s_offs + (E + 1);
  for (int e = threadIdx.x; e <= E; e += blockDim.x)
    s_nb[e] = (e < E) ? (int32_t)(((int64_t)max(slice_sizes[e], 0) + ((1 << log2bs) - 1)) >> log2bs) : 0;
  __syncthreads();
  block_exclusive_scan(s_nb, s_offs, E + 1, s_warp);
  __syncthreads();
  int32_t* dst = row == 0 ? slice_offs : block_offs + (int64_t)(row - 1) * ld_block_offs;
  if (blockIdx.y == 0)
    for (int e = threadIdx.x; e <= E; e += blockDim.x) dst[e] = s_offs[e];
  if (row == 0) return;
  const int32_t total = s_offs[E];
  int32_t* sched = block_sched + (int64_t)(row - 1) * ld_sched;
  const int64_t p0 = (int64_t)blockIdx.y * kSchedChunk;
  for (int64_t p = p0 + threadIdx.x; p < min(p0 + kSchedChunk, n_sched); p += blockDim.x) {
    int32_t v = -1;
    if (p < total) {
      int lo = 0, hi = E;  // largest e with offs[e] <= p
      while (hi - lo > 1) {
        int mid = (lo + hi) >> 1;
        if (s_offs[mid] <= p) lo = mid; else hi = mid;
      }
      v = (int32_t)(((uint32_t)(p - s_offs[lo]) << 16) | (uint32_t)lo);
    }
    sched[p] = v;
  }
}

// Stable compaction by one block: out[rank(i)] = val(i) for kept i, tail filled with -1. Returns the count.
template <typename ValFn, typename KeepFn>
__device__ int block_compact(int32_t* out, int64_t n, ValFn val, KeepFn keep, int32_t* s_warp) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  int carry = 0;
  for (int64_t base = 0; base < n; base += blockDim.x) {
    const int64_t i = base + threadIdx.x;
    const bool kp = (i < n) && keep(i);
    const unsigned m = __ballot_sync(0xFFFFFFFFu, kp);
    if (lane == 0) s_warp[warp] = __popc(m);
    __syncthreads();
    int off = 0, tot = 0;
    for (int w = 0; w < nwarps; ++w) {
      int c = s_warp[w];
      if (w < warp) off += c;
      tot += c;
    }
    if (kp) out[carry + off + __popc(m & ((1u << lane) - 1u))] = val(i);
    carry += tot;
    __syncthreads();
  }
  for (int64_t i = carry + threadIdx.x; i < n; i += blockDim.x) out[i] = -1;
  return carry;
}

__global__ void __launch_bounds__(1024) ragged_remap_kernel(
    const int32_t* __restrict__ slice_sizes, const int32_t* __restrict__ slice_offs,
    const int32_t* __restrict__ block_offs, int64_t ld_block_offs, const int32_t* __restrict__ block_sched,
    int64_t ld_sched, int64_t n_sched, const int32_t* __restrict__ slice_map, int E, int32_t* __restrict__ o_sizes,
    int32_t* __restrict__ o_offs, int32_t* __restrict__ o_block_offs, int32_t* __restrict__ o_sched) {
  __shared__ int32_t s_warp[32];
  const int b = blockIdx.x;
  auto keep_slice = [&](int64_t i) { return i < E && slice_map[i] != -1; };
  if (b == 0) {
    block_compact(o_sizes, E, [&](int64_t i) { return slice_sizes[i]; }, keep_slice, s_warp);
    __syncthreads();
    block_compact(o_offs, E + 1, [&](int64_t i) { return slice_offs[i]; }, keep_slice, s_warp);
    __syncthreads();
  }
  const int32_t* bo = block_offs + (int64_t)b * ld_block_offs;
  const int32_t* bs = block_sched + (int64_t)b * ld_sched;
  int32_t* obo = o_block_offs + (int64_t)b * ld_block_offs;
  int32_t* obs = o_sched + (int64_t)b * ld_sched;
  const int n_kept = block_compact(obo, E + 1, [&](int64_t i) { return bo[i]; }, keep_slice, s_warp);
  __syncthreads();
  const int n_blk = block_compact(
      obs, n_sched,
      [&](int64_t i) {
        uint32_t v = (uint32_t)bs[i];
        return (int32_t)((v & 0xFFFF0000u) | (uint32_t)slice_map[v & 0xFFFFu]);
      },
      [&](int64_t i) {
        uint32_t v = (uint32_t)bs[i];
        uint32_t s = v & 0xFFFFu;
        return s != 0xFFFFu && (int)s < E && slice_map[s] != -1;
      },
      s_warp);
  __syncthreads();
  if (threadIdx.x == 0) obo[n_kept] = n_blk;
}

}  // namespace

extern "C" __attribute__((visibility("default"))) int moe_topk_fwd(const void* logits, int dtype, int64_t T, int E, int k, int apply_softmax,
                            int64_t ld_logits, void* vals, int64_t ld_vals, int16_t* indx, int64_t ld_indx,
                            uint32_t* bitmatrix, int64_t bm_stride_row, int64_t bm_stride_word,
                            const int32_t* n_rows_dev, int use_provided_indx, void* stream) {
  MOE_CHECK_ARG(T >= 0 && E > 0 && E < 32768, "moe_topk_fwd: need 0 < n_expts < 32768, got %d", E);
  MOE_CHECK_ARG(k > 0 && k <= kMaxTopK && k <= E, "moe_topk_fwd: need 0 < k <= min(%d, n_expts), got %d", kMaxTopK, k);
  if (T == 0) return MOE_OK;
  MOE_CHECK_ARG(logits && vals && indx && bitmatrix, "moe_topk_fwd: NULL pointer");
  cudaStream_t st = (cudaStream_t)stream;
  if (!use_provided_indx && n_rows_dev == nullptr && (k == 1 || k == 2 || k == 4 || k == 8 || k == 16)) {
    const int qgrid = (int)cdiv64(T, 64);
#define MOE_TOPK_QUAD(KK)                                                                                                 \
  MOE_DISPATCH_FLOAT(dtype, Tv, {                                                                                         \
    MOE_CHECK_CUDA(launch_pdl(topk_quad_kernel<Tv, KK, false>, dim3(qgrid), dim3(256), 0, st, (const Tv*)logits, ld_logits, \
                              T, E, apply_softmax, (Tv*)vals, ld_vals, indx, ld_indx, bitmatrix, bm_stride_row,             \
                              bm_stride_word, nullptr));                                                                    \
  })
    switch (k) {
      case 1: MOE_TOPK_QUAD(1); break;
      case 2: MOE_TOPK_QUAD(2); break;
      case 4: MOE_TOPK_QUAD(4); break;
      case 8: MOE_TOPK_QUAD(8); break;
      default: MOE_TOPK_QUAD(16); break;
    }
#undef MOE_TOPK_QUAD
    MOE_CHECK_LAUNCH();
    return MOE_OK;
  }
  const int grid = (int)cdiv64(T, kWarpsPerBlock);
  MOE_DISPATCH_FLOAT(dtype, Tv, {
    topk_kernel<Tv><<<grid, kWarpsPerBlock * 32, 0, st>>>((const Tv*)logits, ld_logits, T, E, k, apply_softmax,
                                                          (Tv*)vals, ld_vals, indx, ld_indx, bitmatrix, bm_stride_row,
                                                          bm_stride_word, n_rows_dev, use_provided_indx);
  });
  MOE_CHECK_LAUNCH();
  return MOE_OK;
}

extern "C" __attribute__((visibility("default"))) size_t moe_bitmatrix_metadata_workspace(int64_t T, int E, int k) {
  (void)k;
  const int64_t nb = cdiv64(T > 0 ? T : 1, kTokPerBlock);
  return (size_t)((nb * E + E) * (int64_t)sizeof(int32_t));
}

extern "C" __attribute__((visibility("default"))) int moe_bitmatrix_metadata(const int16_t* indx, int64_t ld_indx, int64_t T, int E, int k,
                                      const int32_t* n_rows_dev, int32_t* col_sum, int32_t* col_sorted,
                                      int32_t* row_sorted, void* workspace, size_t workspace_bytes, void* stream) {
  MOE_CHECK_ARG(T >= 0 && E > 0 && k > 0, "moe_bitmatrix_metadata: bad extents T=%lld E=%d k=%d", (long long)T, E, k);
  MOE_CHECK_ARG(col_sum, "moe_bitmatrix_metadata: col_sum is NULL");
  cudaStream_t st = (cudaStream_t)stream;
  if (T == 0) {
    MOE_CHECK_CUDA(cudaMemsetAsync(col_sum, 0, sizeof(int32_t) * (size_t)E, st));
    return MOE_OK;
  }
  MOE_CHECK_ARG(indx && col_sorted && row_sorted && workspace, "moe_bitmatrix_metadata: NULL pointer");
  MOE_CHECK_ARG(workspace_bytes >= moe_bitmatrix_metadata_workspace(T, E, k),
                "moe_bitmatrix_metadata: workspace too small (%zu < %zu)", workspace_bytes,
                moe_bitmatrix_metadata_workspace(T, E, k));
  if (T * k <= kSortWideEntries && E <= 256) {
    const size_t smem = (size_t)(2 * kSortWideCopies + 3 + 32) * E * sizeof(int32_t);      // <= 43 KB
    MOE_CHECK_CUDA(launch_pdl(bm_wide_kernel, dim3((unsigned)cdiv64(T * k, kSortWideBlock)), dim3(kSortWideBlock), smem, st, indx, ld_indx, (int)T, E, k,
                              n_rows_dev, col_sum, col_sorted, row_sorted));
    MOE_CHECK_LAUNCH();
    return MOE_OK;
  }
  const size_t smem_rank = (size_t)8 * E * sizeof(int32_t);
  MOE_CHECK_ARG(smem_rank <= 200 * 1024, "moe_bitmatrix_metadata: n_expts=%d too large for the shared-memory counters", E);
  const int64_t nb = cdiv64(T, kTokPerBlock);
  int32_t* partial = (int32_t*)workspace;
  int32_t* col_offs = partial + nb * E;
  MOE_CHECK_CUDA(launch_pdl(bm_hist_kernel, dim3((unsigned)nb), dim3(256), (size_t)E * sizeof(int32_t), st, indx, ld_indx, T, E, k,
                            n_rows_dev, partial, col_sorted, row_sorted));
  MOE_CHECK_LAUNCH();
  MOE_CHECK_CUDA(launch_pdl(bm_scan_kernel, dim3(1), dim3(1024), 0, st, partial, nb, E, col_sum, col_offs));
  MOE_CHECK_LAUNCH();
  if (smem_rank > 48 * 1024)
    MOE_CHECK_CUDA(cudaFuncSetAttribute(bm_rank_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_rank));
  MOE_CHECK_CUDA(launch_pdl(bm_rank_kernel, dim3((unsigned)nb), dim3(256), smem_rank, st, indx, ld_indx, T, E, k, n_rows_dev, partial,
                            col_offs, col_sorted, row_sorted, PerPosition()));
  MOE_CHECK_LAUNCH();
  return MOE_OK;
}

extern "C" __attribute__((visibility("default"))) int moe_ragged_metadata(const int32_t* slice_sizes, int E, int32_t* slice_offs, int32_t* block_offs,
                                   int64_t ld_block_offs, int32_t* block_sched, int64_t ld_sched, int64_t n_sched,
                                   void* stream) {
  MOE_CHECK_ARG(E > 0 && E < 65535, "moe_ragged_metadata: need 0 < n_slices < 65535, got %d", E);
  MOE_CHECK_ARG(slice_sizes && slice_offs && block_offs && (block_sched || n_sched == 0), "moe_ragged_metadata: NULL pointer");
  MOE_CHECK_ARG(ld_block_offs >= E + 1 && ld_sched >= n_sched, "moe_ragged_metadata: leading dimensions too small");
  const size_t smem = (size_t)2 * (E + 1) * sizeof(int32_t);
  cudaStream_t st = (cudaStream_t)stream;
  if (smem > 48 * 1024)
    MOE_CHECK_CUDA(cudaFuncSetAttribute(ragged_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  dim3 grid(5, (unsigned)(n_sched > 0 ? cdiv64(n_sched, kSchedChunk) : 1));
  ragged_kernel<<<grid, 1024, smem, st>>>(slice_sizes, E, slice_offs, block_offs, ld_block_offs, block_sched, ld_sched,
                                          n_sched);
  MOE_CHECK_LAUNCH();
  return MOE_OK;
}

extern "C" __attribute__((visibility("default"))) int moe_ragged_metadata_remap(const int32_t* slice_sizes, const int32_t* slice_offs,
                                         const int32_t* block_offs, int64_t ld_block_offs, const int32_t* block_sched,
                                         int64_t ld_sched, int64_t n_sched, const int32_t* slice_map, int E,
                                         int32_t* out_slice_sizes, int32_t* out_slice_offs, int32_t* out_block_offs,
                                         int32_t* out_block_sched, void* stream) {
  MOE_CHECK_ARG(E > 0 && E < 65535, "moe_ragged_metadata_remap: need 0 < n_slices < 65535, got %d", E);
  MOE_CHECK_ARG(slice_sizes && slice_offs && block_offs && slice_map && out_slice_sizes && out_slice_offs &&
                    out_block_offs && (n_sched == 0 || (block_sched && out_block_sched)),
                "moe_ragged_metadata_remap: NULL pointer");
  ragged_remap_kernel<<<4, 1024, 0, (cudaStream_t)stream>>>(slice_sizes, slice_offs, block_offs, ld_block_offs,
                                                            block_sched, ld_sched, n_sched, slice_map, E,
                                                            out_slice_sizes, out_slice_offs, out_block_offs,
                                                            out_block_sched);
  MOE_CHECK_LAUNCH();
  return MOE_OK;
}

// ---------------------------------------------------------------------------------------------------------
// moe_route: the whole routing step in one to three launches (the standalone entry points above take more).  Small batches: one launch of five
// independent blocks (route_small_kernel); up to 896 tokens (2048 with short lists): one launch of a cluster of eight (route_cluster_kernel, both at the end of
// this section; rule: route_form).  Others: A, then route_finish_kernel where its blocks are a wave, else B and C.
//   A  topk_quad_kernel<HIST>   top-k + softmax + bitmatrix row of every token, and the expert histogram of each block
//      (route_topk_hist_kernel  of 128 tokens (partial[blk][e]) in the same pass over the logits;
//       for other k)
//   B  route_scan_ragged_kernel six blocks: exclusive scan of partial over the blocks and the expert totals (col_sum);
//                               their exclusive scan (col_offs = slice_offs); block_offs and block schedules of the four
//                               block sizes of the ragged metadata, which depend on the totals only;
//   C  bm_rank_kernel           positions of the entries (unchanged);
//   or  route_finish_kernel     B and C at once: every ranking block adds up the counts it needs itself.
// Every token row is valid in this form (no device-side row bound, no provided indices), so each (token, slot) entry
// receives a position and the index arrays need no -1 pre-fill.
namespace {

constexpr int kRouteTokPerBlock = 128;          // tokens per block of kernels A and C: 128 blocks for 16384 tokens
constexpr int kRouteWarps = 16;                 // warps per block of the warp-per-row form of kernel A: 8 token rows each
constexpr int kRowsPerWarp = kRouteTokPerBlock / kRouteWarps;

// One warp per token row, rows of up to 256 experts held as order-preserving keys in registers.  A pick is two warp
// reductions (redux.sync): the largest value key, then the smallest expert index among the lanes that hold it.
template <typename T>
__global__ void __launch_bounds__(kRouteWarps * 32) route_topk_hist_kernel(
    const T* logits, int64_t ld_logits, int64_t T_rows, int E, int k, int apply_softmax,
    T* vals, int64_t ld_vals, int16_t* indx, int64_t ld_indx,
    uint32_t* bitmatrix, int64_t bm_stride_row, int64_t bm_stride_word, int32_t* partial) {
  extern __shared__ int32_t s_hist[];                     // [E]
  pdl_begin();
  __shared__ float s_val[kRouteWarps][kMaxTopK];
  __shared__ int s_idx[kRouteWarps][kMaxTopK];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int e = threadIdx.x; e < E; e += blockDim.x) s_hist[e] = 0;
  __syncthreads();
  constexpr int kRegKeys = 8;
  const int64_t row0 = (int64_t)blockIdx.x * kRouteTokPerBlock + warp * kRowsPerWarp;
  const int words = (E + 31) >> 5;
  // the next row's logits are loaded before this row's picks start
  uint32_t nxt[kRegKeys];
  auto load_row = [&](int64_t row) {
#pragma unroll
    for (int u = 0; u < kRegKeys; ++u) {
      const int e = lane + 32 * u;
      nxt[u] = (row < T_rows && e < E) ? float_key(to_f32<T>(logits[row * ld_logits + e])) : 0u;
    }
  };
  load_row(row0);
  for (int i = 0; i < kRowsPerWarp; ++i) {
    const int64_t row = row0 + i;
    if (row >= T_rows) break;                              // warp-uniform
    uint32_t key[kRegKeys];
#pragma unroll
    for (int u = 0; u < kRegKeys; ++u) key[u] = nxt[u];
    if (i + 1 < kRowsPerWarp) load_row(row + 1);
    uint32_t alive = 0;
#pragma unroll
    for (int u = 0; u < kRegKeys; ++u)
      if (lane + 32 * u < E) alive |= 1u << u;
    for (int j = 0; j < k; ++j) {
      uint32_t bk = 0;
      int bu = -1;
#pragma unroll
      for (int u = 0; u < kRegKeys; ++u)
        if (((alive >> u) & 1u) && (bu < 0 || key[u] > bk)) { bk = key[u]; bu = u; }
      const uint32_t m = __reduce_max_sync(0xFFFFFFFFu, bu >= 0 ? bk : 0u);
      const uint32_t cand = (bu >= 0 && bk == m) ? (uint32_t)(lane + 32 * bu) : 0x7FFFFFFFu;
      const uint32_t win = __reduce_min_sync(0xFFFFFFFFu, cand);
      if ((int)(win & 31u) == lane && win != 0x7FFFFFFFu) alive &= ~(1u << (win >> 5));
      if (lane == 0) {
        s_idx[warp][j] = (int)win;
        s_val[warp][j] = key_float(m);
      }
    }
    __syncwarp();
    if (apply_softmax) {
      float mx = -INFINITY;
      for (int j = 0; j < k; ++j) mx = fmaxf(mx, s_val[warp][j]);
      float sum = 0.0f;
      for (int j = 0; j < k; ++j) sum += expf(s_val[warp][j] - mx);
      for (int j = lane; j < k; j += 32) vals[row * ld_vals + j] = from_f32<T>(__fdiv_rn(expf(s_val[warp][j] - mx), sum));
    } else {
      for (int j = lane; j < k; j += 32) vals[row * ld_vals + j] = from_f32<T>(s_val[warp][j]);
    }
    for (int j = lane; j < k; j += 32) {
      const int e = s_idx[warp][j];
      indx[row * ld_indx + j] = (int16_t)e;
      atomicAdd(&s_hist[e], 1);
    }
    for (int w = lane; w < words; w += 32) {
      uint32_t bits = 0;
      for (int j = 0; j < k; ++j) {
        const int e = s_idx[warp][j];
        if ((e >> 5) == w) bits |= 1u << (e & 31);
      }
      bitmatrix[row * bm_stride_row + (int64_t)w * bm_stride_word] = bits;
    }
    __syncwarp();
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) partial[(int64_t)blockIdx.x * E + e] = s_hist[e];
}

// One row of the ragged metadata from the slice sizes in shared memory (s_size[0..E), s_size[E] = 0): row 0 =
// slice_offs (= expert offsets, also written to col_offs when given), rows 1..4 = block_offs and block schedule of the
// block sizes 16..128.  All threads of the block call it.
__device__ void ragged_row(int row, const int32_t* s_size, int E, int32_t* s_nb, int32_t* s_offs, int32_t* s_warp,
                           int32_t* __restrict__ slice_offs, int32_t* __restrict__ col_offs, int32_t* __restrict__ block_offs,
                           int64_t ld_block_offs, int32_t* __restrict__ block_sched, int64_t ld_sched, int64_t n_sched) {
  const int log2bs = row == 0 ? 0 : row + 3;
  for (int i = threadIdx.x; i <= E; i += blockDim.x)
    s_nb[i] = (i < E) ? (int32_t)(((int64_t)s_size[i] + ((1 << log2bs) - 1)) >> log2bs) : 0;
  __syncthreads();
  block_exclusive_scan(s_nb, s_offs, E + 1, s_warp);
  __syncthreads();
  int32_t* dst = row == 0 ? slice_offs : block_offs + (int64_t)(row - 1) * ld_block_offs;
  for (int i = threadIdx.x; i <= E; i += blockDim.x) {
    dst[i] = s_offs[i];
    if (row == 0 && i < E && col_offs) col_offs[i] = s_offs[i];
  }
  if (row > 0) {
    const int32_t tot = s_offs[E];
    int32_t* sched = block_sched + (int64_t)(row - 1) * ld_sched;
    for (int64_t p = threadIdx.x; p < n_sched; p += blockDim.x) {
      int32_t v = -1;
      if (p < tot) {
        int lo = 0, hi = E;  // largest e with offs[e] <= p
        while (hi - lo > 1) {
          const int mid = (lo + hi) >> 1;
          if (s_offs[mid] <= p) lo = mid; else hi = mid;
        }
        v = (int32_t)(((uint32_t)(p - s_offs[lo]) << 16) | (uint32_t)lo);
      }
      sched[p] = v;
    }
  }
  __syncthreads();
}

// Six blocks of 1024 threads.  n_experts <= 1024.
__global__ void __launch_bounds__(1024) route_scan_ragged_kernel(const int32_t* partial_in,
                                                                 int32_t* partial_out, int64_t n_blocks, int E,
                                                                 int32_t* col_sum, int32_t* col_offs,
                                                                 int32_t* slice_offs, int32_t* block_offs,
                                                                 int64_t ld_block_offs, int32_t* block_sched,
                                                                 int64_t ld_sched, int64_t n_sched) {
  extern __shared__ int32_t s_mem[];             // [1024] segment sums, then [E + 1] sizes, [E + 1] scan input, [E + 1] offsets
  __shared__ int32_t s_warp[33];
  pdl_begin();
  int32_t* s_seg = s_mem;
  int32_t* s_size = s_mem + 1024;
  int32_t* s_nb = s_size + (E + 1);
  int32_t* s_offs = s_nb + (E + 1);
  // ---- 1. exclusive scan of partial[.][e] over the blocks of tokens, by S segments of blocks per expert -------------
  int Ep = 1;
  while (Ep < E) Ep <<= 1;
  const int S = 1024 / Ep;                        // threads (segments) per expert
  const int e = threadIdx.x % Ep, seg = threadIdx.x / Ep;
  const int64_t per = (n_blocks + S - 1) / S;
  const int64_t b_lo = min((int64_t)seg * per, n_blocks), b_hi = min(b_lo + per, n_blocks);
  int sum = 0;
  int first[16];                                  // the first 16 counts of this thread's segment stay in registers
#pragma unroll
  for (int u = 0; u < 16; ++u) first[u] = 0;
  if (e < E) {
#pragma unroll
    for (int u = 0; u < 16; ++u) first[u] = b_lo + u < b_hi ? partial_in[(b_lo + u) * E + e] : 0;
#pragma unroll
    for (int u = 0; u < 16; ++u) sum += first[u];
    for (int64_t b0 = b_lo + 16; b0 < b_hi; b0 += 8) {
      int v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = b0 + u < b_hi ? partial_in[(b0 + u) * E + e] : 0;
#pragma unroll
      for (int u = 0; u < 8; ++u) sum += v[u];
    }
  }
  s_seg[threadIdx.x] = sum;
  __syncthreads();
  int run = 0, total = 0;
  for (int s2 = 0; s2 < S; ++s2) {
    const int v = s_seg[s2 * Ep + e];
    if (s2 < seg) run += v;
    total += v;
  }
  // Six blocks share the work after the totals, which each of them forms for itself: block 0 turns the partial counts
  // into running offsets and writes col_sum, blocks 1..5 each build one row of the ragged metadata.  (One block doing
  // all of it was a chain of five scans with their barriers: 17 us for 16384 tokens.)
  const int role = blockIdx.x;
  if (e < E) {
    if (role == 0) {
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        if (b_lo + u < b_hi) partial_out[(b_lo + u) * E + e] = run;
        run += first[u];
      }
      for (int64_t b0 = b_lo + 16; b0 < b_hi; b0 += 8) {
        int v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = b0 + u < b_hi ? partial_in[(b0 + u) * E + e] : 0;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          if (b0 + u < b_hi) partial_out[(b0 + u) * E + e] = run;
          run += v[u];
        }
      }
      if (seg == 0) col_sum[e] = total;
    }
    if (seg == 0) s_size[e] = total;
  }
  if (threadIdx.x == 0) s_size[E] = 0;
  __syncthreads();
  if (role == 0) return;
  // ---- 2. expert offsets, then the ragged metadata: row 0 = slice_offs (= col_offs), rows 1..4 = block sizes 16..128 --
  ragged_row(role - 1, s_size, E, s_nb, s_offs, s_warp, slice_offs, col_offs, block_offs, ld_block_offs, block_sched, ld_sched,
             n_sched);
}

// Second and last launch of batches whose blocks are a wave: blocks 0 .. n_blocks - 1 add up the counts of the blocks before theirs and
// of all (64 KB for 16384 tokens and 128 experts, from L2) and rank their entries, five more build the ragged metadata.  With the sums in a
// launch between (route_scan_ragged_kernel) 2049 tokens of 128 experts, k = 4, take 14.5 us, so 11.3 (rule and figures where it is launched).
__global__ void __launch_bounds__(1024) route_finish_kernel(const int16_t* indx, int64_t ld_indx, int64_t T_rows, int E, int k, const int32_t* partial,
                                                            int n_blocks, int32_t* col_sum, int32_t* col_sorted, int32_t* row_sorted,
                                                            int32_t* slice_offs, int32_t* block_offs, int64_t ld_block_offs,
                                                            int32_t* block_sched, int64_t ld_sched, int64_t n_sched, const PerPosition out) {
  // [1024] segment sums, [1024] of them before this block, [E + 1] sizes, [E + 1] scan input, [E + 1] offsets, [E] entries before,
  // [warps in use][E] counters, [entries] experts (int16)
  extern __shared__ int32_t s_mem[];
  __shared__ int32_t s_warp[33];
  pdl_begin();
  int32_t* s_tot = s_mem;
  int32_t* s_bef = s_tot + 1024;
  int32_t* s_size = s_bef + 1024;
  int32_t* s_nb = s_size + (E + 1);
  int32_t* s_offs = s_nb + (E + 1);
  int32_t* s_before = s_offs + (E + 1);
  int32_t* s_cnt = s_before + E;
  const int own = (int)blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool ranks = own < n_blocks;
  const int64_t tok0 = (int64_t)own * kRouteTokPerBlock;
  const int n = ranks ? (int)min((int64_t)kRouteTokPerBlock, T_rows - tok0) * k : 0;
  const int rounds = (kRouteTokPerBlock * k + 1023) >> 10, per = rounds * 32, warps = (kRouteTokPerBlock * k + per - 1) / per;
  int16_t* s_pick = reinterpret_cast<int16_t*>(s_cnt + warps * E);
  // ---- counts of an expert, by S segments of blocks ----
  int Ep = 1;
  while (Ep < E) Ep <<= 1;
  const int S = 1024 / Ep, e = threadIdx.x % Ep, seg = threadIdx.x / Ep;
  const int seg_blocks = (n_blocks + S - 1) / S, lo = min(seg * seg_blocks, n_blocks), hi = min(lo + seg_blocks, n_blocks);
  int tot = 0, bef = 0;
  if (e < E)
    for (int b0 = lo; b0 < hi; b0 += 16) {
      int v[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) v[u] = b0 + u < hi ? partial[(int64_t)(b0 + u) * E + e] : 0;
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        tot += v[u];
        if (b0 + u < own) bef += v[u];
      }
    }
  s_tot[threadIdx.x] = tot;
  s_bef[threadIdx.x] = bef;
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    const int token = j / k;
    s_pick[j] = indx[(tok0 + token) * ld_indx + (j - token * k)];
  }
  for (int i = threadIdx.x; i < warps * E; i += blockDim.x) s_cnt[i] = 0;
  __syncthreads();
  if (seg == 0 && e < E) {
    int total = 0, before = 0;
    for (int i = 0; i < S; ++i) {
      total += s_tot[i * Ep + e];
      before += s_bef[i * Ep + e];
    }
    s_size[e] = total;
    s_before[e] = before;
  }
  if (threadIdx.x == 0) s_size[E] = 0;
  int32_t* my = s_cnt + warp * E;
  if (ranks && warp < warps)
    for (int r = 0; r < rounds; ++r) {
      const int j = warp * per + r * 32 + lane, c = j < n ? s_pick[j] : -1;
      const unsigned peers = __match_any_sync(0xFFFFFFFFu, c);
      if (c >= 0 && (peers & ((1u << lane) - 1u)) == 0) my[c] += __popc(peers);
      __syncwarp();
    }
  __syncthreads();
  if (!ranks) {
    if (own == n_blocks)
      for (int i = threadIdx.x; i < E; i += blockDim.x) col_sum[i] = s_size[i];
    ragged_row(own - n_blocks, s_size, E, s_nb, s_offs, s_warp, slice_offs, nullptr, block_offs, ld_block_offs, block_sched, ld_sched, n_sched);
    return;
  }
  // ---- stable expert-major positions: a warp ranks `per` entries in order, on top of the counts of the warps and blocks before it ----
  block_exclusive_scan(s_size, s_offs, E, s_warp);
  for (int i = threadIdx.x; i < E; i += blockDim.x) {
    int run = s_offs[i] + s_before[i];
    for (int w0 = 0; w0 < warps; w0 += 8) {
      int v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = w0 + u < warps ? s_cnt[(w0 + u) * E + i] : 0;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        if (w0 + u < warps) s_cnt[(w0 + u) * E + i] = run;
        run += v[u];
      }
    }
  }
  __syncthreads();
  if (warp < warps)
    for (int r = 0; r < rounds; ++r) {
      const int j = warp * per + r * 32 + lane, c = j < n ? s_pick[j] : -1;
      const unsigned peers = __match_any_sync(0xFFFFFFFFu, c);
      const int before = __popc(peers & ((1u << lane) - 1u));
      const int base = c >= 0 ? my[c] : 0;
      __syncwarp();
      if (c >= 0 && before == 0) my[c] = base + __popc(peers);
      __syncwarp();
      if (c >= 0) {
        const int pos = base + before;
        const int64_t flat = tok0 * k + j;
        row_sorted[flat] = pos;
        col_sorted[pos] = (int32_t)flat;
        if (out.token) {
          const int64_t token = tok0 + j / k;
          out.token[pos] = (int32_t)token;
          if (out.weight) out.weight[pos] = out.vals[token * out.ld_vals + j % k];
        }
      }
    }
}

// The whole routing step of a small batch (at most 256 tokens, at most 256 experts, k in {1, 2, 4, 8, 16}; see route_form) in ONE launch
// of five blocks of 1024 threads that do not wait on one another: every block selects the top-k of every row for itself
// (`parts` lanes per row: all that 1024 threads can give a row, up to a warp; 128 KB of logits at most) and counts the picks;
// block 0 stores the selection, the expert offsets (ragged row 0) and the positions of the entries, blocks 1..4 each build
// the block_offs row and the schedule of one block size.  Repeating the selection five times costs less than what it
// replaces: a chain of kernel boundaries (three launches) or of block barriers (one block doing all five rows took 20 us at
// 64 tokens).  What is left is a chain of latencies: with four lanes per row whatever their number and the picks read back
// from global memory by one warp per 32 tokens, 1 and 64 tokens of 128 experts took 11.6 and 12.7 us in a graph, so 4.3 and 8.3.
template <typename T, int K>
__global__ void __launch_bounds__(1024) route_small_kernel(
    const T* logits, int64_t ld_logits, int T_rows, int E, int parts, int apply_softmax, T* vals,
    int64_t ld_vals, int16_t* indx, int64_t ld_indx, uint32_t* bitmatrix, int64_t bm_stride_row,
    int64_t bm_stride_word, int32_t* col_sum, int32_t* col_sorted, int32_t* row_sorted,
    int32_t* slice_offs, int32_t* block_offs, int64_t ld_block_offs, int32_t* block_sched,
    int64_t ld_sched, int64_t n_sched, const PerPosition out) {
  // [E + 1] sizes, [E + 1] scan input, [E + 1] offsets, [n] values, [n] picks (int16), [warps in use][E] counters (uint16)
  extern __shared__ int32_t s_mem[];
  __shared__ int32_t s_warp[33];
  pdl_begin();
  const int n = T_rows * K;
  int32_t* s_size = s_mem;
  int32_t* s_nb = s_size + (E + 1);
  int32_t* s_offs = s_nb + (E + 1);
  float* s_val = reinterpret_cast<float*>(s_offs + (E + 1));
  int16_t* s_pick = reinterpret_cast<int16_t*>(s_val + n);
  uint16_t* s_cnt = reinterpret_cast<uint16_t*>(s_pick + n);
  const int role = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rounds = (n + 1023) >> 10, per = rounds * 32, warps = (n + per - 1) / per;      // entries of a warp, warps with entries
  for (int e = threadIdx.x; e <= E; e += blockDim.x) s_size[e] = 0;
  if (role == 0)
    for (int i = threadIdx.x; i < warps * E; i += blockDim.x) s_cnt[i] = 0;
  __syncthreads();
  {
    const int part = threadIdx.x & (parts - 1), row = threadIdx.x / parts;
    const bool live = row < T_rows;
    if (__any_sync(0xFFFFFFFFu, live)) {
      const T* x = logits + (live ? row : 0) * ld_logits;
      const TopK<K> tk = quad_select<T, K>(x, E, part, parts);
      if (live) {
        if (role == 0) {
          quad_store<T, K>(tk, part, row, E, apply_softmax, vals, ld_vals, indx, ld_indx, bitmatrix, bm_stride_row,
                           bm_stride_word, s_size, parts, s_pick + row * K, s_val + row * K);
        } else if (part == 0) {
#pragma unroll
          for (int i = 0; i < K; ++i) atomicAdd(&s_size[tk.idx[i]], 1);
        }
      }
    }
  }
  __syncthreads();                               // the picks are counted (block 0: and stored)
  if (role > 0) {
    ragged_row(role, s_size, E, s_nb, s_offs, s_warp, slice_offs, nullptr, block_offs, ld_block_offs, block_sched, ld_sched, n_sched);
    return;
  }
  for (int e = threadIdx.x; e < E; e += blockDim.x) col_sum[e] = s_size[e];
  // stable expert-major positions: a warp ranks `per` entries in order, on top of the counts of the warps before it
  uint16_t* my = s_cnt + warp * E;
  if (warp < warps)
    for (int r = 0; r < rounds; ++r) {
      const int j = warp * per + r * 32 + lane, c = j < n ? s_pick[j] : -1;
      const unsigned peers = __match_any_sync(0xFFFFFFFFu, c);
      if (c >= 0 && (peers & ((1u << lane) - 1u)) == 0) my[c] += (uint16_t)__popc(peers);
      __syncwarp();
    }
  ragged_row(0, s_size, E, s_nb, s_offs, s_warp, slice_offs, nullptr, block_offs, ld_block_offs, block_sched, ld_sched, n_sched);
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    int run = s_offs[e];
    for (int w0 = 0; w0 < warps; w0 += 8) {
      int v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = w0 + u < warps ? s_cnt[(w0 + u) * E + e] : 0;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        if (w0 + u < warps) s_cnt[(w0 + u) * E + e] = (uint16_t)run;
        run += v[u];
      }
    }
  }
  __syncthreads();
  if (warp >= warps) return;
  for (int r = 0; r < rounds; ++r) {
    const int j = warp * per + r * 32 + lane, c = j < n ? s_pick[j] : -1;
    const unsigned peers = __match_any_sync(0xFFFFFFFFu, c);
    const int before = __popc(peers & ((1u << lane) - 1u));
    const int base = c >= 0 ? my[c] : 0;
    __syncwarp();
    if (c >= 0 && before == 0) my[c] = (uint16_t)(base + __popc(peers));
    __syncwarp();
    if (c >= 0) {
      const int pos = base + before;
      row_sorted[j] = pos;
      col_sorted[pos] = j;
      if (out.token) {
        out.token[pos] = j / K;
        if (out.weight) out.weight[pos] = s_val[j];
      }
    }
  }
}

constexpr int kRouteSmallTokens = 256;

// The whole routing step of a batch of up to 896 to 2048 tokens (see route_form) in one launch of one cluster: eight blocks take an eighth of the tokens each, read
// one another's expert counts through distributed shared memory behind a cluster barrier, and rank their own entries on top of
// them; blocks 3 to 7 build a row of the ragged metadata each.

template <typename T, int K>
__global__ void __launch_bounds__(1024) route_cluster_kernel(
    const T* logits, int64_t ld_logits, int T_rows, int E, int parts, int apply_softmax, T* vals, int64_t ld_vals, int16_t* indx,
    int64_t ld_indx, uint32_t* bitmatrix, int64_t bm_stride_row, int64_t bm_stride_word, int32_t* col_sum, int32_t* col_sorted,
    int32_t* row_sorted, int32_t* slice_offs, int32_t* block_offs, int64_t ld_block_offs, int32_t* block_sched, int64_t ld_sched,
    int64_t n_sched, const PerPosition out) {
  // [E + 1] own counts, [E + 1] sizes, [E + 1] scan input, [E + 1] offsets, [E] entries of the blocks before, [n] values, [n] picks (int16),
  // [warps in use][E] counters (uint16)
  extern __shared__ int32_t s_mem[];
  __shared__ int32_t s_warp[33];
  pdl_begin();
  const int rank = (int)cluster_rank(), per_block = (T_rows + kRouteCluster - 1) / kRouteCluster, tok0 = rank * per_block;
  const int tokens = max(0, min(per_block, T_rows - tok0)), n = tokens * K, n_max = per_block * K;
  int32_t* s_own = s_mem;
  int32_t* s_size = s_own + (E + 1);
  int32_t* s_nb = s_size + (E + 1);
  int32_t* s_offs = s_nb + (E + 1);
  int32_t* s_before = s_offs + (E + 1);
  float* s_val = reinterpret_cast<float*>(s_before + E);
  int16_t* s_pick = reinterpret_cast<int16_t*>(s_val + n_max);
  uint16_t* s_cnt = reinterpret_cast<uint16_t*>(s_pick + n_max);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rounds = (n_max + 1023) >> 10, per = rounds * 32, warps = (n_max + per - 1) / per;      // entries of a warp, warps with entries
  for (int e = threadIdx.x; e <= E; e += blockDim.x) s_own[e] = 0;
  for (int i = threadIdx.x; i < warps * E; i += blockDim.x) s_cnt[i] = 0;
  __syncthreads();
  {
    const int part = threadIdx.x & (parts - 1), row = threadIdx.x / parts;
    const bool live = row < tokens;
    if (__any_sync(0xFFFFFFFFu, live)) {
      const TopK<K> tk = quad_select<T, K>(logits + (int64_t)(tok0 + (live ? row : 0)) * ld_logits, E, part, parts);
      if (live)
        quad_store<T, K>(tk, part, tok0 + row, E, apply_softmax, vals, ld_vals, indx, ld_indx, bitmatrix, bm_stride_row, bm_stride_word, s_own,
                         parts, s_pick + row * K, s_val + row * K);
    }
  }
  __syncthreads();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  // meanwhile the counts of the warps' shares
  uint16_t* my = s_cnt + warp * E;
  if (warp < warps)
    for (int r = 0; r < rounds; ++r) {
      const int j = warp * per + r * 32 + lane, c = j < n ? s_pick[j] : -1;
      const unsigned peers = __match_any_sync(0xFFFFFFFFu, c);
      if (c >= 0 && (peers & ((1u << lane) - 1u)) == 0) my[c] += (uint16_t)__popc(peers);
      __syncwarp();
    }
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    int v[kRouteCluster], before = 0, total = 0;
#pragma unroll
    for (int i = 0; i < kRouteCluster; ++i) v[i] = ld_cluster(s_own + e, (uint32_t)i);
#pragma unroll
    for (int i = 0; i < kRouteCluster; ++i) {
      if (i < rank) before += v[i];
      total += v[i];
    }
    s_size[e] = total;
    s_before[e] = before;
    if (rank == 0) col_sum[e] = total;
  }
  if (threadIdx.x == 0) s_size[E] = 0;
  __syncthreads();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");      // the others' counts have been read
  // stable expert-major positions: a warp ranks `per` entries in order, on top of the counts of the warps and blocks before it
  if (rank == kRouteCluster - 5)
    ragged_row(0, s_size, E, s_nb, s_offs, s_warp, slice_offs, nullptr, block_offs, ld_block_offs, block_sched, ld_sched, n_sched);
  else
    block_exclusive_scan(s_size, s_offs, E, s_warp);
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    int run = s_offs[e] + s_before[e];
    for (int w0 = 0; w0 < warps; w0 += 8) {
      int v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = w0 + u < warps ? s_cnt[(w0 + u) * E + e] : 0;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        if (w0 + u < warps) s_cnt[(w0 + u) * E + e] = (uint16_t)run;
        run += v[u];
      }
    }
  }
  __syncthreads();
  if (warp < warps)
    for (int r = 0; r < rounds; ++r) {
      const int j = warp * per + r * 32 + lane, c = j < n ? s_pick[j] : -1;
      const unsigned peers = __match_any_sync(0xFFFFFFFFu, c);
      const int before = __popc(peers & ((1u << lane) - 1u));
      const int base = c >= 0 ? my[c] : 0;
      __syncwarp();
      if (c >= 0 && before == 0) my[c] = (uint16_t)(base + __popc(peers));
      __syncwarp();
      if (c >= 0) {
        const int pos = base + before, flat = tok0 * K + j;
        row_sorted[flat] = pos;
        col_sorted[pos] = flat;
        if (out.token) {
          out.token[pos] = flat / K;
          if (out.weight) out.weight[pos] = s_val[j];
        }
      }
    }
  if (rank > kRouteCluster - 5)
    ragged_row(rank - (kRouteCluster - 5), s_size, E, s_nb, s_offs, s_warp, slice_offs, nullptr, block_offs, ld_block_offs, block_sched, ld_sched,
               n_sched);
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");        // no block leaves while its counts are read
}

}  // namespace

extern "C" __attribute__((visibility("default"))) size_t moe_route_workspace(int64_t T, int E, int k) {
  (void)k;
  const int64_t nb = cdiv64(T > 0 ? T : 1, kRouteTokPerBlock);
  return (size_t)((2 * nb * E + E) * (int64_t)sizeof(int32_t));
}

// us on the device, calls of a graph (small, cluster, two launches, three launches):
//   128 experts, k = 4:  16 tokens 5.6, 6.4;  32  7.7, 6.5;  64  8.1, 7.0;  256  13.6, 10.0, 10.4;  300  -, 8.5, 10.5, 13.6;  512  -, 10.5, 10.7, 13.6;
//                        768  -, 10.4, 11.2, 14.1;  1024  -, 12.2, 11.5, 14.2;  1536  -, 13.8, 11.3, 14.4;  2048  -, 16.7, 11.6, 14.4
//   64 experts, k = 8:   16 tokens 7.4, 7.0;  256  15.5, 13.9, 12.4;  300  -, 10.3, 12.4, 17.1;  768  -, 12.6, 12.9, 17.5;
//                        1024  -, 15.2, 12.9, 17.6;  1536  -, 15.4, 13.2, 17.9;  2048  -, 18.9, 13.5, 18.0
//   64 experts, k = 4:   32 tokens 7.7, 6.4;  96  6.8, 7.2;  256  10.6, 9.9, 8.8;  768  -, 9.1, 9.3;  1536  -, 11.4, 9.8, 13.1
//   32 experts, k = 4:   64 tokens 7.4, 6.8;  96  6.3, 7.2;  256  8.8, 9.8, 7.9;  300  -, 7.9, 8.0, 11.9;  1024  -, 9.7, 8.4;  2048  -, 11.3, 8.6, 12.8
//   8 experts, k = 2:    64 tokens 5.3, 6.0;  256  5.2, 7.6, 6.6;  300  -, 6.5, 6.7, 12.5;  2048  -, 7.4, 7.2, 12.9
//   256 experts, k = 16: 64 tokens 26.8, 11.7, 36.7;  768  -, 29.7, 39.9;  1536  -, 44.2, 40.5;  2048  -, 56.1, 41.5
// and (cluster, two launches) of short lists:
//   k = 1:  8 experts 900 tokens 6.8, 6.7;  1280  6.2, 7.0;  1536  6.3, 6.8;  64 experts 1024  7.2, 7.6;  1280  7.6, 7.6;  128 experts 1024  8.1, 9.1;
//           1280  9.0, 8.8;  256 experts 1024  9.8, 11.4;  1280  12.0, 11.5
//   k = 2:  8 experts 900 tokens 7.3, 7.1;  1280  6.6, 7.1;  1536  6.8, 7.1;  32 experts 900  7.6, 7.2;  128 experts 1024  9.4, 9.8;  1280  10.0, 9.4;
//           256 experts 1024  11.7, 12.2;  1280  13.0, 12.3
// The small form repeats the whole selection in five blocks, the cluster has an eighth of it in each of eight and two barriers; past 768 to 1024
// tokens eight SMs are fewer than the selection wants, and two launches are ahead.  With long lists (E k > 1024) the finish of those takes
// longest and the line lies at 1536.  Lists of one or two picks leave the cluster little to sort: from 64 experts on its line lies at 1024, and the shortest
// (E k <= 16) go back to it where it has four lanes per token, from 1025 to 1536.  (From 129 to 256 tokens the rule does not follow the table: two launches
// would be up to 1.8 us ahead with four picks and more, and the cluster's 32 lanes per token take longer there than 16 do at 300.)
// These are the lines of a layer step, whose products keep the device ahead of the host.  A call by itself takes 12 us of the host with one launch and 14 with two,
// more than the device has to do up to E k = 512, so there the cluster's lines are at 1536 and 2048 (us per call in a loop, cluster and two launches: 1024
// tokens of 128 experts, k = 4, 12.4, 14.1; 1536 14.1, 13.9; 1536 of 32 experts, k = 8, 13.4, 14.0; 2048 of 32 experts, k = 4, 12.1, 14.1; but 900 of 64
// experts, k = 8, 14.9, 13.9; of 200, k = 4, 14.8, 14.0).
enum { ROUTE_SMALL, ROUTE_CLUSTER, ROUTE_LAUNCHES };
static int route_form(int64_t T, int E, int k, bool step) {
  if (!(k == 1 || k == 2 || k == 4 || k == 8 || k == 16)) return ROUTE_LAUNCHES;
  if (T <= kRouteSmallTokens) return T >= 24 && k >= 4 && (E * k >= 512 || T <= 64) ? ROUTE_CLUSTER : ROUTE_SMALL;
  if (!step && k <= 8 && E * k <= (k <= 4 ? 512 : 256)) return T <= (E * k <= 128 ? 2048 : 1536) ? ROUTE_CLUSTER : ROUTE_LAUNCHES;
  if (E * k <= 16 && T > 1024) return T <= 1536 ? ROUTE_CLUSTER : ROUTE_LAUNCHES;
  return T <= (E * k > 1024 ? 1536 : k <= 2 && E >= 64 ? 1024 : 896) ? ROUTE_CLUSTER : ROUTE_LAUNCHES;
}

static int route_launch(
    const void* logits, int dtype, int64_t T, int E, int k, int apply_softmax, int64_t ld_logits, void* vals, int64_t ld_vals,
    int16_t* indx, int64_t ld_indx, uint32_t* bitmatrix, int64_t bm_stride_row, int64_t bm_stride_word, int32_t* col_sum,
    int32_t* col_sorted, int32_t* row_sorted, int32_t* slice_offs, int32_t* block_offs, int64_t ld_block_offs,
    int32_t* block_sched, int64_t ld_sched, int64_t n_sched, void* workspace, size_t workspace_bytes, const PerPosition& out,
    void* stream) {
  MOE_CHECK_ARG(T > 0 && E > 0 && k > 0 && k <= kMaxTopK && k <= E, "moe_route: bad extents T=%lld E=%d k=%d", (long long)T, E, k);
  if (E > 256) {
    moe_set_error("moe_route: the fused routing handles up to 256 experts (got %d); use the separate entry points", E);
    return MOE_ERR_UNSUPPORTED;
  }
  MOE_CHECK_ARG(logits && vals && indx && bitmatrix && col_sum && col_sorted && row_sorted && slice_offs && block_offs &&
                    (block_sched || n_sched == 0) && workspace,
                "moe_route: NULL pointer");
  MOE_CHECK_ARG(ld_block_offs >= E + 1 && ld_sched >= n_sched, "moe_route: leading dimensions too small");
  MOE_CHECK_ARG(workspace_bytes >= moe_route_workspace(T, E, k), "moe_route: workspace too small (%zu < %zu)", workspace_bytes,
                moe_route_workspace(T, E, k));
  cudaStream_t st = (cudaStream_t)stream;
  const int form = route_form(T, E, k, out.weight != nullptr);
  if (form == ROUTE_SMALL) {
    const int n = (int)T * k, warps = (n + 31) / 32 < 32 ? (n + 31) / 32 : 32;
    const size_t smem_s = (size_t)(3 * (E + 1) + n) * sizeof(int32_t) + (size_t)(n + warps * E) * sizeof(int16_t);   // < 48 KB
    const int parts = T <= 32 ? 32 : T <= 64 ? 16 : T <= 128 ? 8 : 4;
#define MOE_ROUTE_SMALL(KK)                                                                                              \
  MOE_DISPATCH_FLOAT(dtype, Tv, {                                                                                         \
    MOE_CHECK_CUDA(launch_pdl(route_small_kernel<Tv, KK>, dim3(5), dim3(1024), smem_s, st, (const Tv*)logits, ld_logits,    \
                              (int)T, E, parts, apply_softmax, (Tv*)vals, ld_vals, indx, ld_indx, bitmatrix, bm_stride_row, \
                              bm_stride_word, col_sum, col_sorted, row_sorted, slice_offs, block_offs, ld_block_offs,       \
                              block_sched, ld_sched, n_sched, out));                                                        \
  })
    switch (k) {
      case 1: MOE_ROUTE_SMALL(1); break;
      case 2: MOE_ROUTE_SMALL(2); break;
      case 4: MOE_ROUTE_SMALL(4); break;
      case 8: MOE_ROUTE_SMALL(8); break;
      default: MOE_ROUTE_SMALL(16); break;
    }
#undef MOE_ROUTE_SMALL
    MOE_CHECK_LAUNCH();
    return MOE_OK;
  }
  if (form == ROUTE_CLUSTER) {
    const int per_block = ((int)T + kRouteCluster - 1) / kRouteCluster, n = per_block * k, warps = (n + 31) / 32 < 32 ? (n + 31) / 32 : 32;
    const size_t smem_c = (size_t)(5 * E + 4 + n) * sizeof(int32_t) + (size_t)(n + warps * E) * sizeof(int16_t);      // < 48 KB
    const int parts = per_block <= 32 ? 32 : per_block <= 64 ? 16 : per_block <= 128 ? 8 : 4;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kRouteCluster);
    cfg.blockDim = dim3(1024);
    cfg.dynamicSmemBytes = smem_c;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = kRouteCluster; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
#define MOE_ROUTE_CLUSTER(KK)                                                                                            \
  MOE_DISPATCH_FLOAT(dtype, Tv, {                                                                                         \
    MOE_CHECK_CUDA(cudaLaunchKernelEx(&cfg, route_cluster_kernel<Tv, KK>, (const Tv*)logits, ld_logits, (int)T, E, parts,    \
                                      apply_softmax, (Tv*)vals, ld_vals, indx, ld_indx, bitmatrix, bm_stride_row,            \
                                      bm_stride_word, col_sum, col_sorted, row_sorted, slice_offs, block_offs,               \
                                      ld_block_offs, block_sched, ld_sched, n_sched, out));                                  \
  })
    switch (k) {
      case 1: MOE_ROUTE_CLUSTER(1); break;
      case 2: MOE_ROUTE_CLUSTER(2); break;
      case 4: MOE_ROUTE_CLUSTER(4); break;
      case 8: MOE_ROUTE_CLUSTER(8); break;
      default: MOE_ROUTE_CLUSTER(16); break;
    }
#undef MOE_ROUTE_CLUSTER
    MOE_CHECK_LAUNCH();
    return MOE_OK;
  }
  const int64_t nb = cdiv64(T, kRouteTokPerBlock);
  int32_t* partial = (int32_t*)workspace;          // counts per block of tokens, their running offsets, expert offsets
  int32_t* scanned = partial + nb * E;
  int32_t* col_offs = scanned + nb * E;
#define MOE_ROUTE_QUAD(KK)                                                                                               \
  MOE_DISPATCH_FLOAT(dtype, Tv, {                                                                                         \
    MOE_CHECK_CUDA(launch_pdl(topk_quad_kernel<Tv, KK, true>, dim3((unsigned)nb), dim3(4 * kRouteTokPerBlock),              \
                              (size_t)E * sizeof(int32_t), st, (const Tv*)logits, ld_logits, T, E, apply_softmax,           \
                              (Tv*)vals, ld_vals, indx, ld_indx, bitmatrix, bm_stride_row, bm_stride_word, partial));       \
  })
  switch (k) {
    case 1: MOE_ROUTE_QUAD(1); break;
    case 2: MOE_ROUTE_QUAD(2); break;
    case 4: MOE_ROUTE_QUAD(4); break;
    case 8: MOE_ROUTE_QUAD(8); break;
    case 16: MOE_ROUTE_QUAD(16); break;
    default:
      MOE_DISPATCH_FLOAT(dtype, Tv, {
        MOE_CHECK_CUDA(launch_pdl(route_topk_hist_kernel<Tv>, dim3((unsigned)nb), dim3(kRouteWarps * 32), (size_t)E * sizeof(int32_t),
                                  st, (const Tv*)logits, ld_logits, T, E, k, apply_softmax, (Tv*)vals, ld_vals, indx, ld_indx,
                                  bitmatrix, bm_stride_row, bm_stride_word, partial));
      });
  }
#undef MOE_ROUTE_QUAD
  MOE_CHECK_LAUNCH();
  const int entries = kRouteTokPerBlock * k, warps = entries / 32 < 32 ? entries / 32 : 32;
  const size_t smem_f = (size_t)(2048 + 3 * (E + 1) + E + warps * E) * sizeof(int32_t) + (size_t)entries * sizeof(int16_t);
  // Two launches while the blocks are a wave, and with long lists while there are at most 64 of 128 tokens (and the five of the ragged
  // metadata): every one of them reads the counts of all.  us with two and three launches: 128 experts, k = 4: 8192 tokens 11.9, 16.1;
  // 16384 16.7, 17.7; 18304 18.1, 18.6; 24576 26.9, 23.5.  k = 8: 16384 25.0, 26.1; 24576 38.2, 36.5.  200 experts, k = 6: 8192 32.6, 38.4;
  // 12288 51.4, 40.4.  256 experts, k = 8: 8192 22.1, 29.3; 12288 35.6, 31.6.  The line goes by E k: 256 experts, k = 4 are on the
  // long side of it by their counts (8192 15.2, 19.7; 12288 23.4, 21.4; 16384 24.3, 23.1), 128 experts, k = 16 on the short one
  // (16384 41.2, 44.1).
  if (nb + 5 <= (E * k <= 1024 ? moe_sm_count() : 64 + 5) && smem_f <= 48 * 1024) {
    MOE_CHECK_CUDA(launch_pdl(route_finish_kernel, dim3((unsigned)nb + 5), dim3(1024), smem_f, st, indx, ld_indx, T, E, k, partial, (int)nb, col_sum,
                              col_sorted, row_sorted, slice_offs, block_offs, ld_block_offs, block_sched, ld_sched, n_sched, out));
    MOE_CHECK_LAUNCH();
    return MOE_OK;
  }
  const size_t smem_b = (size_t)(1024 + 3 * (E + 1)) * sizeof(int32_t);
  MOE_CHECK_CUDA(launch_pdl(route_scan_ragged_kernel, dim3(6), dim3(1024), smem_b, st, partial, scanned, nb, E, col_sum, col_offs,
                            slice_offs, block_offs, ld_block_offs, block_sched, ld_sched, n_sched));
  MOE_CHECK_LAUNCH();
  const size_t smem_rank = (size_t)(kRouteTokPerBlock / 32) * E * sizeof(int32_t);
  MOE_CHECK_CUDA(launch_pdl(bm_rank_kernel, dim3((unsigned)nb), dim3(kRouteTokPerBlock), smem_rank, st, indx, ld_indx, T, E, k, nullptr,
                            scanned, col_offs, col_sorted, row_sorted, out));
  MOE_CHECK_LAUNCH();
  return MOE_OK;
}

extern "C" __attribute__((visibility("default"))) int moe_route(
    const void* logits, int dtype, int64_t T, int E, int k, int apply_softmax, int64_t ld_logits, void* vals, int64_t ld_vals,
    int16_t* indx, int64_t ld_indx, uint32_t* bitmatrix, int64_t bm_stride_row, int64_t bm_stride_word, int32_t* col_sum,
    int32_t* col_sorted, int32_t* row_sorted, int32_t* slice_offs, int32_t* block_offs, int64_t ld_block_offs,
    int32_t* block_sched, int64_t ld_sched, int64_t n_sched, void* workspace, size_t workspace_bytes, void* stream) {
  return route_launch(logits, dtype, T, E, k, apply_softmax, ld_logits, vals, ld_vals, indx, ld_indx, bitmatrix, bm_stride_row,
                      bm_stride_word, col_sum, col_sorted, row_sorted, slice_offs, block_offs, ld_block_offs, block_sched, ld_sched,
                      n_sched, workspace, workspace_bytes, PerPosition(), stream);
}

extern "C" __attribute__((visibility("default"))) int moe_route_positions(
    const float* logits, int64_t T, int E, int k, int apply_softmax, int64_t ld_logits, float* vals, int64_t ld_vals,
    int16_t* indx, int64_t ld_indx, uint32_t* bitmatrix, int64_t bm_stride_row, int64_t bm_stride_word, int32_t* col_sum,
    int32_t* col_sorted, int32_t* row_sorted, int32_t* slice_offs, int32_t* block_offs, int64_t ld_block_offs,
    int32_t* block_sched, int64_t ld_sched, int64_t n_sched, int32_t* token_of_position, float* weight_of_position, void* workspace,
    size_t workspace_bytes, void* stream) {
  MOE_CHECK_ARG(token_of_position, "moe_route_positions: NULL pointer");
  PerPosition out;
  out.token = token_of_position; out.weight = weight_of_position; out.vals = vals; out.ld_vals = ld_vals;
  return route_launch(logits, MOE_F32, T, E, k, apply_softmax, ld_logits, vals, ld_vals, indx, ld_indx, bitmatrix, bm_stride_row,
                      bm_stride_word, col_sum, col_sorted, row_sorted, slice_offs, block_offs, ld_block_offs, block_sched, ld_sched,
                      n_sched, workspace, workspace_bytes, out, stream);
}

// ---------------------------------------------------------------------------------------------------------
// moe_bitmatrix_metadata_noalloc: the same histogram + expert-major sort for hosts that cannot give this
// library a scratch buffer because they cannot allocate one at that point -- a serving process that handed
// all device memory to its own pools at start-up, or a latency-critical section in which cudaMalloc (which
// synchronises the device) is not acceptable.  The three sort passes need nb * E + E ints of scratch
// (nb = ceil(T / 256)); here that scratch is a fixed array inside the library image (up to 32768 entries of 256 experts the sort is
// one launch and does not touch it).
//
// Cost: every GPU that loads libmoe_b200.so carries kNoAllocScratchBytes (1 MiB) of device memory until the
// process exits, whether or not this entry point is ever called.
static __device__ __align__(256) int32_t g_bm_scratch[(1 << 20) / sizeof(int32_t)];
constexpr size_t kNoAllocScratchBytes = sizeof(int32_t) * ((1 << 20) / sizeof(int32_t));

// Device address of g_bm_scratch, looked up once per device.  In host code the name g_bm_scratch is only a
// handle for the runtime; the address a kernel can use comes from cudaGetSymbolAddress with that device current.
static void* g_bm_scratch_addr[64] = {nullptr};

extern "C" __attribute__((visibility("default"))) size_t moe_bitmatrix_metadata_noalloc_capacity(void) {
  return kNoAllocScratchBytes;
}

extern "C" __attribute__((visibility("default"))) int moe_bitmatrix_metadata_noalloc(
    const int16_t* indx, int64_t ld_indx, int64_t T, int E, int k, const int32_t* n_rows_dev, int32_t* col_sum,
    int32_t* col_sorted, int32_t* row_sorted, void* stream) {
  MOE_CHECK_ARG(T >= 0 && E > 0 && k > 0, "moe_bitmatrix_metadata_noalloc: bad extents T=%lld E=%d k=%d", (long long)T, E, k);
  const size_t need = moe_bitmatrix_metadata_workspace(T, E, k);
  MOE_CHECK_ARG(need <= kNoAllocScratchBytes,
                "moe_bitmatrix_metadata_noalloc: T=%lld tokens x E=%d experts needs %zu bytes of scratch, the built-in "
                "scratch holds %zu (ceil(T/256) * E + E ints must fit); use moe_bitmatrix_metadata with a caller buffer",
                (long long)T, E, need, kNoAllocScratchBytes);
  int dev = -1;
  MOE_CHECK_CUDA(cudaGetDevice(&dev));
  MOE_CHECK_ARG(dev >= 0 && dev < 64, "moe_bitmatrix_metadata_noalloc: device index %d out of range", dev);
  if (g_bm_scratch_addr[dev] == nullptr) {
    // first call on this device: resolve the symbol (not an allocation; the array is part of the module image)
    void* p = nullptr;
    MOE_CHECK_CUDA(cudaGetSymbolAddress(&p, g_bm_scratch));
    MOE_CHECK_ARG(p != nullptr, "moe_bitmatrix_metadata_noalloc: cudaGetSymbolAddress returned NULL");
    g_bm_scratch_addr[dev] = p;
  }
  // Nothing in the scratch has to start at zero: pass 1 writes every partial[block][expert] and pass 2 every
  // col_offs[expert] before they are read.
  return moe_bitmatrix_metadata(indx, ld_indx, T, E, k, n_rows_dev, col_sum, col_sorted, row_sorted,
                                g_bm_scratch_addr[dev], kNoAllocScratchBytes, stream);
}
