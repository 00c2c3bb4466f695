// Router: logits = x @ Wg + bg on the tensor cores with the top-k selection (+ softmax over the selected logits) and
// the expert bitmatrix in the epilogue -- the logits never travel through HBM and a routing step loses a launch.
//
// The reference runs the two steps apart: `logits = matmul(x, wg, bg)` then `topk(logits, k)`
// (triton_kernels bench/bench_mlp.py:70, topk.py:25-141); the selection rule, the softmax and the bitmatrix layout
// are those of topk_details/_topk_forward.py:91-150 (largest value first, equal values to the smaller expert index).
//
// One CTA per (block of 128 tokens, share of K).  Warp 0 streams x and Wg^T tiles (128 x 64 bf16 and E x 64 bf16, TMA,
// 128-byte swizzle) through a ring of stages, warp 1 issues tcgen05.mma.kind::f16 (M = 128 tokens, N = E experts) into
// one fp32 accumulator in tensor memory, warps 2-17 select: they spill the accumulator to shared memory and several
// threads per token row add the bias and keep the k best in registers.  With few tokens K is cut into slices so that many SMs pull the
// operands: the slices of a token block are spread over a cluster, every CTA leaves the sum of its slices in its own shared memory, and
// behind a cluster barrier each sums a share of the rows over all of them (distributed shared memory; everything in the order of the
// slices) and selects for it.  With the sort behind it, K = 2880, 128 experts, in a graph: 1 token 15.1 us, 64 17.0, 1024 25.0, 4100 30.1,
// 16384 39.5; as partial sums in an fp32 scratch by red.global.add, with the selection in the CTA that came last: 19.9, 23.9, 33.7, 35.7, 42.5.
// What bounds it: an SM takes in 32 B a cycle, 32 KB a k step.
// Every mbarrier wait is bounded.
#include "gemm_tc_common.cuh"
#include "topk_select.cuh"

namespace {

constexpr int RT_THREADS = 576;        // warp 0 producer, 1 MMA, 2-17 selection
constexpr int RT_MAT_LD = 136;         // row pitch of the logits matrix in shared memory: 8 (mod 32) keeps the P x rows of a warp on distinct banks
constexpr int RT_STAGES_MAX = 6;
constexpr int RT_BLOCK_T = 128;

struct RouterParams {
  int64_t T;
  int E, n_mma, k, KT;            // experts, E rounded up to 16, picks per token, 64-k steps
  int slices, splits, stages;     // of K, CTAs they are spread over
  int apply_softmax;
  int round_bf16;                 // logits rounded to bf16 before the selection (a bf16 router output, as the two-launch form has it)
  const void* bias; int bias_dtype;
  float* logits_out; int64_t ld_logits;
  void* vals; int vals_dtype; int64_t ld_vals;
  int16_t* indx; int64_t ld_indx;
  uint32_t* bitmatrix; int64_t bm_stride_row, bm_stride_word;
  int32_t* status;
};

template <int K>
__device__ __forceinline__ void rt_store_row(const RouterParams& p, int64_t row, const TopK<K>& tk) {
  float v[K];
  int e[K];
#pragma unroll
  for (int i = 0; i < K; ++i) {
    v[i] = sel_key_float(tk.key[i]);
    e[i] = tk.idx[i];
  }
  if (p.apply_softmax) {
    const float mx = v[0];
    float sum = 0.0f;
#pragma unroll
    for (int i = 0; i < K; ++i) sum += expf(v[i] - mx);
#pragma unroll
    for (int i = 0; i < K; ++i) v[i] = __fdiv_rn(expf(v[i] - mx), sum);
  }
#pragma unroll
  for (int i = 0; i < K; ++i) {
    if (p.vals_dtype == MOE_F32) ((float*)p.vals)[row * p.ld_vals + i] = v[i];
    else ((__nv_bfloat16*)p.vals)[row * p.ld_vals + i] = __float2bfloat16(v[i]);
    p.indx[row * p.ld_indx + i] = (int16_t)e[i];
  }
  const int words = (p.E + 31) >> 5;
  for (int w = 0; w < words; ++w) {
    uint32_t bits = 0;
#pragma unroll
    for (int i = 0; i < K; ++i)
      if ((e[i] >> 5) == w) bits |= 1u << (e[i] & 31);
    p.bitmatrix[row * p.bm_stride_row + (int64_t)w * p.bm_stride_word] = bits;
  }
}

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// a word at the same place of shared memory in slice `rank` of the cluster
__device__ __forceinline__ uint32_t ld_slice_u32(uint32_t at, int splits, int rank) {
  uint32_t v;
  if (splits == 1) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(at) : "memory");
  else asm volatile("{\n\t.reg .b32 ra;\n\tmapa.shared::cluster.u32 ra, %1, %2;\n\tld.shared::cluster.u32 %0, [ra];\n\t}" : "=r"(v) : "r"(at), "r"(rank) : "memory");
  return v;
}

template <int K>
__global__ void __launch_bounds__(RT_THREADS, 1)
router_topk_kernel(const RouterParams p, const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap w_map) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sbase = smem_u32(smem);
  float* mat = reinterpret_cast<float*>(smem);
  __shared__ __align__(8) uint64_t bars[2 * RT_STAGES_MAX + 4];
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort;
  __shared__ float s_bias[256];
  const int warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;     // warp-uniform for the compiler
  const int STAGES = p.stages;
  const uint32_t X_BYTES = RT_BLOCK_T * 128u, W_BYTES = (uint32_t)p.n_mma * 128u;
  const uint32_t stage_bytes = X_BYTES + ((W_BYTES + 1023u) & ~1023u);
  auto BAR_FULL = [&](int s) { return smem_u32(&bars[s]); };
  auto BAR_EMPTY = [&](int s) { return smem_u32(&bars[RT_STAGES_MAX + s]); };
  auto BAR_ACC = [&](int a) { return smem_u32(&bars[2 * RT_STAGES_MAX + a]); };              // a slice's sums are complete
  auto BAR_ACC_FREE = [&](int a) { return smem_u32(&bars[2 * RT_STAGES_MAX + 2 + a]); };     // and have been read
  Ctl ctl{&s_abort, p.status};
  const uint32_t acc_cols = p.n_mma <= 32 ? 32u : p.n_mma <= 64 ? 64u : p.n_mma <= 128 ? 128u : 256u;
  const uint32_t tmem_cols = p.slices > p.splits ? 2u * acc_cols : acc_cols;

  if (threadIdx.x == 0) {
    for (int s = 0; s < RT_STAGES_MAX; ++s) {
      mbar_init(BAR_FULL(s), 1);
      mbar_init(BAR_EMPTY(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(BAR_ACC(a), 1);
      mbar_init(BAR_ACC_FREE(a), 16);
    }
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x == 32) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&x_map) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&w_map) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, s_tmem, 0);
  pdl_begin();

  const int64_t blk = blockIdx.x;
  const int split = blockIdx.y;                 // rank in the cluster of a token block's slices
  const int sl0 = p.slices * split / p.splits, n_slices = p.slices * (split + 1) / p.splits - sl0;
  auto slice_k = [&](int i) { return (int)((int64_t)p.KT * (sl0 + i) / p.slices); };      // first k step of this CTA's slice i

  if (warp == 0) {
    bool ok = true;
    int it = 0;
    for (int i = 0; i < n_slices && ok; ++i) {
      const int kt0 = slice_k(i), n_steps = slice_k(i + 1) - kt0;
      for (int j = 0; j < n_steps; ++j, ++it) {
        const int s = it % STAGES;
        ok = __all_sync(0xFFFFFFFFu, mbar_wait(BAR_EMPTY(s), ((it / STAGES) & 1u) ^ 1u, ctl, 801));
        if (!ok) break;
        const uint32_t st = sbase + (uint32_t)s * stage_bytes;
        elect_expect_tx(BAR_FULL(s), X_BYTES + W_BYTES);
        // token blocks start at different k steps: CTAs that run side by side do not all ask for the same Wg tile
        const int kt = kt0 + (int)((j + blk * 5) % n_steps);
        elect_tile_2d(st, &x_map, kt * 64, (int)(blk * RT_BLOCK_T), BAR_FULL(s));
        elect_tile_2d(st + X_BYTES, &w_map, kt * 64, 0, BAR_FULL(s));
      }
    }
    if (!ok && lane == 0) {
      const int lo = it > STAGES ? it - STAGES : 0;
      for (int j = lo; j < it; ++j)
        for (uint32_t i = 0; i < (1u << 16) && !mbar_test(BAR_FULL(j % STAGES), (j / STAGES) & 1u); ++i) __nanosleep(64);
    }
    __syncwarp();
  } else if (warp == 1) {
    bool ok = true;
    const uint32_t idesc = make_idesc(p.n_mma);
    int it = 0;
    for (int i = 0; i < n_slices && ok; ++i) {
      const int n_steps = slice_k(i + 1) - slice_k(i);
      const uint32_t acc = tmem + (uint32_t)(i & 1) * acc_cols;
      if (i >= 2) {
        ok = __all_sync(0xFFFFFFFFu, mbar_wait(BAR_ACC_FREE(i & 1), ((i >> 1) & 1u) ^ 1u, ctl, 803));
        tc_fence_after();
      }
      for (int j = 0; j < n_steps && ok; ++j, ++it) {
        const int s = it % STAGES;
        ok = __all_sync(0xFFFFFFFFu, mbar_wait(BAR_FULL(s), (it / STAGES) & 1u, ctl, 802));
        if (!ok) break;
        tc_fence_after();
        const uint32_t st = sbase + (uint32_t)s * stage_bytes;
        const uint32_t a_lo = DESC_LO | (st >> 4), b_lo = DESC_LO | ((st + X_BYTES) >> 4);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) elect_mma_bf16(acc, a_lo + kk * 2, b_lo + kk * 2, idesc, (j | kk) ? 1u : 0u);
        elect_commit(BAR_EMPTY(s));
      }
      elect_commit(BAR_ACC(i & 1));     // arrives when every MMA above has retired
      if (!ok)                          // aborting: let the MMAs that were already issued retire before tensor memory is freed
        for (uint32_t w = 0; w < (1u << 16) && !mbar_test(BAR_ACC(i & 1), (i >> 1) & 1u); ++w) __nanosleep(64);
    }
    __syncwarp();
  } else {
    // ---- 16 warps: the sums of this CTA's slices, in their order, into shared memory as [expert][token row] (the operand stages are free
    // by then) ----
    const int qd = warp & 3, grp = (warp - 2) >> 2;            // lane quarter of tensor memory, share of its columns
    const int sid = threadIdx.x - 64;
    // the bias once per CTA, while the main loop runs (read per logit from global memory it made the selection wait on
    // one load after the other)
    if (sid < 256) s_bias[sid] = (p.bias && sid < p.E) ? load_bias(p.bias, p.bias_dtype, sid) : 0.0f;
    float sum[4][16];
    bool ok = true;
    for (int i = 0; i < n_slices && ok; ++i) {
      ok = __all_sync(0xFFFFFFFFu, mbar_wait(BAR_ACC(i & 1), (i >> 1) & 1u, ctl, 804));
      if (!ok) break;
      tc_fence_after();
      const uint32_t taddr = tmem + (uint32_t)(i & 1) * acc_cols + ((uint32_t)(qd * 32) << 16);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int c0 = grp * 16 + c * 64;
        if (c0 < p.n_mma) {
          uint32_t v[16];
          tmem_ld16(taddr + (uint32_t)c0, v);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) sum[c][j] = i ? sum[c][j] + __uint_as_float(v[j]) : __uint_as_float(v[j]);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(BAR_ACC_FREE(i & 1));
    }
    if (ok) {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int c0 = grp * 16 + c * 64;
        if (c0 < p.n_mma) {
#pragma unroll
          for (int j = 0; j < 16; ++j) mat[(c0 + j) * RT_MAT_LD + qd * 32 + lane] = sum[c][j];
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (p.splits > 1) cluster_barrier();
  if (warp >= 2) {
    // ---- selection: P threads per token row (adjacent lanes), each walks every P-th expert with its own best-k list, the lists of a row
    // meet by shuffles.  A single thread per row spent 12 us of dependent compare-and-select chains on 128 experts. ----
    const int sid = threadIdx.x - 64;
    const int rows_blk = (int)min((int64_t)RT_BLOCK_T, p.T - blk * RT_BLOCK_T);
    int lr = 0;
    while ((1 << lr) < rows_blk) ++lr;
    lr = max(0, lr - (31 - __clz(p.splits)));                  // this CTA's share of the rows: 2^lr from r0 on (none for some CTAs)
    const int r0 = split << lr, rows = min(1 << lr, rows_blk - r0);
    bool ok = true;
    for (int i = 0; i < p.splits; ++i) ok = ok && ld_slice_u32(smem_u32((const void*)&s_abort), p.splits, i) == 0;
    if (ok && rows > 0) {
      if (p.splits > 1) {
        const int total = p.n_mma << lr;
        for (int i0 = sid; i0 < total; i0 += 512 * 4) {
          float sum[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int i = i0 + u * 512;
            sum[u] = 0.0f;
            if (i < total) {
              const uint32_t at = smem_u32(mat + (i >> lr) * RT_MAT_LD + r0 + (i & ((1 << lr) - 1)));
#pragma unroll 1
              for (int j = 0; j < p.splits; j += 2) {
                const float x = __uint_as_float(ld_slice_u32(at, p.splits, j));
                const float y = j + 1 < p.splits ? __uint_as_float(ld_slice_u32(at, p.splits, j + 1)) : 0.0f;
                sum[u] += x;
                if (j + 1 < p.splits) sum[u] += y;
              }
            }
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) {                        // (only this CTA reads these rows of its own matrix)
            const int i = i0 + u * 512;
            if (i < total) mat[(i >> lr) * RT_MAT_LD + r0 + (i & ((1 << lr) - 1))] = sum[u];
          }
        }
        asm volatile("bar.sync 1, 512;" ::: "memory");
      }
      // P threads per row: 4 for a full block, 8 for at most 64 rows (more threads per row would spend in merge rounds what they save on
      // the walk)
      const int lp = rows <= 64 ? 3 : 2;
      const int P = 1 << lp;
      const int part = sid & (P - 1);
      const int rr = sid >> lp;
      if (__any_sync(0xFFFFFFFFu, rr < rows)) {
        const int64_t row = blk * RT_BLOCK_T + r0 + rr;
        const bool live = rr < rows;
        constexpr int NSUB = K <= 4 ? 2 : 1;
        TopK<K> sub[NSUB];
        const int rq = (r0 + rr) & (RT_BLOCK_T - 1);
#pragma unroll 1
        for (int e0 = part; e0 < p.E; e0 += P * NSUB * 4) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
#pragma unroll
            for (int u = 0; u < NSUB; ++u) {        // the lists alternate: independent chains side by side
              const int e = e0 + (j * NSUB + u) * P;
              if (e < p.E) {
                float x = mat[e * RT_MAT_LD + rq] + s_bias[e];
                if (p.round_bf16) x = __bfloat162float(__float2bfloat16(x));
                if (p.logits_out && live) p.logits_out[row * p.ld_logits + e] = x;
                sub[u].push(x, e);
              }
            }
          }
        }
        TopK<K> tk = sub[0];
#pragma unroll
        for (int u = 1; u < NSUB; ++u) tk.merge(sub[u].key, sub[u].idx);
        tk.merge_lanes(P);
        if (live && part == 0) rt_store_row<K>(p, row, tk);
      }
    }
    __syncwarp();
  }
  if (p.splits > 1) cluster_barrier();                  // no CTA leaves while its logits are read

  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols) : "memory");
  }
}

int rt_make_map(const void* base, int64_t rows, int64_t K, int64_t ld, int box_rows, CUtensorMap* map) {
  static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
  static std::mutex mu;
  {
    std::lock_guard<std::mutex> lk(mu);
    if (!encode) {
      void* fn = nullptr;
      cudaDriverEntryPointQueryResult qr;
      MOE_CHECK_CUDA(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &qr));
      if (qr != cudaDriverEntryPointSuccess || !fn) {
        moe_set_error("moe_router_topk: the driver does not provide cuTensorMapEncodeTiled");
        return MOE_ERR_UNSUPPORTED;
      }
      encode = (PFN_cuTensorMapEncodeTiled_v12000)fn;
    }
  }
  const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    moe_set_error("moe_router_topk: cuTensorMapEncodeTiled failed with code %d (rows %lld, K %lld, pitch %lld)", (int)r,
                  (long long)rows, (long long)K, (long long)ld);
    return MOE_ERR_CUDA;
  }
  return MOE_OK;
}

struct RouterPlan {
  int64_t blocks;
  int n_mma, KT, slices, splits, stages;
};

RouterPlan rt_plan(int64_t T, int64_t K, int E) {
  RouterPlan pl;
  pl.blocks = cdiv64(T, RT_BLOCK_T);
  pl.n_mma = (E + 15) / 16 * 16;
  pl.KT = (int)cdiv64(K, 64);
  // Few token blocks: cut K so that many SMs pull a share of the operands.  Slices get longer as blocks get more: at least 2 k steps
  // with one block, 12 from six on.  They go to the CTAs of a cluster, eight at most (the portable size), several to each where there are
  // more.  Not a matter of speed alone: the error of a slice's sum grows with its steps (64 tokens, K = 2880: 22 slices 1.1e-7 from the
  // exact logits, eight 2.3e-7; 6000 tokens: three 6.4e-7, two 9.9e-7), and its last bit can become a step of the logit rounded to bf16.
  int64_t s = moe_sm_count() / (pl.blocks > 0 ? pl.blocks : 1);
  const int64_t min_steps = pl.blocks >= 6 ? 12 : 2 * pl.blocks;
  if (s > pl.KT / min_steps) s = pl.KT / min_steps;
  pl.slices = s < 1 ? 1 : (int)s;
  pl.splits = pl.slices > 8 ? 8 : pl.slices;
  const int stage_bytes = RT_BLOCK_T * 128 + ((pl.n_mma * 128 + 1023) & ~1023);
  int st = (200 * 1024) / stage_bytes;
  pl.stages = st > RT_STAGES_MAX ? RT_STAGES_MAX : st;
  return pl;
}

}  // namespace

extern "C" __attribute__((visibility("default"))) size_t moe_router_topk_workspace_bytes(int64_t T, int64_t K, int E) {
  (void)T; (void)K; (void)E;
  return 0;                                             // the partial sums stay on chip
}

extern "C" __attribute__((visibility("default"))) int moe_router_topk(
    const void* x, int64_t T, int64_t K, int64_t ld_x, const void* wg_t, int64_t ld_wg, const void* bias, int bias_dtype, int E,
    int k, int apply_softmax, int round_bf16, float* logits_out, int64_t ld_logits, void* vals, int vals_dtype, int64_t ld_vals, int16_t* indx,
    int64_t ld_indx, uint32_t* bitmatrix, int64_t bm_stride_row, int64_t bm_stride_word, void* workspace, size_t workspace_bytes,
    int32_t* status, void* stream) {
  if (T == 0) return MOE_OK;
  MOE_CHECK_ARG(x && wg_t && vals && indx && bitmatrix, "moe_router_topk: NULL argument");
  MOE_CHECK_ARG(T > 0 && K > 0 && E > 0, "moe_router_topk: T, K and E must be positive");
  if (E > 256 || !(k == 1 || k == 2 || k == 4 || k == 8 || k == 16) || k > E) {
    moe_set_error("moe_router_topk: needs at most 256 experts and k in {1, 2, 4, 8, 16} (got E = %d, k = %d)", E, k);
    return MOE_ERR_UNSUPPORTED;
  }
  if (K % 8 != 0 || ld_x % 8 != 0 || ld_wg % 8 != 0 || (uintptr_t)x % 16 != 0 || (uintptr_t)wg_t % 16 != 0) {
    moe_set_error("moe_router_topk: x and Wg^T need 16-byte aligned rows (K, pitches multiples of 8 bf16)");
    return MOE_ERR_UNSUPPORTED;
  }
  MOE_CHECK_ARG(vals_dtype == MOE_F32 || vals_dtype == MOE_BF16, "moe_router_topk: values are fp32 or bf16");
  MOE_CHECK_ARG(!bias || bias_dtype == MOE_F32 || bias_dtype == MOE_BF16, "moe_router_topk: bias is fp32 or bf16");
  MOE_CHECK_ARG(T < (1ll << 31) - 256, "moe_router_topk: too many tokens");
  const RouterPlan pl = rt_plan(T, K, E);
  cudaStream_t st = (cudaStream_t)stream;
  RouterParams p;
  p.T = T; p.E = E; p.n_mma = pl.n_mma; p.k = k; p.KT = pl.KT; p.slices = pl.slices; p.splits = pl.splits; p.stages = pl.stages;
  p.apply_softmax = apply_softmax; p.round_bf16 = round_bf16;
  p.bias = bias; p.bias_dtype = bias_dtype;
  p.logits_out = logits_out; p.ld_logits = ld_logits;
  p.vals = vals; p.vals_dtype = vals_dtype; p.ld_vals = ld_vals;
  p.indx = indx; p.ld_indx = ld_indx;
  p.bitmatrix = bitmatrix; p.bm_stride_row = bm_stride_row; p.bm_stride_word = bm_stride_word;
  p.status = status;
  (void)workspace; (void)workspace_bytes;
  CUtensorMap x_map, w_map;
  if (int rc = rt_make_map(x, T, K, ld_x, RT_BLOCK_T, &x_map)) return rc;
  if (int rc = rt_make_map(wg_t, E, K, ld_wg, pl.n_mma, &w_map)) return rc;
  const int stage_bytes = RT_BLOCK_T * 128 + ((pl.n_mma * 128 + 1023) & ~1023);
  const int smem = pl.stages * stage_bytes + 1024;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)pl.blocks, (unsigned)pl.splits);
  cfg.blockDim = dim3(RT_THREADS);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = 1; at[1].val.clusterDim.y = (unsigned)pl.splits; at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = pl.splits > 1 ? 2 : 1;
#define RT_LAUNCH(KK)                                                                                                    \
  do {                                                                                                                   \
    MOE_CHECK_CUDA(cudaFuncSetAttribute(router_topk_kernel<KK>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));     \
    MOE_CHECK_CUDA(cudaLaunchKernelEx(&cfg, router_topk_kernel<KK>, p, x_map, w_map));                                   \
  } while (0)
  switch (k) {
    case 1: RT_LAUNCH(1); break;
    case 2: RT_LAUNCH(2); break;
    case 4: RT_LAUNCH(4); break;
    case 8: RT_LAUNCH(8); break;
    default: RT_LAUNCH(16); break;
  }
#undef RT_LAUNCH
  MOE_CHECK_LAUNCH();
  return MOE_OK;
}
