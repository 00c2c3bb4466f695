// moe_grouped_gemm: argument validation and kernel selection for the ragged grouped GEMM.
#include "gemm_common.cuh"

int moe_gemm_simt_launch(const GemmParams& p, int x_dtype, int y_dtype, int w_kind, int64_t grid_m, cudaStream_t st);
int moe_gemm_tc_launch(const GemmParams& p, const MoeGemmArgs& a, cudaStream_t st);
bool moe_gemm_tc_supported(const MoeGemmArgs& a, const char** why);
int moe_gemm_tc_pair_launch(const GemmParams& p, const MoeGemmArgs& a, cudaStream_t st);
bool moe_gemm_tc_pair_supported(const MoeGemmArgs& a, const char** why);
int moe_gemm_stream_launch(const GemmParams& p, const MoeGemmArgs& a, cudaStream_t st);
bool moe_gemm_stream_supported(const MoeGemmArgs& a, const char** why);
int moe_gemm_mx_launch(const GemmParams& p, const MoeGemmArgs& a, const TokenOut& out, bool packed, cudaStream_t st);
int moe_gemm_mx_terms(const MoeGemmArgs& a);
bool moe_gemm_mx_token_out(const MoeGemmArgs& a, TokenOut& out);
bool moe_gemm_mx_pair_token_out(const MoeGemmArgs& a, TokenOut& out);
bool moe_gemm_mx_supported(const MoeGemmArgs& a, const char** why);
bool moe_gemm_mx_pair_wanted(const MoeGemmArgs& a);
int64_t moe_gemm_mx_pair_workspace(const MoeGemmArgs& a);
int moe_gemm_mx_pair_launch(const GemmParams& p, const MoeGemmArgs& a, const TokenOut& out, bool packed, cudaStream_t st);

// upper bound on the number of row blocks (triton_kernels tensor_details/ragged_tensor.py:73-77)
static int64_t n_blocks_bound(int64_t n_slices, int64_t n_rows, int64_t block) {
  if (n_rows <= n_slices) return n_rows;
  int64_t a = n_slices - n_rows - 1;                 // negative
  int64_t fl = -((-a + block - 1) / block);          // floor division
  return n_slices - 1 - fl;
}

namespace {

enum Kernel { K_MX_PAIR, K_MX, K_STREAM, K_TC, K_TC_PAIR, K_SIMT };
const char* const KERNEL_NAME[] = {"gemm_mx_pair_kernel", "gemm_mx_kernel", "gemm_stream_kernel", "gemm_tc_kernel", "gemm_tc_pair_kernel",
                                   "gemm_simt_kernel"};

int check_args(const MoeGemmArgs* a) {
  MOE_CHECK_ARG(a != nullptr, "moe_grouped_gemm: args is NULL");
  MOE_CHECK_ARG(a->E > 0 && a->K >= 0 && a->N >= 0 && a->M >= 0, "moe_grouped_gemm: bad extents E=%d K=%d N=%d M=%lld",
                a->E, a->K, a->N, (long long)a->M);
  if (a->M == 0 || a->N == 0) return MOE_OK;
  MOE_CHECK_ARG(a->x && a->w && (a->y || a->n_y_peers > 0), "moe_grouped_gemm: NULL x / w / y");
  MOE_CHECK_ARG(a->w_kind == MOE_W_DENSE || a->w_scale, "moe_grouped_gemm: MXFP4 weights need w_scale");
  MOE_CHECK_ARG(a->w_kind == MOE_W_DENSE || a->K % 32 == 0, "moe_grouped_gemm: MXFP4 weights need K %% 32 == 0 (K=%d)", a->K);
  MOE_CHECK_ARG(a->activation == MOE_ACT_NONE || (a->activation == MOE_ACT_SWIGLU && a->N % 2 == 0),
                "moe_grouped_gemm: SwiGLU needs an even N");
  if (a->slice_sizes) {
    MOE_CHECK_ARG(a->slice_offs && a->block_offs_16 && a->block_sched_16, "moe_grouped_gemm: ragged metadata incomplete");
  } else {
    MOE_CHECK_ARG(a->E == 1, "moe_grouped_gemm: without ragged metadata there must be one weight matrix");
  }
  MOE_CHECK_ARG(a->n_y_peers >= 0 && a->n_y_peers <= MOE_MAX_PEERS, "moe_grouped_gemm: n_y_peers must be 0..%d", MOE_MAX_PEERS);
  if (a->n_y_peers > 0) {
    MOE_CHECK_ARG(a->y_rows_per_peer > 0, "moe_grouped_gemm: y_rows_per_peer must be positive with y_peers");
    for (int i = 0; i < a->n_y_peers; ++i)
      MOE_CHECK_ARG(a->y_peers[i] != nullptr && (uintptr_t)a->y_peers[i] % 16 == 0,
                    "moe_grouped_gemm: y_peers[%d] is NULL or not 16-byte aligned", i);
  }
  return MOE_OK;
}

// The kernel of a call, or the status (and error) of a refused one.  `workspace`: the block-scaled kernels' workspace is there.
int choose_kernel(const MoeGemmArgs& a, bool workspace, Kernel& out) {
  const char* why = "";
  const bool mx_asked = a.kernel == MOE_GEMM_MX || a.kernel == MOE_GEMM_MX_F8 || a.kernel == MOE_GEMM_MX_F4;
  // default tiles on the block-scaled pair kernel; without its workspace they stay with the kernels below
  if (a.w_kind == MOE_W_MX4_B200 && (mx_asked || workspace) && moe_gemm_mx_pair_wanted(a)) {
    out = K_MX_PAIR;
    return MOE_OK;
  }
  if (a.w_kind == MOE_W_MX4_B200MX || mx_asked) {
    // weights laid out for the block-scaled MMA: that kernel or nothing
    if (!moe_gemm_mx_supported(a, &why) || (a.kernel != MOE_GEMM_AUTO && !mx_asked)) {
      moe_set_error("moe_grouped_gemm: block-scaled kernel not applicable: %s", *why ? why : "another kernel was requested");
      return MOE_ERR_UNSUPPORTED;
    }
    out = moe_gemm_mx_pair_wanted(a) ? K_MX_PAIR : K_MX;
    return MOE_OK;
  }
  const bool tc = moe_gemm_tc_supported(a, &why);
  if ((a.kernel == MOE_GEMM_TCGEN05 || a.kernel == MOE_GEMM_TCGEN05_PAIR || a.kernel == MOE_GEMM_STREAM) && !tc) {
    moe_set_error("moe_grouped_gemm: tcgen05 kernel not applicable: %s", why);
    return MOE_ERR_UNSUPPORTED;
  }
  if (!tc || a.kernel == MOE_GEMM_SIMT) {
    MOE_CHECK_ARG(a.w_kind == MOE_W_DENSE || a.w_kind == MOE_W_MX4_CANONICAL,
                  "moe_grouped_gemm: the SIMT kernel takes dense or canonical MXFP4 weights (%s)", why);
    out = K_SIMT;
    return MOE_OK;
  }
  // A few rows per expert (decode): the weight-streaming kernel, bound by HBM rather than by pipeline hand-offs.
  const bool streams = moe_gemm_stream_supported(a, &why);
  if (a.kernel == MOE_GEMM_STREAM && !streams) {
    moe_set_error("moe_grouped_gemm: streaming kernel not applicable: %s", why);
    return MOE_ERR_UNSUPPORTED;
  }
  if (a.kernel == MOE_GEMM_STREAM ||
      (a.kernel == MOE_GEMM_AUTO && streams && a.tile_m == 0 && a.tile_n == 0 && a.M <= 10 * (int64_t)a.E)) {
    out = K_STREAM;
    return MOE_OK;
  }
  // (the bf16 kernel on pairs of SMs, 256 x 256 tiles, runs on request only)
  if (a.kernel == MOE_GEMM_TCGEN05_PAIR && !moe_gemm_tc_pair_supported(a, &why)) {
    moe_set_error("moe_grouped_gemm: SM-pair tcgen05 kernel not applicable: %s", why);
    return MOE_ERR_UNSUPPORTED;
  }
  out = a.kernel == MOE_GEMM_TCGEN05_PAIR ? K_TC_PAIR : K_TC;
  return MOE_OK;
}

}  // namespace

extern "C" __attribute__((visibility("default"))) const char* moe_gemm_kernel_name(const MoeGemmArgs* a) {
  if (check_args(a) != MOE_OK) return nullptr;
  if (a->M == 0 || a->N == 0) return "";
  Kernel k;
  return choose_kernel(*a, true, k) == MOE_OK ? KERNEL_NAME[k] : nullptr;
}

static bool has_workspace(const MoeGemmArgs* a) { return a->mx_workspace && a->mx_workspace_bytes >= moe_gemm_mx_pair_workspace(*a); }

// The product on the kernel chosen for it.  out: its rows go there instead of y (block-scaled kernels); packed: its tokens are in
// the workspace already.
static int run_product(const MoeGemmArgs* a, Kernel kernel, const TokenOut& out, bool packed, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  GemmParams p;
  p.x = a->x; p.ld_x = a->ld_x; p.rows_x = a->rows_x;
  p.w = a->w; p.w_stride_e = a->w_stride_e; p.w_stride_k = a->w_stride_k; p.w_stride_n = a->w_stride_n;
  p.w_scale = a->w_scale; p.ws_stride_e = a->ws_stride_e; p.ws_stride_k = a->ws_stride_k; p.ws_stride_n = a->ws_stride_n;
  p.E = a->E; p.K = a->K; p.N = a->N;
  p.slice_sizes = a->slice_sizes; p.slice_offs = a->slice_offs;
  p.block_offs = nullptr; p.block_sched = nullptr;
  p.M = a->M;
  p.bias = a->bias; p.bias_dtype = a->bias_dtype; p.ld_bias = a->ld_bias;
  p.gather_indx = a->gather_indx; p.scatter_indx = a->scatter_indx;
  p.betas = a->betas; p.gammas = a->gammas;
  p.out_alpha = a->out_alpha; p.has_out_alpha = a->has_out_alpha;
  p.activation = a->activation; p.act_alpha = a->act_alpha; p.act_limit = a->act_limit; p.act_has_limit = a->act_has_limit;
  p.y = a->n_y_peers > 0 ? a->y_peers[0] : a->y; p.ld_y = a->ld_y;
  p.status = a->status;
  p.n_y_peers = a->n_y_peers; p.y_rows_per_peer = a->y_rows_per_peer;
  for (int i = 0; i < MOE_MAX_PEERS; ++i) p.y_peers[i] = i < a->n_y_peers ? a->y_peers[i] : nullptr;

  if (kernel == K_MX_PAIR) return moe_gemm_mx_pair_launch(p, *a, out, packed, st);
  if (kernel == K_MX) return moe_gemm_mx_launch(p, *a, out, packed, st);
  if (kernel == K_STREAM) return moe_gemm_stream_launch(p, *a, st);
  if (kernel == K_TC || kernel == K_TC_PAIR) {
    // Large gathered problems: copy the gathered rows once into the caller's scratch, then stream them by TMA.
    const bool big = (a->tile_m == 0 || a->tile_m == 256) && (a->tile_m == 256 || a->M / a->E >= 12);
    if (a->gather_indx && a->gather_scratch && big && a->gather_scratch_bytes >= (int64_t)a->M * a->K * 2) {
      const int rc = moe_gather_rows(a->x, a->ld_x * 2, a->gather_indx, a->M, (int64_t)a->K * 2, a->gather_scratch,
                                     (int64_t)a->K * 2, stream);
      if (rc != MOE_OK) return rc;
      p.x = a->gather_scratch; p.ld_x = a->K; p.rows_x = a->M; p.gather_indx = nullptr;
    }
    return kernel == K_TC_PAIR ? moe_gemm_tc_pair_launch(p, *a, st) : moe_gemm_tc_launch(p, *a, st);
  }

  int64_t grid_m;
  if (a->slice_sizes) {
    p.block_offs = a->block_offs_16 + 2 * a->ld_block_offs;     // block size 64
    p.block_sched = a->block_sched_16 + 2 * a->ld_block_sched;
    grid_m = n_blocks_bound(a->E, a->M, 64);
  } else {
    grid_m = cdiv64(a->M, 64);
  }
  if (grid_m == 0) return MOE_OK;
  return moe_gemm_simt_launch(p, a->x_dtype, a->y_dtype, a->w_kind, grid_m, st);
}

extern "C" __attribute__((visibility("default"))) int moe_grouped_gemm(const MoeGemmArgs* a, void* stream) {
  if (const int rc = check_args(a)) return rc;
  if (a->M == 0 || a->N == 0) return MOE_OK;
  Kernel kernel;
  if (const int rc = choose_kernel(*a, has_workspace(a), kernel)) return rc;
  return run_product(a, kernel, TokenOut(), false, stream);
}

// Whether product a may leave its rows as the tokens of product b, and where.  Both run on block-scaled kernels; b takes exactly a's
// rows (all of them, at the pitch they would be written with), in the same ragged structure, from workspace of its own that holds
// nothing a reads; nothing but bias and activation is between.  bf16 rows: a limit on the activation, which bounds them far below where two terms stop holding a value (the pack kernels have a way for such rows):
// |silu(g)| <= max(limit, 0.28 / alpha) and the factor <= limit + 1.
static bool hands_over(const MoeGemmArgs& a, Kernel ka, const MoeGemmArgs& b, Kernel kb, TokenOut& out) {
  if ((ka != K_MX_PAIR && ka != K_MX) || (kb != K_MX_PAIR && kb != K_MX)) return false;
  if (a.activation != MOE_ACT_SWIGLU || a.N % 64 != 0 || a.N != 2 * b.K || a.M != b.M || a.E != b.E || b.x != a.y || b.x_dtype != a.y_dtype ||
      b.ld_x != a.ld_y || b.rows_x < b.M || b.gather_indx || b.x_scale || a.scatter_indx || a.betas || a.gammas || a.has_out_alpha || a.n_y_peers > 0)
    return false;
  if (!a.slice_sizes || a.slice_sizes != b.slice_sizes || a.slice_offs != b.slice_offs || a.block_offs_16 != b.block_offs_16 ||
      a.block_sched_16 != b.block_sched_16)
    return false;
  const uint8_t* wb = (const uint8_t*)b.mx_workspace;
  auto within = [&](const void* at, int64_t bytes) {
    return at && (const uint8_t*)at < wb + b.mx_workspace_bytes && wb < (const uint8_t*)at + bytes;
  };
  if (within(a.mx_workspace, a.mx_workspace_bytes) || within(a.x, a.rows_x * a.ld_x * (a.x_dtype == MOE_BF16 ? 2 : 1)) ||
      within(a.x_scale, a.rows_x * a.ld_x_scale) || within(a.gather_indx, a.M * 4) || within(a.x_positions, a.rows_x * a.x_k * 4) ||
      within(a.x_experts, a.rows_x * a.x_k * 2))
    return false;
  const bool bf16 = a.y_dtype == MOE_BF16;
  if (bf16 && !(a.act_has_limit && a.act_limit > 0.0f && a.act_limit < 1e9f && a.act_alpha > 1e-9f)) return false;
  if (!bf16 && a.y_dtype != MOE_F8E4M3) return false;
  if ((uintptr_t)wb % 1024 != 0 || !(kb == K_MX_PAIR ? moe_gemm_mx_pair_token_out(b, out) : moe_gemm_mx_token_out(b, out))) return false;
  // (a kernel has its own tokens' terms to write: the rules choose the same for both products but at the edges)
  const int terms = ka == K_MX ? moe_gemm_mx_terms(a) : bf16 ? 2 : 1;
  if (out.terms == terms && a.x_dtype == a.y_dtype) return true;
  out = TokenOut();
  return false;
}

extern "C" __attribute__((visibility("default"))) int moe_grouped_gemm_chain(const MoeGemmArgs* a, const MoeGemmArgs* b, void* stream) {
  if (const int rc = check_args(a)) return rc;
  if (const int rc = check_args(b)) return rc;
  if (a->M == 0 || a->N == 0 || b->M == 0 || b->N == 0) {
    const int rc = moe_grouped_gemm(a, stream);
    return rc ? rc : moe_grouped_gemm(b, stream);
  }
  Kernel ka, kb;
  if (const int rc = choose_kernel(*a, has_workspace(a), ka)) return rc;
  if (const int rc = choose_kernel(*b, has_workspace(b), kb)) return rc;
  TokenOut out;
  const bool over = hands_over(*a, ka, *b, kb, out);
  const int rc = run_product(a, ka, out, false, stream);
  return rc ? rc : run_product(b, kb, TokenOut(), over, stream);
}
