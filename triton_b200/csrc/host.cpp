// Native host path of the operators: allocation of outputs and temporaries through torch's caching allocator, argument
// blocks and calls into libmoe_b200.so, for the sequences that Python spent longer on than the GPU (an eager layer step of
// 16 tokens: 180 us of host work for 100 us of kernels).  No computation happens here; the library is the one the Python
// binding loaded (its handle is passed in), and every entry point keeps its checks and messages.
#include <torch/extension.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include "../../include/moe_b200.h"

namespace py = pybind11;
using at::Tensor;
using OptTensor = std::optional<Tensor>;

namespace {

struct Lib {
#define MOE_HOST_FUNCTIONS(X)                                                                                            \
  X(moe_last_error) X(moe_route) X(moe_route_positions) X(moe_route_workspace) X(moe_grouped_gemm) X(moe_gemm_mx_workspace_bytes) \
  X(moe_reduce) X(moe_downcast_mxfp4) X(moe_upcast_mxfp4) X(moe_bitmatrix_metadata) X(moe_bitmatrix_metadata_workspace) \
  X(moe_router_topk) X(moe_copy2) X(moe_step_graph_create) X(moe_step_graph_launch) X(moe_step_graph_destroy) \
  X(moe_gemm_kernel_name) X(moe_grouped_gemm_chain)
#define X(name) decltype(&::name) name = nullptr;
  MOE_HOST_FUNCTIONS(X)
#undef X
} lib;

PyObject* inapplicable = nullptr;        // exception class of a refused tuning constraint

void bind(int64_t handle, py::object inapplicable_cls) {
#define X(name)                                                                      \
  lib.name = reinterpret_cast<decltype(&::name)>(dlsym(reinterpret_cast<void*>(handle), #name)); \
  if (!lib.name) throw std::runtime_error("libmoe_b200 does not export " #name);
  MOE_HOST_FUNCTIONS(X)
#undef X
  inapplicable = inapplicable_cls.inc_ref().ptr();
}

[[noreturn]] void raise(PyObject* cls, const std::string& msg) {
  PyErr_SetString(cls, msg.c_str());
  throw py::error_already_set();
}

void check(int status, const char* what, bool tuning = false) {
  if (status == 0) return;
  const char* m = lib.moe_last_error();
  if (status == 3 && tuning) raise(inapplicable, m ? m : "");
  raise(status == 3 ? PyExc_NotImplementedError : (status == 1 ? PyExc_ValueError : PyExc_RuntimeError),
        std::string(what) + " failed (status " + std::to_string(status) + "): " + (m ? m : ""));
}

void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return MOE_F32;
    case at::kHalf: return MOE_F16;
    case at::kBFloat16: return MOE_BF16;
    case at::kFloat8_e4m3fn: return MOE_F8E4M3;
    default: raise(PyExc_ValueError, std::string("unsupported dtype ") + c10::toString(t));
  }
}
int dtype_code(const Tensor& t) { return dtype_code(t.scalar_type()); }

void need_cuda(const Tensor& t) {
  if (!t.is_cuda()) raise(PyExc_ValueError, "triton_b200 operators take CUDA tensors only (no CPU path)");
}

Tensor empty(at::IntArrayRef shape, at::ScalarType t, const Tensor& like) {
  return at::empty(shape, at::TensorOptions().dtype(t).device(like.device()));
}

// part of `base` from element `offset` on.  Made directly: as narrow / view / select through the dispatcher the parts of a routing
// result took a third of the call's host time (604 tokens: 29 us, so 18.6).
Tensor part(const Tensor& base, int64_t offset, at::IntArrayRef shape, at::IntArrayRef strides) {
  auto impl = c10::make_intrusive<at::TensorImpl>(c10::TensorImpl::VIEW, c10::Storage(base.storage()), base.key_set(), base.dtype());
  impl->set_storage_offset(base.storage_offset() + offset);
  impl->set_sizes_and_strides(shape, strides);
  return Tensor(std::move(impl));
}

int64_t cdiv(int64_t a, int64_t b) { return (a + b - 1) / b; }
int64_t pad512(int64_t n) { return std::max<int64_t>(cdiv(n, 512) * 512, 512); }
// upper bound on the blocks of 16 rows (RaggedTensorMetadata.max_n_blocks)
int64_t max_blocks16(int64_t E, int64_t n) { return n <= E ? n : E - 1 + cdiv(n + 1 - E, 16); }

// ---- routing -----------------------------------------------------------------------------------------------------
// -> vals, indx, bitmatrix view [T, words], col_sum, col_sorted, row_sorted, slice_offs, block_offs, block_schedule, token of
// every position (float logits; else None)
py::tuple route(const Tensor& logits, int64_t k, bool softmax) {
  need_cuda(logits);
  const int64_t T = logits.size(0), E = logits.size(1), n = T * k;
  const int code = dtype_code(logits);
  Tensor vals = empty({T, k}, logits.scalar_type(), logits), indx = empty({T, k}, at::kShort, logits);
  const int64_t t_pad = cdiv(T, 32) * 32, words = cdiv(E, 32);
  Tensor bm_all = empty({words, t_pad}, at::kInt, logits), bm = part(bm_all, 0, {T, words}, {1, t_pad});
  const int64_t mnb = max_blocks16(E, n), lo = pad512(E + 1), ls = pad512(mnb);
  // the index arrays, the metadata rows and the scratch are parts of one buffer; every row of the metadata starts on 2 KB
  const size_t ws = lib.moe_route_workspace(T, (int)E, (int)k);
  const int64_t at_sched = 5 * lo, at_col = at_sched + 4 * ls, at_row = at_col + n, at_tok = at_row + n, at_sum = at_tok + n,
                at_work = cdiv(at_sum + E, 64) * 64;
  Tensor buf = empty({at_work + cdiv((int64_t)ws, 4)}, at::kInt, logits);
  Tensor sched = part(buf, at_sched, {4, mnb}, {ls, 1}), col_sorted = part(buf, at_col, {n}, {1}), row_sorted = part(buf, at_row, {n}, {1});
  Tensor tokens = part(buf, at_tok, {n}, {1}), col_sum = part(buf, at_sum, {E}, {1});
  int32_t* b = buf.data_ptr<int32_t>();
  const bool positions = code == MOE_F32;
  if (positions)
    check(lib.moe_route_positions(logits.data_ptr<float>(), T, (int)E, (int)k, softmax, logits.stride(0), vals.data_ptr<float>(), k,
                                  indx.data_ptr<int16_t>(), k, (uint32_t*)bm.data_ptr(), bm.stride(0), bm.stride(1),
                                  col_sum.data_ptr<int32_t>(), col_sorted.data_ptr<int32_t>(), row_sorted.data_ptr<int32_t>(), b, b + lo,
                                  lo, b + 5 * lo, ls, mnb, tokens.data_ptr<int32_t>(), nullptr, b + at_work, ws, stream()),
          "moe_route_positions");
  else
    check(lib.moe_route(logits.data_ptr(), code, T, (int)E, (int)k, softmax, logits.stride(0), vals.data_ptr(), k,
                      indx.data_ptr<int16_t>(), k, (uint32_t*)bm.data_ptr(), bm.stride(0), bm.stride(1), col_sum.data_ptr<int32_t>(),
                      col_sorted.data_ptr<int32_t>(), row_sorted.data_ptr<int32_t>(), b, b + lo, lo, b + 5 * lo, ls, mnb, b + at_work,
                      ws, stream()),
        "moe_route");
  return py::make_tuple(vals, indx, bm, col_sum, col_sorted, row_sorted, part(buf, 0, {E + 1}, {1}), part(buf, lo, {4, E + 1}, {lo, 1}), sched,
                        positions ? py::cast(tokens) : py::none());
}

// -> col_sum, col_sorted, row_sorted
py::tuple bitmatrix_metadata(const Tensor& indx, int64_t E, const OptTensor& n_rows) {
  need_cuda(indx);
  if (n_rows) need_cuda(*n_rows);
  const int64_t T = indx.size(0), k = indx.size(1), n = T * k;
  const size_t ws = lib.moe_bitmatrix_metadata_workspace(T, (int)E, (int)k);
  const int64_t at_work = cdiv(2 * n + E, 64) * 64;
  Tensor buf = empty({at_work + cdiv((int64_t)ws, 4)}, at::kInt, indx);
  Tensor col_sorted = part(buf, 0, {n}, {1}), row_sorted = part(buf, n, {n}, {1}), col_sum = part(buf, 2 * n, {E}, {1});
  check(lib.moe_bitmatrix_metadata(indx.data_ptr<int16_t>(), indx.stride(0), T, (int)E, (int)k,
                                   n_rows ? n_rows->data_ptr<int32_t>() : nullptr, col_sum.data_ptr<int32_t>(),
                                   col_sorted.data_ptr<int32_t>(), row_sorted.data_ptr<int32_t>(), buf.data_ptr<int32_t>() + at_work, ws, stream()),
        "moe_bitmatrix_metadata");
  return py::make_tuple(col_sum, col_sorted, row_sorted);
}

// ---- grouped GEMM ------------------------------------------------------------------------------------------------
// Temporary bytes of one call: the block-scaled kernels' token workspace, else the bf16 kernel's gathered rows (2048 and more:
// the library decides whether to use them), else none.
int64_t temp_bytes(MoeGemmArgs& g, bool gathers, bool& workspace) {
  const bool tiles = g.w_kind == MOE_W_MX4_B200 || g.w_kind == MOE_W_MX4_B200MX;
  const int64_t ws = tiles ? (int64_t)lib.moe_gemm_mx_workspace_bytes(&g) : 0;
  workspace = ws > 0;
  if (workspace) return ws;
  return gathers && g.w_kind == MOE_W_MX4_B200 && g.x_dtype == MOE_BF16 && g.M >= 2048 ? g.M * g.K * 2 : 0;
}
void set_temp(MoeGemmArgs& g, void* at, int64_t bytes, bool workspace) {
  if (bytes == 0) return;
  if (workspace) { g.mx_workspace = at; g.mx_workspace_bytes = bytes; }
  else { g.gather_scratch = at; g.gather_scratch_bytes = bytes; }
}

int run_gemm(MoeGemmArgs& g, const Tensor& like) {
  bool workspace;
  const int64_t bytes = temp_bytes(g, g.gather_indx != nullptr, workspace);
  Tensor temp;
  if (bytes > 0) {
    temp = empty({bytes + 1024}, at::kByte, like);
    set_temp(g, (void*)(((uintptr_t)temp.data_ptr() + 1023) / 1024 * 1024), bytes, workspace);
  }
  return lib.moe_grouped_gemm(&g, stream());
}

const int32_t* i32(const OptTensor& t, std::vector<Tensor>& keep) {
  if (!t) return nullptr;
  keep.push_back(t->to(at::kInt).contiguous());              // (both are no-ops on what this package makes)
  return keep.back().data_ptr<int32_t>();
}
const float* f32(const OptTensor& t, std::vector<Tensor>& keep) {
  if (!t) return nullptr;
  keep.push_back(t->to(at::kFloat).contiguous());
  return keep.back().data_ptr<float>();
}

void set_tuning(MoeGemmArgs& g, const py::tuple& t) {
  g.kernel = t[0].cast<int>(); g.tile_m = t[1].cast<int>(); g.tile_n = t[2].cast<int>(); g.idle_sms = t[3].cast<int>();
}

void set_weights(MoeGemmArgs& g, int kind, const Tensor& w, const OptTensor& ws) {
  g.w_kind = kind;
  need_cuda(w);
  g.w = w.data_ptr();
  if (kind == MOE_W_DENSE) {
    g.w_stride_e = w.stride(0); g.w_stride_k = w.stride(1); g.w_stride_n = w.stride(2);
    return;
  }
  g.w_scale = (const uint8_t*)ws->data_ptr();
  if (kind == MOE_W_MX4_CANONICAL) {
    g.w_stride_e = w.stride(0); g.w_stride_k = 1; g.w_stride_n = w.stride(2);
    g.ws_stride_e = ws->stride(0); g.ws_stride_k = ws->stride(1); g.ws_stride_n = ws->stride(2);
  }
}

// y is the caller's output tensor or None (allocated here); `ragged` is (slice_sizes, slice_offs, block_offs, schedule, expected
// rows per expert or 0) or None;
// `peers` is (device addresses, rows per peer) or None.
Tensor gemm(const Tensor& a, int kind, const Tensor& w, const OptTensor& ws, int64_t E, int64_t K, int64_t N, const py::object& ragged,
            const OptTensor& bias, const OptTensor& gather, const OptTensor& scatter, const OptTensor& betas, const OptTensor& gammas,
            std::optional<double> out_alpha, const py::object& swiglu, const OptTensor& y, py::object out_dtype, const OptTensor& a_scale,
            const py::tuple& tuning, const Tensor& status, const py::object& peers) {
  need_cuda(a);
  std::vector<Tensor> keep;
  keep.reserve(8);
  MoeGemmArgs g{};
  g.x = a.data_ptr(); g.x_dtype = dtype_code(a); g.ld_x = a.stride(0); g.rows_x = a.size(0);
  set_weights(g, kind, w, ws);
  g.E = (int)E; g.K = (int)K; g.N = (int)N;
  g.M = gather ? gather->size(0) : a.size(0);
  if (!ragged.is_none()) {
    const py::tuple r = ragged;
    const Tensor sizes = r[0].cast<Tensor>(), offs = r[1].cast<Tensor>(), boffs = r[2].cast<Tensor>(), sched = r[3].cast<Tensor>();
    if (boffs.stride(1) != 1 || sched.stride(1) != 1) raise(PyExc_AssertionError, "ragged metadata rows must be contiguous");
    g.slice_sizes = sizes.data_ptr<int32_t>(); g.slice_offs = offs.data_ptr<int32_t>();
    g.block_offs_16 = boffs.data_ptr<int32_t>(); g.block_sched_16 = sched.data_ptr<int32_t>();
    g.ld_block_offs = boffs.stride(0); g.ld_block_sched = sched.stride(0);
    g.rows_per_expert = r[4].cast<int>();
  }
  if (bias) { g.bias = bias->data_ptr(); g.bias_dtype = dtype_code(*bias); g.ld_bias = bias->stride(0); }
  g.gather_indx = i32(gather, keep); g.scatter_indx = i32(scatter, keep);
  g.betas = f32(betas, keep); g.gammas = f32(gammas, keep);
  if (out_alpha) { g.out_alpha = (float)*out_alpha; g.has_out_alpha = 1; }
  if (!swiglu.is_none()) {
    const py::tuple s = swiglu;
    g.activation = MOE_ACT_SWIGLU; g.act_alpha = s[0].cast<float>();
    if (!s[1].is_none()) { g.act_limit = s[1].cast<float>(); g.act_has_limit = 1; }
  }
  Tensor out = y ? *y : empty({g.M, swiglu.is_none() ? N : N / 2}, torch::python::detail::py_object_to_dtype(out_dtype), a);
  g.y = out.data_ptr(); g.y_dtype = dtype_code(out); g.ld_y = out.stride(0);
  if (!peers.is_none()) {
    const py::tuple pr = peers;
    const auto handles = pr[0].cast<std::vector<int64_t>>();
    g.n_y_peers = (int)handles.size(); g.y_rows_per_peer = pr[1].cast<int64_t>();
    for (size_t i = 0; i < handles.size(); ++i) g.y_peers[i] = (void*)handles[i];
  }
  if (a_scale) { g.x_scale = (const uint8_t*)a_scale->data_ptr(); g.ld_x_scale = a_scale->stride(0); }
  set_tuning(g, tuning);
  g.status = status.data_ptr<int32_t>();
  check(run_gemm(g, a), "moe_grouped_gemm", true);
  return out;
}

// name of the kernel of a ragged product of M rows on aligned operands in weight tiles `kind` (no tensors: a question to the dispatch)
std::string gemm_kernel(int kind, int64_t E, int64_t K, int64_t N, int64_t M, py::object x_dtype, py::object y_dtype, const py::tuple& tuning,
                        int rows_per_expert, bool swiglu) {
  MoeGemmArgs g{};
  void* const some = (void*)(uintptr_t)4096;
  g.x = g.y = some; g.w = some; g.w_scale = (const uint8_t*)some; g.w_kind = kind;
  g.slice_sizes = g.slice_offs = g.block_offs_16 = g.block_sched_16 = (const int32_t*)some;
  g.E = (int)E; g.K = (int)K; g.N = (int)N; g.M = g.rows_x = M; g.ld_x = K; g.ld_y = N;
  g.x_dtype = dtype_code(torch::python::detail::py_object_to_dtype(x_dtype));
  g.y_dtype = dtype_code(torch::python::detail::py_object_to_dtype(y_dtype));
  set_tuning(g, tuning);
  g.rows_per_expert = rows_per_expert;
  g.activation = swiglu ? MOE_ACT_SWIGLU : MOE_ACT_NONE;
  const char* name = lib.moe_gemm_kernel_name(&g);
  if (!name) raise(inapplicable, lib.moe_last_error());
  return name;
}

// ---- one layer step ------------------------------------------------------------------------------------------------
struct Carver {                          // parts of one buffer, each on its own 1 KB boundary
  int64_t bytes = 0;
  int64_t take(int64_t n) { const int64_t at = bytes; bytes += cdiv(n, 1024) * 1024; return at; }
};

// w: (w_kind, values, scales, bias, K, N)
void set_product(MoeGemmArgs& g, const py::tuple& w, int64_t E, int64_t n, const py::tuple& tuning, const Tensor& status) {
  set_weights(g, w[0].cast<int>(), w[1].cast<Tensor>(), w[2].cast<Tensor>());
  const Tensor bias = w[3].cast<Tensor>();
  g.bias = bias.data_ptr(); g.bias_dtype = dtype_code(bias); g.ld_bias = bias.stride(0);
  g.E = (int)E; g.K = w[4].cast<int>(); g.N = w[5].cast<int>(); g.M = n;
  set_tuning(g, tuning);
  g.status = status.data_ptr<int32_t>();
}

// routing -> fc1 (+ bias, SwiGLU) -> fc2 (+ bias, x routing weight) -> sum over the k slots.  Every temporary is a part of one
// buffer: two allocations per step.  fc1's temporary is over when fc2's output begins and shares its place; fc2's is apart, since fc1 may
// write its rows there.
Tensor layer(const Tensor& x, const Tensor& logits, int64_t k, const py::tuple& w1, const py::tuple& w2, double alpha,
             std::optional<double> limit, const py::tuple& tuning, const Tensor& status) {
  need_cuda(x); need_cuda(logits);
  const int64_t T = x.size(0), E = logits.size(1), n = T * k;
  const bool fp8 = x.scalar_type() == at::kFloat8_e4m3fn;
  MoeGemmArgs g1{}, g2{};
  set_product(g1, w1, E, n, tuning, status);
  set_product(g2, w2, E, n, tuning, status);
  g1.x_dtype = dtype_code(x); g2.x_dtype = g1.x_dtype;
  g1.x = x.data_ptr(); g1.ld_x = x.stride(0); g1.rows_x = T;
  const int64_t ff = g1.N / 2, d = g2.N, h_size = fp8 ? 1 : 2;
  static int32_t present = 0;            // only tells the size query that there is ragged metadata
  g1.slice_sizes = g2.slice_sizes = &present;
  const int64_t lo = pad512(E + 1), mnb = max_blocks16(E, n), ls = pad512(mnb), words = cdiv(E, 32), t_pad = cdiv(T, 32) * 32;
  const int64_t route_ws = (int64_t)lib.moe_route_workspace(T, (int)E, (int)k);
  g1.ld_x = x.stride(0); g2.ld_x = ff;   // (the size query looks at types, pitches and the activation too)
  g1.y_dtype = fp8 ? MOE_F8E4M3 : MOE_BF16; g2.y_dtype = MOE_BF16;
  g1.activation = MOE_ACT_SWIGLU; g1.act_alpha = (float)alpha;
  bool ws1, ws2;
  const int64_t t1 = temp_bytes(g1, true, ws1), t2 = temp_bytes(g2, false, ws2);
  Carver c;
  const int64_t o_vals = c.take(n * 4), o_indx = c.take(n * 2), o_bm = c.take(words * t_pad * 4), o_sum = c.take(E * 4), o_col = c.take(n * 4),
                o_row = c.take(n * 4), o_offs = c.take(5 * lo * 4), o_sched = c.take(4 * ls * 4), o_rws = c.take(route_ws), o_tok = c.take(n * 4),
                o_gam = c.take(n * 4), o_h = c.take(n * ff * h_size), o_y = c.take(std::max(n * d * 2, t1)), o_tmp = c.take(t2);
  Tensor buf = empty({c.bytes + 1024}, at::kByte, x), z = empty({T, d}, at::kBFloat16, x);
  uint8_t* base = (uint8_t*)(((uintptr_t)buf.data_ptr() + 1023) / 1024 * 1024);
  void* st = stream();
  int32_t* offs = (int32_t*)(base + o_offs);
  int32_t* sched = (int32_t*)(base + o_sched);
  check(lib.moe_route_positions(logits.data_ptr<float>(), T, (int)E, (int)k, 1, logits.stride(0), (float*)(base + o_vals), k,
                                (int16_t*)(base + o_indx), k, (uint32_t*)(base + o_bm), 1, t_pad, (int32_t*)(base + o_sum),
                                (int32_t*)(base + o_col), (int32_t*)(base + o_row), offs, offs + lo, lo, sched, ls, mnb,
                                (int32_t*)(base + o_tok), (float*)(base + o_gam), base + o_rws, (size_t)route_ws, st),
        "moe_route_positions");
  for (MoeGemmArgs* g : {&g1, &g2}) {
    g->slice_sizes = (int32_t*)(base + o_sum); g->slice_offs = offs;
    g->block_offs_16 = offs + lo; g->block_sched_16 = sched;
    g->ld_block_offs = lo; g->ld_block_sched = ls;
  }
  set_temp(g1, base + o_y, t1, ws1);
  set_temp(g2, base + o_tmp, t2, ws2);
  g1.gather_indx = (int32_t*)(base + o_tok);
  g1.x_positions = (int32_t*)(base + o_row); g1.x_experts = (int16_t*)(base + o_indx); g1.x_k = (int)k;
  if (limit) { g1.act_limit = (float)*limit; g1.act_has_limit = 1; }
  g1.y = base + o_h; g1.ld_y = ff;
  g2.x = base + o_h; g2.rows_x = n;
  g2.scatter_indx = (int32_t*)(base + o_col); g2.gammas = (float*)(base + o_gam);
  g2.y = base + o_y; g2.ld_y = d;
  check(lib.moe_grouped_gemm_chain(&g1, &g2, st), "moe_grouped_gemm", true);
  check(lib.moe_reduce(base + o_y, MOE_BF16, k, T, d, d, k * d, 1, nullptr, 0, 0, 0, 0, nullptr, 0, 0, 0, z.data_ptr(), MOE_BF16, d, 1, st),
        "moe_reduce");
  return z;
}

// ---- quantiser, combine --------------------------------------------------------------------------------------------
// [batch, outer, quant] element strides of `t` with its last axis quantised; false when the leading axes do not merge into two
bool collapse3(const Tensor& t, int64_t (&e)[2], int64_t (&s)[2]) {
  int m = 0;
  int64_t sz[2] = {1, 1}, st[2] = {0, 0};
  for (int64_t i = 0; i + 1 < t.dim(); ++i) {
    if (t.size(i) == 1) continue;
    if (m > 0 && st[m - 1] == t.stride(i) * t.size(i)) { sz[m - 1] *= t.size(i); st[m - 1] = t.stride(i); continue; }
    if (m == 2) return false;
    sz[m] = t.size(i); st[m] = t.stride(i); ++m;
  }
  for (int i = 0; i < 2; ++i) {          // missing axes go in front
    const int from = i - (2 - m);
    e[i] = from >= 0 ? sz[from] : 1; s[i] = from >= 0 ? st[from] : 0;
  }
  return true;
}

// the same for a copy when they do not merge (always contiguous, so they do then)
Tensor collapsed(const Tensor& t, int64_t (&e)[2], int64_t (&s)[2]) {
  if (collapse3(t, e, s)) return t;
  Tensor c = t.contiguous();
  collapse3(c, e, s);
  return c;
}

py::tuple downcast(const Tensor& x, int64_t axis, int mode) {
  need_cuda(x);
  const int code = dtype_code(x);
  Tensor xt = x.transpose(axis, -1);
  const int64_t L = x.size(axis);
  std::vector<int64_t> shape = xt.sizes().vec();
  shape.back() = L / 2;
  Tensor q = empty(shape, at::kByte, x);
  shape.back() = L / 32;
  Tensor s = empty(shape, at::kByte, x);
  if (x.numel() > 0) {
    int64_t e[2], st[2];
    xt = collapsed(xt, e, st);
    check(lib.moe_downcast_mxfp4(xt.data_ptr(), code, e[0], e[1], L, st[0], st[1], xt.stride(-1), q.data_ptr<uint8_t>(),
                                 s.data_ptr<uint8_t>(), mode, stream()),
          "moe_downcast_mxfp4");
  }
  return py::make_tuple(q.transpose(axis, -1), s.transpose(axis, -1));
}

Tensor upcast(const Tensor& q_, const Tensor& s_, py::object dtype, int64_t axis) {
  need_cuda(q_); need_cuda(s_);
  Tensor q = q_.transpose(axis, -1).contiguous(), s = s_.transpose(axis, -1).contiguous();
  const int64_t L = q.size(-1) * 2;
  if (s.size(-1) * 32 != L) raise(PyExc_AssertionError, "scale shape does not match the packed values");
  std::vector<int64_t> shape = q_.sizes().vec();
  shape[axis] = L;
  Tensor out = empty(shape, torch::python::detail::py_object_to_dtype(dtype), q_);
  if (out.numel() > 0) {
    int64_t e[2], st[2];
    Tensor ot = collapsed(out.transpose(axis, -1), e, st);
    check(lib.moe_upcast_mxfp4(q.data_ptr<uint8_t>(), s.data_ptr<uint8_t>(), ot.data_ptr(), dtype_code(out), e[0], e[1], L, st[0], st[1],
                               ot.stride(-1), stream()),
          "moe_upcast_mxfp4");
    if (ot.data_ptr() != out.data_ptr()) out.transpose(axis, -1).copy_(ot);
  }
  return out;
}

// sum over `dim` without mask or scale; y is the caller's output or None
Tensor reduce(const Tensor& x, int64_t dim, const OptTensor& y_, py::object y_dtype) {
  need_cuda(x);
  if (y_) need_cuda(*y_);
  const int64_t a = dim == 0 ? 1 : 0, b = dim == 2 ? 1 : 2;
  Tensor y = y_ ? *y_ : empty({x.size(a), x.size(b)}, torch::python::detail::py_object_to_dtype(y_dtype), x);
  if (y.numel() > 0)
    check(lib.moe_reduce(x.data_ptr(), dtype_code(x), x.size(dim), x.size(a), x.size(b), x.stride(dim), x.stride(a), x.stride(b), nullptr, 0,
                         0, 0, 0, nullptr, 0, 0, 0, y.data_ptr(), dtype_code(y), y.stride(0), y.stride(1), stream()),
          "moe_reduce");
  return y;
}

// ---- router --------------------------------------------------------------------------------------------------------
// -> vals, indx, bitmatrix view; wg in the kernel's memory order
py::tuple router(const Tensor& x, const Tensor& wg, const OptTensor& bg, int64_t k, bool softmax, bool round_bf16, const OptTensor& logits,
                 const Tensor& status) {
  need_cuda(x); need_cuda(wg);
  if (bg) need_cuda(*bg);
  const int64_t T = x.size(0), K = x.size(1), E = wg.size(1);
  Tensor vals = empty({T, k}, round_bf16 ? at::kBFloat16 : at::kFloat, x), indx = empty({T, k}, at::kShort, x);
  const int64_t t_pad = cdiv(T, 32) * 32, words = cdiv(E, 32);
  Tensor bm_all = empty({words, t_pad}, at::kInt, x), bm = part(bm_all, 0, {T, words}, {1, t_pad});
  if (T > 0)
    check(lib.moe_router_topk(x.data_ptr(), T, K, x.stride(0), wg.data_ptr(), wg.stride(1), bg ? bg->data_ptr() : nullptr,
                              bg ? dtype_code(*bg) : 0, (int)E, (int)k, softmax, round_bf16, logits ? logits->data_ptr<float>() : nullptr, E,
                              vals.data_ptr(), dtype_code(vals), k, indx.data_ptr<int16_t>(), k, (uint32_t*)bm.data_ptr(), bm.stride(0),
                              bm.stride(1), nullptr, 0, status.data_ptr<int32_t>(), stream()),
          "moe_router_topk");
  return py::make_tuple(vals, indx, bm);
}

// ---- inputs and result of a replayed step --------------------------------------------------------------------------
bool plain_copy(const Tensor& dst, const Tensor& src) {
  return src.is_cuda() && src.device() == dst.device() && src.scalar_type() == dst.scalar_type() && src.sizes() == dst.sizes() &&
         src.is_contiguous() && dst.is_contiguous() && (uintptr_t)src.data_ptr() % 16 == 0 && (uintptr_t)dst.data_ptr() % 16 == 0;
}

// src -> dst of both pairs: one launch where they are plain copies on the current device, else what copy_ does
void copy2(const Tensor& dst0, const Tensor& src0, const Tensor& dst1, const Tensor& src1) {
  if (plain_copy(dst0, src0) && plain_copy(dst1, src1) && dst0.device() == dst1.device() &&
      dst0.device().index() == c10::cuda::current_device()) {
    check(lib.moe_copy2(dst0.data_ptr(), src0.data_ptr(), (int64_t)src0.nbytes(), dst1.data_ptr(), src1.data_ptr(), (int64_t)src1.nbytes(),
                        stream()),
          "moe_copy2");
    return;
  }
  Tensor d0 = dst0, d1 = dst1;
  d0.copy_(src0, true);
  d1.copy_(src1, true);
}

Tensor copy_of(const Tensor& src) {
  if (!src.is_contiguous() || !src.is_cuda() || (uintptr_t)src.data_ptr() % 16 != 0 || src.device().index() != c10::cuda::current_device())
    return src.clone();
  Tensor out = at::empty(src.sizes(), src.options());
  check(lib.moe_copy2(out.data_ptr(), src.data_ptr(), (int64_t)src.nbytes(), nullptr, nullptr, 0, stream()), "moe_copy2");
  return out;
}

// A captured layer step with its copies (moe_step_graph_create): x and logits in, a new tensor out.  roots_wait: the first kernel of the
// captured step waits for the one before by itself.
class StepGraph {
 public:
  StepGraph(int64_t graph, bool roots_wait, const Tensor& x, const Tensor& logits, const Tensor& z) : x_(x), logits_(logits), z_(z) {
    check(lib.moe_step_graph_create(reinterpret_cast<void*>(graph), roots_wait, x.data_ptr(), (int64_t)x.nbytes(), logits.data_ptr(), (int64_t)logits.nbytes(),
                                    z.data_ptr(), (int64_t)z.nbytes(), &step_),
          "moe_step_graph_create");
  }
  ~StepGraph() { lib.moe_step_graph_destroy(step_); }
  StepGraph(const StepGraph&) = delete;
  StepGraph& operator=(const StepGraph&) = delete;
  // None where the inputs are not plain copies of the step's on the current device, or the stream is being captured
  std::optional<Tensor> run(const Tensor& x, const Tensor& logits) {
    if (!plain_copy(x_, x) || !plain_copy(logits_, logits) || x_.device().index() != c10::cuda::current_device() ||
        c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None)
      return std::nullopt;
    Tensor out = at::empty(z_.sizes(), z_.options());
    check(lib.moe_step_graph_launch(step_, x.data_ptr(), logits.data_ptr(), out.data_ptr(), stream()), "moe_step_graph_launch");
    return out;
  }

 private:
  Tensor x_, logits_, z_;
  void* step_ = nullptr;
};

}  // namespace

PYBIND11_MODULE(_host, m) {
  py::class_<StepGraph>(m, "StepGraph").def(py::init<int64_t, bool, const Tensor&, const Tensor&, const Tensor&>()).def("run", &StepGraph::run);
  m.def("copy2", &copy2);
  m.def("copy_of", &copy_of);
  m.def("bind", &bind);
  m.def("route", &route);
  m.def("bitmatrix_metadata", &bitmatrix_metadata);
  m.def("gemm", &gemm);
  m.def("gemm_kernel", &gemm_kernel, py::arg("kind"), py::arg("E"), py::arg("K"), py::arg("N"), py::arg("M"), py::arg("x_dtype"),
        py::arg("y_dtype"), py::arg("tuning"), py::arg("rows_per_expert") = 0, py::arg("swiglu") = false);
  m.def("layer", &layer);
  m.def("downcast", &downcast);
  m.def("upcast", &upcast);
  m.def("reduce", &reduce);
  m.def("router", &router);
}
