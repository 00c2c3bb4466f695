"""Performance cases: what a user of this package has it do, through its public entry points.

`listed()` names the cases that stand for the work, `draw(rng)` picks further ones from the same ranges, `prepare` makes
what a program holds before the call (inputs, quantised weights, a captured graph), `run` is one pass through the public
API, `work` the bytes and operations the pass cannot do without, `tolerance` what another correct implementation may
differ by.

Kinds
  layer     one MoE layer step (routing, fc1 + SwiGLU, fc2 x routing weight, combine).  `api`:
              "graph"      `GraphedMoeLayer`, the decode path: a step captured once per token count, called with new inputs
              "eager"      `moe_layer_forward`
              "operators"  the layer composed from `routing`, `matmul`, `matmul`, `reduce`, weights in the default layouts
                           (how a program written against the operators runs it)
            `dtype` "bf16", or "e4m3" for fp8 tokens
  router    `router_topk`: router product fused with the top-k selection
  routing   `routing`: top-k of given logits, expert sort, ragged metadata
  quantise  `downcast_to_mxfp` of a matrix and `upcast_from_mxfp` of the result
  weights   load-time preparation of expert weights: quantise along K, default and block-scaled layouts"""
import torch

import triton_b200 as tb
from triton_b200.moe import GraphedMoeLayer, moe_layer_forward
from triton_b200.tensor_details.layout import (B200BlockScaledScaleLayout, B200BlockScaledValueLayout,
                                               make_default_matmul_mxfp4_w_layout, make_default_matmul_mxfp4_w_scale_layout)
from triton_b200.testing import make_synthetic_layer

DEV = "cuda"
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
GRAPH_MAX_TOKENS = 1024               # decode-sized steps are replayed, larger ones run eagerly


def _layer(name, tokens, experts, top_k, d_model, d_ff, api, dtype="bf16", skew=True):
    return {"name": name, "kind": "layer", "tokens": tokens, "experts": experts, "top_k": top_k, "d_model": d_model,
            "d_ff": d_ff, "api": api, "dtype": dtype, "skew": skew}


def listed():
    return [
        # decode of a single stream: four experts of 128 are read, launches and latency count
        _layer("decode 1 token", 1, 128, 4, 2880, 2880, "graph"),
        # decode of a serving batch: the step streams the weights of about half the experts
        _layer("decode 64 tokens", 64, 128, 4, 2880, 2880, "graph"),
        # a decode-sized step of a program that captures no graph
        _layer("step 16 tokens eager", 16, 32, 4, 2880, 2880, "eager"),
        # a small model: every launch is short
        _layer("small layer 256 tokens", 256, 8, 2, 512, 1024, "eager", skew=False),
        # a ragged mid-sized batch (mixed decode and short prompts): nine rows per expert on average
        _layer("mixed batch 300 tokens", 300, 128, 4, 2880, 2880, "eager"),
        # a program written against the operators, prompt-sized, 150 rows per expert on average
        _layer("operators 1200 tokens", 1200, 32, 4, 2880, 2880, "operators"),
        # prefill: the largest step
        _layer("prefill 16384 tokens", 16384, 128, 4, 2880, 2880, "eager"),
        # prefill with fp8 tokens in and between the two products
        _layer("prefill 8192 tokens fp8", 8192, 32, 4, 2880, 2880, "eager", dtype="e4m3"),
        # the router of a prompt batch
        {"name": "router 4100 tokens", "kind": "router", "tokens": 4100, "d_model": 2880, "experts": 128, "top_k": 4},
        # routing of given logits at prefill size
        {"name": "routing 16384 tokens", "kind": "routing", "tokens": 16384, "experts": 128, "top_k": 4},
        # quantise a matrix with outliers and read it back
        {"name": "quantise 8192 x 8192", "kind": "quantise", "rows": 8192, "cols": 8192, "axis": 1, "dtype": "bf16"},
        # load time: expert weights of a gate + up projection, quantised along K (strided) and laid out
        {"name": "weights 16 x 2880 x 5760", "kind": "weights", "experts": 16, "k": 2880, "n": 5760},
    ]


MAX_LAYER_WORK = 16384 * 4 * 2880 * 2880           # tokens x top_k x d_model x d_ff of the largest listed step
MAX_LAYER_WORK_FP8 = 8192 * 4 * 2880 * 2880
MAX_WEIGHTS = 128 * 2880 * 2880


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(lo * (hi / lo) ** rng.random())))


def draw(rng):
    kind = rng.choices(["layer", "router", "routing", "quantise", "weights"], weights=[60, 8, 12, 12, 8])[0]
    if kind == "layer":
        experts = rng.choice([8, 16, 32, 64, 128])
        top_k = rng.choice([1, 2, 4, 4, 8])
        sizes = [512, 736, 1024, 1440, 2048, 2880, 2880, 2880, 4096]
        d_model, d_ff = rng.choice(sizes), rng.choice(sizes)
        while experts * d_model * d_ff > MAX_WEIGHTS:
            experts //= 2
        dtype = rng.choices(["bf16", "e4m3"], weights=[5, 1])[0]
        cap = (MAX_LAYER_WORK if dtype == "bf16" else MAX_LAYER_WORK_FP8) // (top_k * d_model * d_ff)
        tokens = _log_int(rng, 1, min(16384, cap))
        apis = ["eager"]
        if dtype == "bf16":
            apis.append("operators")
            if tokens <= GRAPH_MAX_TOKENS:
                apis += ["graph", "graph"]
        return _layer("", tokens, experts, top_k, d_model, d_ff, rng.choice(apis), dtype, skew=rng.random() < 0.75)
    if kind == "router":
        return {"kind": kind, "tokens": _log_int(rng, 1, 16384), "d_model": rng.choice([512, 736, 1024, 1440, 2048, 2880, 4096]),
                "experts": rng.choice([8, 16, 32, 64, 100, 128, 256]), "top_k": rng.choice([1, 2, 4, 8])}
    if kind == "routing":
        experts = rng.choice([8, 16, 32, 60, 64, 100, 128, 200, 256])
        return {"kind": kind, "tokens": _log_int(rng, 1, 32768), "experts": experts, "top_k": rng.choice([1, 2, 4, 4, 6, 8])}
    if kind == "quantise":
        cols = 32 * _log_int(rng, 1, 512)
        return {"kind": kind, "rows": 32 * _log_int(rng, 1, min(512, 8192 * 8192 // (32 * cols))), "cols": cols,
                "axis": rng.choice([0, 1]), "dtype": rng.choices(["bf16", "fp16", "fp32"], weights=[4, 1, 1])[0]}
    k, n = rng.choice([512, 736, 1024, 1440, 2048, 2880]), rng.choice([512, 1024, 1472, 2048, 2880, 5760])
    return {"kind": kind, "experts": rng.randint(1, max(1, 16 * 2880 * 5760 // (k * n) if k * n > 2880 * 2880 else 32)), "k": k, "n": n}


# ---------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return {"layer": _prepare_layer, "router": _prepare_router, "routing": _prepare_routing, "quantise": _prepare_quantise,
            "weights": _prepare_weights}[case["kind"]](case, seed, g)


def run(state):
    return state["run"](state)


def _tokens(T, d, g):
    return torch.randn(T, d, device=DEV, generator=g).bfloat16()


def _logits(case, g):
    """Router logits N(0,1); skewed: plus a per-expert bias N(0,1), so that experts get very different row counts."""
    logits = torch.randn(case["tokens"], case["experts"], device=DEV, generator=g)
    return logits + torch.randn(case["experts"], device=DEV, generator=g) if case.get("skew", True) else logits


def _prepare_layer(case, seed, g):
    T, E, k, d = case["tokens"], case["experts"], case["top_k"], case["d_model"]
    operators = case["api"] == "operators"
    lw = make_synthetic_layer(E, d, case["d_ff"], torch.device(DEV), seed=seed, block_scaled=not operators)
    x, logits = _tokens(T, d, g), _logits(case, g)
    if case["dtype"] == "e4m3":
        x = x.to(torch.float8_e4m3fn)
    state = {"x": x, "logits": logits, "lw": lw, "k": k}
    if case["api"] == "graph":
        state.update(run=_run_graph, layer=GraphedMoeLayer(lw, k, T, d, E, torch.device(DEV)))
    elif operators:
        state.update(run=_run_operators, pc1=tb.PrecisionConfig(b_mx_scale=lw.w1_scale, b_microblock_size=32),
                     pc2=tb.PrecisionConfig(b_mx_scale=lw.w2_scale, b_microblock_size=32),
                     act=tb.FusedActivation(tb.FnSpecs("swiglu", tb.swiglu_fn, ("alpha", "limit"), reduction_n=2),
                                            (lw.alpha, lw.limit)))
    else:
        state.update(run=_run_eager)
    return state


def _run_graph(s):
    return s["layer"](s["x"], s["logits"])


def _run_eager(s):
    return moe_layer_forward(s["x"], s["logits"], s["lw"], s["k"])


def _run_operators(s):
    x, lw, k = s["x"], s["lw"], s["k"]
    ragged, gather_idx, scatter_idx, sparse = tb.routing(s["logits"], k)
    gammas = sparse.vals.reshape(-1)[scatter_idx]
    h = tb.matmul(x, lw.w1, lw.b1, ragged, gather_indx=gather_idx, precision_config=s["pc1"], fused_activation=s["act"])
    y = tb.matmul(h, lw.w2, lw.b2, ragged, scatter_indx=scatter_idx, precision_config=s["pc2"], gammas=gammas)
    z, _ = tb.reduce(y.view(x.shape[0], k, -1), dim=1)
    return z


def _prepare_router(case, seed, g):
    d, E = case["d_model"], case["experts"]
    wg = tb.prepare_router_weight((torch.randn(d, E, device=DEV, generator=g) / d ** 0.5).bfloat16())
    return {"run": _run_router, "x": _tokens(case["tokens"], d, g), "wg": wg, "k": case["top_k"],
            "bg": torch.randn(E, device=DEV, generator=g)}


def _run_router(s):
    sp = tb.router_topk(s["x"], s["wg"], s["bg"], s["k"])
    # The expert sort of `mask_metadata` runs in this call too and shows in `col_sum`.  Its permutations are left to the
    # routing case: logits are rounded to bf16, so two correct sums may order a tie differently, and one such token shifts
    # every later position of the sort.
    return {"vals": sp.vals, "indx": sp.indx, "mask": sp.mask.storage.data, "col_sum": sp.mask_metadata.col_sum}


def _prepare_routing(case, seed, g):
    return {"run": _run_routing, "logits": _logits(case, g), "k": case["top_k"]}


def _run_routing(s):
    ragged, gather_idx, scatter_idx, sp = tb.routing(s["logits"], s["k"])
    return {"vals": sp.vals, "indx": sp.indx, "mask": sp.mask.storage.data, "gather": gather_idx, "scatter": scatter_idx,
            "row_sorted": sp.mask_metadata.row_sorted_indx, "col_sum": sp.mask_metadata.col_sum, "slice_offs": ragged.slice_offs,
            "block_offs": ragged.block_offs_data, "block_schedule": ragged.block_schedule_data}


def _prepare_quantise(case, seed, g):
    shape = (case["rows"], case["cols"])
    x = torch.randn(shape, device=DEV, generator=g)
    x = torch.where(torch.rand(shape, device=DEV, generator=g) < 0.01, x * 100, x)          # 1 % outliers
    return {"run": _run_quantise, "x": x.to(DTYPES[case["dtype"]]), "axis": case["axis"]}


def _run_quantise(s):
    q, scale = tb.downcast_to_mxfp(s["x"], torch.uint8, axis=s["axis"])
    return {"q": q, "scale": scale, "back": tb.upcast_from_mxfp(q, scale, s["x"].dtype, axis=s["axis"])}


def _prepare_weights(case, seed, g):
    w = torch.empty((case["experts"], case["k"], case["n"]), dtype=torch.bfloat16, device=DEV)
    for e in range(case["experts"]):
        w[e] = torch.randn(case["k"], case["n"], device=DEV, generator=g) * 0.02
    return {"run": _run_weights, "w": w}


def _run_weights(s):
    q, scale = tb.downcast_to_mxfp(s["w"], torch.uint8, axis=1)
    tq, ts = tb.wrap_torch_tensor(q, dtype=tb.FP4), tb.wrap_torch_tensor(scale)
    made = (tb.convert_layout(tq, make_default_matmul_mxfp4_w_layout(mx_axis=-2)),
            tb.convert_layout(ts, make_default_matmul_mxfp4_w_scale_layout(mx_axis=-2)),
            tb.convert_layout(tq, B200BlockScaledValueLayout()), tb.convert_layout(ts, B200BlockScaledScaleLayout()))
    return [t.storage.data for t in made]


# ---------------------------------------------------------------------------------------------------------
def _active_experts(case):
    """Experts that get at least one row, from one simulated batch (skewed routing leaves many idle at decode sizes)."""
    T, E, k = case["tokens"], case["experts"], case["top_k"]
    g = torch.Generator().manual_seed(0)
    logits = torch.randn(T, E, generator=g) + (torch.randn(E, generator=g) if case["skew"] else 0)
    return int(logits.topk(k, dim=1).indices.unique().numel())


def work(case):
    kind = case["kind"]
    if kind == "layer":
        T, E, k, d, ff = (case[n] for n in ("tokens", "experts", "top_k", "d_model", "d_ff"))
        per_expert = 3 * d * ff // 2 + 3 * d * ff // 32 + (2 * ff + d) * 2          # packed values, scales, biases
        nbytes = _active_experts(case) * per_expert + T * d * (1 if case["dtype"] == "e4m3" else 2) + T * E * 4 + T * d * 2
        return {"bytes": nbytes, "flops": 6 * T * k * d * ff}
    if kind == "router":
        T, d, E, k = (case[n] for n in ("tokens", "d_model", "experts", "top_k"))
        return {"bytes": T * d * 2 + d * E * 2 + T * k * (2 + 2) + T * ((E + 31) // 32) * 4 + 2 * T * k * 4, "flops": 2 * T * d * E}
    if kind == "routing":
        T, E, k = (case[n] for n in ("tokens", "experts", "top_k"))
        # logits in; values, indices, bitmatrix, gather / scatter / row-sorted indices and the schedules out
        return {"bytes": T * E * 4 + T * k * (4 + 2) + T * ((E + 31) // 32) * 4 + 3 * T * k * 4 + 4 * (E + T * k // 16) * 4, "flops": 0}
    if kind == "quantise":
        n, size = case["rows"] * case["cols"], {"bf16": 2, "fp16": 2, "fp32": 4}[case["dtype"]]
        return {"bytes": 2 * n * size + 2 * (n // 2 + n // 32), "flops": 0}
    n = case["experts"] * case["k"] * case["n"]
    return {"bytes": 2 * n + 2 * (n // 2 + n // 32), "flops": 0}       # bf16 in; two packed forms with their scales out


def tolerance(case):
    kind = case["kind"]
    if kind == "layer":
        return {"rel": 1e-2}                     # bf16 outputs of bf16 (or e4m3) products with fp32 sums
    if kind == "router":
        return {"rel": 1e-2, "differ": 1e-2}     # bf16 values; ties of bf16-rounded logits
    if kind == "routing":
        return {"rel": 1e-5, "differ": 0.0}      # fp32 softmax over the selected logits; whole numbers are the same
    return "exact"
