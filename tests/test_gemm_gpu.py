"""Ragged grouped GEMM on the GPU against the CPU oracle: the SIMT kernel (canonical / dense weights) and
the tcgen05 kernel (B200 tiled weights), with gather, scatter, bias, betas / gammas, SwiGLU."""
import pytest
import torch

import oracle
import triton_b200 as tb
from triton_b200.tensor import FP4, convert_layout, wrap_torch_tensor
from triton_b200.tensor_details.layout import (B200MXScaleLayout, B200MXValueLayout, BlackwellMXScaleLayout,
                                               BlackwellMXValueLayout)

pytestmark = pytest.mark.gpu

# tolerance of the reference's tests for MXFP4 weights: tests/test_matmul.py:649-650 (max 3e-2, rms unchecked);
# in addition the relative L2 error must stay below 1e-2
MAXTOL_MX4 = 3e-2


def make_problem(E, K, N, sizes, T, seed, device, act=False, gather=True, scatter=False, bias=True, weights=False,
                 w_std=0.02):
    g = torch.Generator().manual_seed(seed)
    sizes = torch.tensor(sizes, dtype=torch.int32)
    M = int(sizes.sum())
    x = torch.randn(T if gather else M, K, generator=g).bfloat16()
    w = (torch.randn(E, K, N, generator=g) * w_std).bfloat16()
    wq, ws = oracle.downcast_to_mxfp_oracle(w, 1)
    wq, ws = wq.contiguous().transpose(1, 2).contiguous().transpose(1, 2), ws.contiguous().transpose(1, 2).contiguous().transpose(1, 2)
    p = dict(E=E, K=K, N=N, M=M, sizes=sizes, x=x, wq=wq, ws=ws)
    p["bias"] = torch.randn(E, N, generator=g) * 0.1 if bias else None
    p["gather"] = torch.randint(0, T, (M,), generator=g, dtype=torch.int32) if gather else None
    p["scatter"] = torch.randperm(M, generator=g).int() if scatter else None
    p["gammas"] = torch.rand(M, generator=g) if weights else None
    p["betas"] = torch.rand(M, generator=g) if weights else None
    p["act"] = (1.702, 7.0) if act else None
    p["wdeq"] = oracle.dequant_weight_oracle(wq, ws)
    return p


def reference(p, fp32_act=True):
    y = oracle.matmul_oracle(p["x"], p["wdeq"], p["bias"], p["sizes"], p["gather"], None, betas=p["betas"],
                             gammas=None if p["act"] else p["gammas"], out_dtype=torch.float32)
    if p["act"]:
        y = oracle.swiglu_oracle(y, *p["act"])
        if p["gammas"] is not None:
            y = y * p["gammas"][:, None]
    y = y.bfloat16()
    if p["scatter"] is not None:
        out = torch.zeros_like(y)
        out[p["scatter"].long()] = y
        y = out
    return y


def run(p, device, layout, kernel="auto", block_m=None, block_n=None):
    dev = lambda t: None if t is None else t.to(device)
    wq = wrap_torch_tensor(dev(p["wq"]), dtype=FP4)
    ws = wrap_torch_tensor(dev(p["ws"]))
    assert wq.shape == [p["E"], p["K"], p["N"]]
    if layout == "b200":
        wq, ws = convert_layout(wq, B200MXValueLayout()), convert_layout(ws, B200MXScaleLayout())
    elif layout == "blackwell":
        wq, ws = convert_layout(wq, BlackwellMXValueLayout()), convert_layout(ws, BlackwellMXScaleLayout())
    md = tb.make_ragged_tensor_metadata(dev(p["sizes"]), p["M"])
    pc = tb.PrecisionConfig(b_mx_scale=ws, b_microblock_size=32)
    fa = None
    if p["act"]:
        fa = tb.FusedActivation(tb.FnSpecs("swiglu", tb.swiglu_fn, ("alpha", "limit"), reduction_n=2), p["act"])
    cons = {"kernel": kernel}
    if block_m:
        cons["block_m"] = block_m
    if block_n:
        cons["block_n"] = block_n
    with tb.scoped_opt_flags_constraints(cons):
        y = tb.matmul(dev(p["x"]), wq, dev(p["bias"]), md, None, dev(p["gather"]), dev(p["scatter"]), pc,
                      betas=dev(p["betas"]), gammas=dev(p["gammas"]), fused_activation=fa)
    tb.matmul_check_status()
    return y


def check(p, y, scatter_valid=None):
    ref = reference(p)
    got = y.cpu()
    if p["scatter"] is None:
        n = p["M"]
        ref, got = ref[:n], got[:n]
    oracle.assert_close_oracle(ref, got, maxtol=MAXTOL_MX4, rmstol=None, what="gemm")
    assert oracle.rel_l2(ref, got) < 1e-2


SMALL = [
    # E, K, N, sizes, T
    (4, 96, 64, [13, 0, 29, 8], 50),
    (1, 64, 32, [5], 9),
    (3, 512, 256, [130, 1, 64], 200),
    (8, 2880, 384, [0, 17, 128, 129, 3, 0, 64, 255], 300),
    (5, 320, 128, [600, 256, 257, 0, 511], 700),
]


@pytest.mark.parametrize("case", SMALL)
@pytest.mark.parametrize("mode", ["plain", "gather", "scatter_w", "swiglu", "all"])
@pytest.mark.parametrize("path", ["simt-canonical", "simt-blackwell", "tcgen05", "tcgen05-256", "tcgen05-256x256", "tcgen05-pair", "stream"])
def test_grouped_gemm(case, mode, path, device):
    E, K, N, sizes, T = case
    opts = dict(plain=dict(gather=False), gather=dict(gather=True),
                scatter_w=dict(gather=True, scatter=True, weights=True), swiglu=dict(gather=True, act=True),
                all=dict(gather=True, scatter=True, weights=True, act=True))[mode]
    p = make_problem(E, K, N, sizes, T, seed=hash((E, K, N, mode)) % 1000, device=device, **opts)
    layout, kernel, block_m, block_n = {
        "simt-canonical": ("canonical", "simt", None, None), "simt-blackwell": ("blackwell", "simt", None, None),
        "tcgen05": ("b200", "tcgen05", 128, 128), "tcgen05-256": ("b200", "tcgen05", 256, 128),
        "tcgen05-256x256": ("b200", "tcgen05", 256, 256), "tcgen05-pair": ("b200", "tcgen05-pair", 0, 0), "stream": ("b200", "stream", 0, 0)}[path]
    y = run(p, device, layout, kernel, block_m, block_n)
    check(p, y)


@pytest.mark.parametrize("kernel", ["tcgen05", "tcgen05-pair"])
@pytest.mark.parametrize("mode", ["gather", "all"])
def test_grouped_gemm_pregathered_rows(kernel, mode, device):
    """2048+ gathered rows with large experts: the rows are first copied into the scratch buffer the host passes and
    the kernel streams them by TMA tile copies."""
    opts = dict(gather=dict(gather=True), all=dict(gather=True, scatter=True, weights=True, act=True))[mode]
    p = make_problem(4, 320, 256, [900, 700, 385, 127], 800, seed=11, device=device, **opts)
    y = run(p, device, "b200", kernel, 0, 0)
    check(p, y)


@pytest.mark.parametrize("kernel", ["simt", "tcgen05"])
@pytest.mark.parametrize("sizes, T", [([13, 0, 29, 8], 50), ([600, 256, 257, 511], 700)])
def test_fused_comm_block_rows(kernel, sizes, T, device):
    """Output rows spread over three buffers (here all on one device): row r of the scattered output lands in row
    r % rows_per_shard of buffer r // rows_per_shard."""
    p = make_problem(4, 320, 128, sizes, T, seed=5, device=device, gather=True, scatter=True, weights=True)
    M = p["M"]
    shards = 3
    rows_per_shard = (M + shards - 1) // shards
    bufs = [torch.zeros(rows_per_shard, 128, dtype=torch.bfloat16, device=device) for _ in range(shards)]
    dev = lambda t: None if t is None else t.to(device)
    layout = "canonical" if kernel == "simt" else "b200"
    wq = wrap_torch_tensor(dev(p["wq"]), dtype=FP4)
    ws = wrap_torch_tensor(dev(p["ws"]))
    if layout == "b200":
        wq, ws = convert_layout(wq, B200MXValueLayout()), convert_layout(ws, B200MXScaleLayout())
    md = tb.make_ragged_tensor_metadata(dev(p["sizes"]), M)
    pc = tb.PrecisionConfig(b_mx_scale=ws, b_microblock_size=32)
    fc = tb.FusedComm([b.data_ptr() for b in bufs], rows_per_shard, bufs[0])
    with tb.scoped_opt_flags_constraints({"kernel": kernel}):
        y0 = tb.matmul(dev(p["x"]), wq, dev(p["bias"]), md, None, dev(p["gather"]), dev(p["scatter"]), pc,
                       betas=dev(p["betas"]), gammas=dev(p["gammas"]), fused_comm=fc)
    tb.matmul_check_status()
    assert y0.data_ptr() == bufs[0].data_ptr()
    y = torch.cat(bufs)[:M]
    check(p, y)


def test_against_reference_fixture(golden, device):
    g = golden("gemm_small")
    wq = wrap_torch_tensor(g["wq"].to(device).transpose(1, 2).contiguous().transpose(1, 2), dtype=FP4)
    ws = wrap_torch_tensor(g["ws"].to(device).transpose(1, 2).contiguous().transpose(1, 2))
    md = tb.make_ragged_tensor_metadata(g["slice_sizes"].to(device), 50)
    for layout in ("canonical", "b200"):
        wq2, ws2 = wq, ws
        if layout == "b200":
            wq2, ws2 = convert_layout(wq, B200MXValueLayout()), convert_layout(ws, B200MXScaleLayout())
        pc = tb.PrecisionConfig(b_mx_scale=ws2, b_microblock_size=32)
        y = tb.matmul(g["x"].to(device), wq2, g["bias"].to(device), md, None, g["gather"].to(device),
                      g["scatter"].to(device), pc, gammas=g["gammas"].to(device))
        tb.matmul_check_status()
        oracle.assert_close_oracle(g["y"], y.cpu(), maxtol=MAXTOL_MX4, rmstol=None, what=layout)


def test_dense_plain_product_library_gemm(device):
    """x @ W + b without routing (the router's logits) goes to the library GEMM; same answer as the SIMT kernel."""
    torch.manual_seed(1)
    x = torch.randn(300, 2880, device=device).bfloat16()
    w = (torch.randn(2880, 128, device=device) * 0.02).bfloat16()
    b = torch.randn(128, device=device)
    y = tb.matmul(x, w, b)
    with tb.scoped_opt_flags_constraints({"kernel": "simt"}):
        y_simt = tb.matmul(x, w, b)
    ref = (x.float().cpu() @ w.float().cpu() + b.cpu()).bfloat16()
    oracle.assert_close_oracle(ref, y.cpu())
    oracle.assert_close_oracle(ref, y_simt.cpu())


def test_dense_weights_simt(device):
    torch.manual_seed(0)
    x = torch.randn(70, 100, device=device).bfloat16()
    w = (torch.randn(100, 48, device=device) * 0.1).bfloat16()
    b = torch.randn(48, device=device)
    y = tb.matmul(x, w, b)
    ref = (x.float().cpu() @ w.float().cpu() + b.cpu()).bfloat16()
    oracle.assert_close_oracle(ref, y.cpu())


def test_weight_layout_round_trip(device):
    torch.manual_seed(0)
    E, K, N = 3, 2880, 200
    q = torch.randint(0, 256, (E, K, N // 2), dtype=torch.uint8, device=device)      # canonical, packed along N
    s = torch.randint(0, 255, (E, K // 32, N), dtype=torch.uint8, device=device)
    tq, ts = wrap_torch_tensor(q, dtype=FP4), wrap_torch_tensor(s)
    assert tq.shape == [E, K, N]
    bq, bs = convert_layout(tq, B200MXValueLayout()), convert_layout(ts, B200MXScaleLayout())
    lib = tb._lib.load()
    assert bq.storage.data.numel() == lib.moe_weight_b200_value_bytes(E, K, N)
    assert bs.storage.data.numel() == lib.moe_weight_b200_scale_bytes(E, K, N)
    from triton_b200.tensor_details.layout import StridedLayout
    assert torch.equal(convert_layout(bq, StridedLayout()).storage.data, q)
    assert torch.equal(convert_layout(bs, StridedLayout()).storage.data, s)
    # through the reference's Blackwell layouts and back
    vq = convert_layout(tq, BlackwellMXValueLayout())
    assert torch.equal(convert_layout(convert_layout(vq, B200MXValueLayout()), StridedLayout()).storage.data, q)
    g_s = oracle.swizzle_mx_scale_bw_oracle(s.cpu())
    assert torch.equal(convert_layout(ts, BlackwellMXScaleLayout()).storage.data.cpu(), g_s)


@pytest.mark.parametrize("E, K, N", [(1, 32, 2), (2, 2880, 200), (3, 160, 130)])
def test_weight_layouts_from_strided_storage(E, K, N, device):
    """The tiled layouts written straight from K-packed storage (rows 16-byte aligned, and a pitch that is not) equal those
    made through the canonical row-major form."""
    from triton_b200.tensor_details.layout import B200BlockScaledScaleLayout, B200BlockScaledValueLayout, StridedLayout
    g = torch.Generator(device=device).manual_seed(K + N)
    for pitch in (K // 2, K // 2 + 4):
        q = torch.randint(0, 256, (E, N, pitch), dtype=torch.uint8, device=device, generator=g)[:, :, : K // 2].transpose(1, 2)
        s = torch.randint(0, 255, (E, N, K // 32), dtype=torch.uint8, device=device, generator=g).transpose(1, 2)
        tq, ts = wrap_torch_tensor(q, dtype=FP4), wrap_torch_tensor(s)
        rq, rs = convert_layout(tq, StridedLayout()), convert_layout(ts, StridedLayout())
        for t, r, layouts in ((tq, rq, (B200MXValueLayout(), B200BlockScaledValueLayout())),
                              (ts, rs, (B200MXScaleLayout(), B200BlockScaledScaleLayout()))):
            for lay in layouts:
                via = lay.make_transformation(list(r.shape), r.dtype == FP4).swizzle_data(r.storage.data)
                assert torch.equal(convert_layout(t, lay).storage.data, via)


@pytest.fixture(scope="module")
def layer_20b():
    """gpt-oss-20b-shaped expert weights (32 experts, d_model 2880, fused gate+up 5760) and their CPU dequantisation."""
    from triton_b200.testing import make_synthetic_layer
    lw = make_synthetic_layer(32, 2880, 2880, "cuda", seed=0, keep_canonical=True)
    w1 = oracle.dequant_weight_oracle(lw.w1_q.cpu(), lw.w1_s.cpu())
    w2 = oracle.dequant_weight_oracle(lw.w2_q.cpu(), lw.w2_s.cpu())
    return lw, w1, w2


@pytest.mark.parametrize("tokens", [1, 16, 64, 512])
def test_gpt_oss_20b_layer_against_oracle(tokens, layer_20b, device):
    """One gpt-oss-20b-shaped MoE layer (top-4, SwiGLU alpha 1.702 limit 7) against the oracle, at the token
    counts the oracle finishes in seconds."""
    from triton_b200.moe import moe_layer_forward
    lw, w1, w2 = layer_20b
    torch.manual_seed(tokens)
    x = torch.randn(tokens, 2880, device=device).bfloat16()
    logits = torch.randn(tokens, 32, device=device)
    z = moe_layer_forward(x, logits, lw, 4)
    tb.matmul_check_status()
    ref = oracle.moe_layer_oracle(x.cpu(), logits.cpu(), w1, lw.b1.cpu(), w2, lw.b2.cpu(), 4, 1.702, 7.0,
                                  fuse_activation_fp32=True)
    oracle.assert_close_oracle(ref, z.cpu(), maxtol=MAXTOL_MX4, rmstol=None, what=f"layer T={tokens}")
    assert oracle.rel_l2(ref, z.cpu()) < 1e-2


@pytest.mark.parametrize("tokens", [4096, 16384])
def test_gpt_oss_20b_layer_full_size_properties(tokens, layer_20b, device):
    """Full-size token counts, checked through properties that need no CPU GEMM: (1) the tensor-core kernel and
    the SIMT kernel (canonical weights) agree; (2) a token's output does not depend on which other tokens are in
    the batch (rows of a sub-batch reproduce bit-for-bit... up to accumulation order: within tolerance)."""
    from triton_b200.moe import moe_layer_forward, MoeLayerWeights
    lw, _, _ = layer_20b
    torch.manual_seed(tokens)
    x = torch.randn(tokens, 2880, device=device).bfloat16()
    logits = torch.randn(tokens, 32, device=device)
    z = moe_layer_forward(x, logits, lw, 4)
    tb.matmul_check_status()
    sub = torch.arange(0, tokens, 37, device=device)[:256]
    lw_c = MoeLayerWeights(wrap_torch_tensor(lw.w1_q, dtype=FP4), wrap_torch_tensor(lw.w1_s), lw.b1,
                           wrap_torch_tensor(lw.w2_q, dtype=FP4), wrap_torch_tensor(lw.w2_s), lw.b2)
    with tb.scoped_opt_flags_constraints({"kernel": "simt"}):
        z_sub = moe_layer_forward(x[sub].contiguous(), logits[sub].contiguous(), lw_c, 4)
    oracle.assert_close_oracle(z_sub.cpu(), z[sub].cpu(), maxtol=MAXTOL_MX4, rmstol=None, what="tcgen05 vs simt")
    assert oracle.rel_l2(z_sub.cpu(), z[sub].cpu()) < 1e-2
    assert torch.isfinite(z.float()).all()


@pytest.mark.parametrize("tokens", [4, 64])
def test_graphed_layer_equals_eager_layer(tokens, layer_20b, device):
    """The layer replayed from a CUDA graph returns exactly what the eager layer returns, for new inputs too."""
    from triton_b200.moe import GraphedMoeLayer, moe_layer_forward
    lw, _, _ = layer_20b
    graphed = GraphedMoeLayer(lw, 4, tokens, 2880, 32, device)
    for seed in (1, 2):
        g = torch.Generator(device=device).manual_seed(seed)
        x = torch.randn(tokens, 2880, device=device, generator=g).bfloat16()
        logits = torch.randn(tokens, 32, device=device, generator=g)
        want = moe_layer_forward(x, logits, lw, 4)
        got = graphed(x, logits).clone()
        tb.matmul_check_status()
        assert torch.equal(want, got)


@pytest.mark.parametrize("form", ["plain", "strided x", "offset x", "other types"])
def test_graphed_layer_takes_inputs_of_any_layout(form, layer_20b, device):
    """Inputs that the step's own copies do not take (strides, alignment, types) are copied ahead of the replay; either way the
    step's buffers hold the call's inputs and result afterwards, and an earlier result stays as it is."""
    from triton_b200.moe import GraphedMoeLayer, moe_layer_forward
    lw, _, _ = layer_20b
    T = 5
    graphed = GraphedMoeLayer(lw, 4, T, 2880, 32, device)
    g = torch.Generator(device=device).manual_seed(3)
    first = graphed(torch.randn(T, 2880, device=device, generator=g).bfloat16(), torch.randn(T, 32, device=device, generator=g))
    kept = first.clone()
    x, logits = torch.randn(T, 2880, device=device, generator=g).bfloat16(), torch.randn(T, 32, device=device, generator=g)
    xi, li = x, logits
    if form == "strided x":
        xi = torch.zeros(T, 2 * 2880, device=device, dtype=torch.bfloat16)[:, :2880].copy_(x)
    elif form == "offset x":
        xi = torch.zeros(T * 2880 + 1, device=device, dtype=torch.bfloat16)[1:].view(T, 2880).copy_(x)
    elif form == "other types":
        xi, li = x.float(), logits.double()
    got = graphed(xi, li)
    assert torch.equal(got, moe_layer_forward(x, logits, lw, 4)) and torch.equal(first, kept)
    assert torch.equal(graphed.x, x) and torch.equal(graphed.logits, logits) and torch.equal(graphed.z, got)
    graphed.z.zero_()
    assert torch.equal(graphed.replay(), got) and got.data_ptr() != graphed.z.data_ptr()
    with pytest.raises(RuntimeError):
        graphed(x[:4], logits[:4])
    tb.matmul_check_status()


# routing of more than 256 experts and of lists that one launch does not take: the first kernel of the captured step is another one
@pytest.mark.parametrize("E, k", [(320, 10), (320, 8), (256, 6), (64, 4)])
def test_graphed_layer_routes_the_logits_of_its_own_call(E, k, device):
    """The step's kernels start behind the copy of the inputs, whichever of them is first: calls with new inputs in turn equal the eager layer's
    (large inputs, so that a kernel that did not wait would meet those of the call before)."""
    from triton_b200.moe import GraphedMoeLayer, moe_layer_forward
    from triton_b200.testing import make_synthetic_layer
    T, d = 1024, 512
    lw = make_synthetic_layer(E, d, 256, device, seed=7, block_scaled=True)
    graphed = GraphedMoeLayer(lw, k, T, d, E, device)
    g = torch.Generator(device=device).manual_seed(E + k)
    inputs = [(torch.randn(T, d, device=device, generator=g).bfloat16(), torch.randn(T, E, device=device, generator=g)) for _ in range(6)]
    want = [moe_layer_forward(x, logits, lw, k) for x, logits in inputs]
    torch.cuda.synchronize()
    got = [graphed(x, logits) for x, logits in inputs]
    tb.matmul_check_status()
    assert all(torch.equal(a, b) for a, b in zip(want, got)) and not torch.equal(want[0], want[1])


def test_graphed_layer_on_several_streams(layer_20b, device):
    """Calls from streams that wait for nothing of one another follow one another on the step's buffers: each result is that of its own inputs."""
    from triton_b200.moe import GraphedMoeLayer, moe_layer_forward
    lw, _, _ = layer_20b
    T = 64
    graphed = GraphedMoeLayer(lw, 4, T, 2880, 32, device)
    g = torch.Generator(device=device).manual_seed(1)
    inputs = [(torch.randn(T, 2880, device=device, generator=g).bfloat16(), torch.randn(T, 32, device=device, generator=g)) for _ in range(12)]
    want = [moe_layer_forward(x, logits, lw, 4) for x, logits in inputs]
    streams = [torch.cuda.Stream(device=device) for _ in range(3)]
    torch.cuda.synchronize()
    got = []
    for i, (x, logits) in enumerate(inputs):
        with torch.cuda.stream(streams[i % 3]):
            got.append(graphed(x, logits))
    torch.cuda.synchronize()
    tb.matmul_check_status()
    assert all(torch.equal(a, b) for a, b in zip(want, got))


def test_graphed_layer_is_refused_inside_a_capture(layer_20b, device):
    """A replay cannot be part of another capture: the call says so, and the layer goes on working."""
    from triton_b200.moe import GraphedMoeLayer, moe_layer_forward
    lw, _, _ = layer_20b
    graphed = GraphedMoeLayer(lw, 4, 5, 2880, 32, device)
    g = torch.Generator(device=device).manual_seed(2)
    x, logits = torch.randn(5, 2880, device=device, generator=g).bfloat16(), torch.randn(5, 32, device=device, generator=g)
    before = graphed(x, logits)
    with pytest.raises(RuntimeError):
        with torch.cuda.graph(torch.cuda.CUDAGraph()):
            graphed(x, logits)
    torch.cuda.synchronize()
    assert torch.equal(graphed(x, logits), before) and torch.equal(before, moe_layer_forward(x, logits, lw, 4))
    tb.matmul_check_status()


def test_host_streaming_layer(layer_20b, device):
    """Steps fed from and returned to pinned host memory through the three-stream pipeline equal the eager layer."""
    from triton_b200.moe import HostStreamingLayer, moe_layer_forward
    lw, _, _ = layer_20b
    T = 300
    pipe = HostStreamingLayer(lambda x, l: moe_layer_forward(x, l, lw, 4), T, 2880, 32, device)
    xs, ls, zs, want = [], [], [], []
    for seed in range(5):
        g = torch.Generator().manual_seed(seed)
        xs.append(torch.randn(T, 2880, generator=g).bfloat16().pin_memory())
        ls.append(torch.randn(T, 32, generator=g).pin_memory())
        zs.append(torch.empty(T, 2880, dtype=torch.bfloat16).pin_memory())
        want.append(moe_layer_forward(xs[-1].to(device), ls[-1].to(device), lw, 4).cpu())
    for i in range(5):
        pipe.submit(xs[i], ls[i], zs[i])
    pipe.drain()
    torch.cuda.synchronize()
    tb.matmul_check_status()
    for i in range(5):
        assert torch.equal(zs[i], want[i]), i


def _sampled_layer_check(lw, n_expts, tokens, device, seed, skew, n_sample=8):
    """Run the layer on `tokens` tokens and compare `n_sample` of its output rows with the CPU oracle, which needs only
    the experts those rows are routed to."""
    from triton_b200.moe import moe_layer_forward
    g = torch.Generator(device=device).manual_seed(seed)
    x = torch.randn(tokens, 2880, device=device, generator=g).bfloat16()
    logits = torch.randn(tokens, n_expts, device=device, generator=g)
    if skew:
        logits = logits + torch.randn(n_expts, device=device, generator=g)
    z = moe_layer_forward(x, logits, lw, 4)
    tb.matmul_check_status()
    rows = torch.linspace(0, tokens - 1, n_sample).round().long().unique()

    def expert_weights(e):
        w1 = oracle.dequant_weight_oracle(lw.w1_q[e:e + 1].cpu(), lw.w1_s[e:e + 1].cpu())[0]
        w2 = oracle.dequant_weight_oracle(lw.w2_q[e:e + 1].cpu(), lw.w2_s[e:e + 1].cpu())[0]
        return w1, lw.b1[e].cpu(), w2, lw.b2[e].cpu()

    ref = oracle.moe_layer_tokens_oracle(x[rows.to(device)].cpu(), logits[rows.to(device)].cpu(), expert_weights, 4, 1.702, 7.0)
    got = z[rows.to(device)].cpu()
    oracle.assert_close_oracle(ref, got, maxtol=MAXTOL_MX4, rmstol=None, what=f"layer E={n_expts} T={tokens}, sampled rows")
    assert oracle.rel_l2(ref, got) < 1e-2
    assert torch.isfinite(z.float()).all()


def test_gpt_oss_120b_layer_benchmark_configuration_against_oracle(device):
    """The benchmarked configuration itself -- 128 experts, 16384 tokens, skewed router: the pair kernel on the default weight
    tiles, bf16 tokens as two e4m3 terms -- against the CPU oracle on sampled tokens."""
    from triton_b200.testing import make_synthetic_layer
    lw = make_synthetic_layer(128, 2880, 2880, device, seed=1000, keep_canonical=True)
    assert lw.kernels(4 * 16384) == ("gemm_mx_pair_kernel",) * 2
    _sampled_layer_check(lw, 128, 16384, device, seed=0, skew=True)


def test_gpt_oss_120b_layer_on_the_bf16_kernel_against_oracle(device):
    """The same on the bf16 kernel, which narrow products of many rows take by themselves: 256 x 256 tiles, TMA activation loads,
    row-gather scratch."""
    from triton_b200.testing import make_synthetic_layer
    lw = make_synthetic_layer(128, 2880, 2880, device, seed=1000, keep_canonical=True)
    with tb.scoped_opt_flags_constraints({"kernel": "tcgen05"}):
        assert lw.kernels(4 * 16384) == ("gemm_tc_kernel",) * 2
        _sampled_layer_check(lw, 128, 16384, device, seed=0, skew=True)


def test_gpt_oss_120b_layer_prefill_on_the_block_scaled_copy_against_oracle(device):
    """The same with both weight copies: the pair kernel on the block-scaled tiles."""
    from triton_b200.testing import make_synthetic_layer
    lw = make_synthetic_layer(128, 2880, 2880, device, seed=1000, keep_canonical=True, block_scaled=True)
    assert lw.use_block_scaled(4 * 16384) and lw.kernels(4 * 16384) == ("gemm_mx_pair_kernel",) * 2
    _sampled_layer_check(lw, 128, 16384, device, seed=0, skew=True)


@pytest.mark.parametrize("tokens", [1, 16, 64, 300, 1200])
def test_gpt_oss_120b_layer_decode_path_against_oracle(tokens, device):
    """Steps of the 128-expert layer with up to 48 rows per expert on average take the block-scaled copy of the weights: 1 to 64
    tokens on the decode kernel in 16-row token blocks (four e2m1 terms), 300 (9 rows per expert) in 32-row blocks (two e4m3
    terms), 1200 (38 rows per expert) on the pair kernel."""
    from triton_b200.testing import make_synthetic_layer
    lw = make_synthetic_layer(128, 2880, 2880, device, seed=1000, keep_canonical=True, block_scaled=True)
    assert lw.use_block_scaled(tokens * 4)
    assert lw.kernels(tokens * 4) == ("gemm_mx_kernel" if tokens <= 300 else "gemm_mx_pair_kernel",) * 2
    _sampled_layer_check(lw, 128, tokens, device, seed=tokens, skew=True, n_sample=min(tokens, 6))


def test_weight_file_and_block_checkpoint_reader(tmp_path, device):
    """A layer saved in its tiled layouts and read back computes the same output bit for bit, and the checkpoint form
    (blocks [E, N, K/32, 16] + scales [E, N, K/32]) converts to the very same tiles."""
    from triton_b200.moe import moe_layer_forward
    from triton_b200.testing import make_synthetic_layer
    from triton_b200.weights_io import from_block_checkpoint, load_layer_weights, save_layer_weights
    E, d, ff, k, T = 8, 512, 256, 2, 100
    lw = make_synthetic_layer(E, d, ff, device, seed=3, keep_canonical=True, block_scaled=True)
    path = tmp_path / "layer.moeb200w"
    save_layer_weights(path, lw)
    back = load_layer_weights(path, device)
    torch.manual_seed(1)
    x = torch.randn(T, d, device=device).bfloat16()
    logits = torch.randn(T, E, device=device)
    z0, z1 = moe_layer_forward(x, logits, lw, k), moe_layer_forward(x, logits, back, k)
    tb.matmul_check_status()
    assert torch.equal(z0, z1)
    # checkpoint form: canonical K-packed bytes regrouped as 16-byte blocks
    blocks1 = lw.w1_q.transpose(1, 2).contiguous().reshape(E, 2 * ff, d // 32, 16)
    blocks2 = lw.w2_q.transpose(1, 2).contiguous().reshape(E, d, ff // 32, 16)
    ck = from_block_checkpoint(blocks1, lw.w1_s.transpose(1, 2).contiguous(), lw.b1, blocks2,
                               lw.w2_s.transpose(1, 2).contiguous(), lw.b2, block_scaled=True)
    for name in ("w1", "w1_scale", "w2", "w2_scale", "w1_bs", "w1_bs_scale", "w2_bs", "w2_bs_scale"):
        assert torch.equal(getattr(ck, name).storage.data, getattr(lw, name).storage.data), name


@pytest.mark.parametrize("tokens, E, k, dtype", [(1, 5, 1, "bf16"), (7, 33, 4, "bf16"), (256, 8, 6, "bf16"), (257, 8, 2, "bf16"),
                                                 (1100, 8, 2, "bf16"), (1, 5, 1, "e4m3"), (300, 33, 4, "e4m3")])
def test_layer_in_one_call_equals_the_operators(tokens, E, k, dtype, device):
    """The step as one native call runs the kernels of the step composed from the operators on the same operands: the results
    are the same bits.  (Sizes: either side of the single-launch routing, k the quad top-k does and does not take, 2048 gathered
    rows and fewer.)"""
    from triton_b200.moe import _NoTimer, _one_call, moe_layer_forward
    from triton_b200.testing import make_synthetic_layer
    lw = make_synthetic_layer(E, 512, 736, device, seed=3, block_scaled=True)
    for weights in ((lw,) if dtype == "e4m3" else (lw, make_synthetic_layer(E, 512, 736, device, seed=3))):
        g = torch.Generator(device=device).manual_seed(tokens + E)
        x = torch.randn(tokens, 512, device=device, generator=g).bfloat16()
        x = x.to(torch.float8_e4m3fn) if dtype == "e4m3" else x
        logits = torch.randn(tokens, E, device=device, generator=g)
        assert _one_call(x, logits, weights, k)
        one = moe_layer_forward(x, logits, weights, k)
        many = moe_layer_forward(x, logits, weights, k, gemm_timer=_NoTimer)
        tb.matmul_check_status()
        assert torch.equal(one, many)


def test_layer_with_a_bias_of_the_wrong_width_is_refused(device):
    """As the operators refuse it: nothing reads past the end of a bias row."""
    from triton_b200.moe import moe_layer_forward
    from triton_b200.testing import make_synthetic_layer
    x, logits = torch.randn(9, 512, device=device).bfloat16(), torch.randn(9, 8, device=device)
    for name in ("b1", "b2"):
        lw = make_synthetic_layer(8, 512, 256, device, seed=3, block_scaled=True)
        setattr(lw, name, getattr(lw, name)[:, :-32].contiguous())
        with pytest.raises(AssertionError):
            moe_layer_forward(x, logits, lw, 2)


@pytest.mark.parametrize("rows_per_expert", [40, 64])
@pytest.mark.parametrize("constraint", [{"kernel": "tcgen05"}, {"kernel": "tcgen05-pair"}, {"kernel": "stream"}, {"block_m": 128}, {"block_n": 256},
                                        {"kernel": "mx"}])
def test_layer_with_both_weight_copies_under_a_constraint(constraint, rows_per_expert, device):
    """Beyond 48 rows per expert a layer with both weight copies runs the kernel or tile that a constraint names: the same bits
    as without the second copy.  Up to there it stays on the block-scaled copy, which refuses a bf16 kernel."""
    from triton_b200.moe import moe_layer_forward
    from triton_b200.testing import make_synthetic_layer
    E, k = 8, 2
    T = rows_per_expert * E // k
    g = torch.Generator(device=device).manual_seed(1)
    x = torch.randn(T, 512, device=device, generator=g).bfloat16()
    logits = torch.randn(T, E, device=device, generator=g)
    both, default = make_synthetic_layer(E, 512, 736, device, seed=3, block_scaled=True), make_synthetic_layer(E, 512, 736, device, seed=3)
    free = moe_layer_forward(x, logits, both, k)
    with tb.scoped_opt_flags_constraints(constraint):
        if rows_per_expert <= 48 and constraint.get("kernel", "mx") != "mx":
            with pytest.raises(tb.InapplicableConstraint):
                moe_layer_forward(x, logits, both, k)
            return
        y = moe_layer_forward(x, logits, both, k)
        tb.matmul_check_status()
        assert oracle.rel_l2(free.cpu(), y.cpu()) < 1e-2
        if rows_per_expert > 48 and "mx" not in constraint.values():
            assert torch.equal(y, moe_layer_forward(x, logits, default, k))


@pytest.mark.parametrize("block_scaled", [False, True])
def test_layer_in_one_call_sizes_its_workspace_for_the_activation(block_scaled, device):
    """fc1 over few k behind SwiGLU takes the bf16 kernel from 512 rows per expert on: the one call asks for its temporaries with the
    activation set, so that it runs what the operators run."""
    from triton_b200.moe import _NoTimer, moe_layer_forward
    from triton_b200.testing import make_synthetic_layer
    E, d, ff, k, T = 8, 512, 2176, 2, 2100
    lw = make_synthetic_layer(E, d, ff, device, seed=3, block_scaled=block_scaled)
    assert lw.kernels(T * k)[0] == "gemm_tc_kernel" and lw.kernels(500 * E)[0] == "gemm_mx_pair_kernel"
    g = torch.Generator(device=device).manual_seed(1)
    x, logits = torch.randn(T, d, device=device, generator=g).bfloat16(), torch.randn(T, E, device=device, generator=g)
    one, many = moe_layer_forward(x, logits, lw, k), moe_layer_forward(x, logits, lw, k, gemm_timer=_NoTimer)
    tb.matmul_check_status()
    assert torch.equal(one, many)


@pytest.mark.parametrize("tokens", [3, 40, 300, 1300])
def test_layer_step_captured_behind_a_join(tokens, device):
    """A step captured where its stream has just joined another one (two predecessors, neither of them a kernel of this package), and a second
    step right behind it on the first one's result: the bits of the eager steps."""
    from triton_b200.moe import moe_layer_forward
    from triton_b200.testing import make_synthetic_layer
    E, d, k = 8, 512, 2
    lw = make_synthetic_layer(E, d, 736, device, seed=3, block_scaled=True)
    g = torch.Generator(device=device).manual_seed(tokens)
    x, logits = torch.randn(tokens, d, device=device, generator=g).bfloat16(), torch.randn(tokens, E, device=device, generator=g)
    side = torch.cuda.Stream(device=device)

    def step():
        side.wait_stream(torch.cuda.current_stream(device))
        with torch.cuda.stream(side):
            xs = x * 2
        ls = logits + 1
        torch.cuda.current_stream(device).wait_stream(side)
        xs.record_stream(torch.cuda.current_stream(device))
        z = moe_layer_forward(xs, ls, lw, k)
        return z, moe_layer_forward(z, ls, lw, k)

    eager = [t.clone() for t in step()]
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = step()
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    tb.matmul_check_status()
    assert all(torch.equal(a, b) for a, b in zip(eager, captured))


@pytest.mark.parametrize("tokens, experts, dtype", [(3, 8, "bf16"), (40, 8, "bf16"), (300, 8, "bf16"), (1300, 8, "bf16"), (2100, 16, "bf16"),
                                                    (40, 8, "e4m3"), (300, 8, "e4m3"), (1300, 8, "e4m3")])
def test_captured_layer_steps_with_changed_inputs(tokens, experts, dtype, device):
    """As above, the second step with routing of its own.  Before every replay tokens, logits (with very different expert
    loads) and weights are overwritten in place: a kernel that reads what the replay before has left gives other bits than the eager steps.
    Routing in one and in two launches, tokens packed by position and by row, both block-scaled kernels."""
    from triton_b200.moe import moe_layer_forward
    from triton_b200.testing import make_synthetic_layer
    d, k, sets = 512, 2, 3
    type_ = torch.float8_e4m3fn if dtype == "e4m3" else torch.bfloat16
    weights = [make_synthetic_layer(experts, d, 736, device, seed=3 + i, block_scaled=True) for i in range(sets + 1)]
    lw = weights.pop()
    names = ["w1", "w1_scale", "b1", "w2", "w2_scale", "b2", "w1_bs", "w1_bs_scale", "w2_bs", "w2_bs_scale"]

    def parts(layer):
        return [t if isinstance(t, torch.Tensor) else t.storage.data for t in (getattr(layer, n) for n in names)]

    g = torch.Generator(device=device).manual_seed(tokens)
    inputs = [[torch.randn(tokens, d, device=device, generator=g)] + [torch.randn(tokens, experts, device=device, generator=g)
               + 3 * torch.randn(experts, device=device, generator=g) for _ in range(2)] for _ in range(sets)]
    x, logits, logits2 = (torch.zeros_like(t) for t in inputs[0])
    side = torch.cuda.Stream(device=device)

    def fill(i):
        for to, frm in zip([x, logits, logits2, *parts(lw)], [*inputs[i], *parts(weights[i])]):
            to.view(torch.uint8).copy_(frm.view(torch.uint8))

    def step():
        side.wait_stream(torch.cuda.current_stream(device))
        with torch.cuda.stream(side):
            xs = (x * 2).to(type_)
        ls = logits + 1
        torch.cuda.current_stream(device).wait_stream(side)
        xs.record_stream(torch.cuda.current_stream(device))
        z = moe_layer_forward(xs, ls, lw, k)
        return z, moe_layer_forward(z.to(type_), logits2, lw, k)

    eager = []
    for i in range(sets):
        fill(i)
        eager.append([t.clone() for t in step()])
        torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = step()
    got = []
    order = [1, 0, 2, 2, 1, 0]
    for i in order:
        fill(i)
        graph.replay()
        got.append([t.clone() for t in captured])
    torch.cuda.synchronize()
    tb.matmul_check_status()
    for i, replayed in zip(order, got):
        assert all(torch.equal(a, b) for a, b in zip(eager[i], replayed))
    assert not torch.equal(eager[0][1], eager[1][1])
