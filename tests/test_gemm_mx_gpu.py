"""The block-scaled grouped GEMM (tcgen05.mma.kind::mxf8f6f4: MXFP4 weights straight into the MMA) on the GPU against
the CPU oracle: e4m3 and MXFP8 activations (the reference's `a_mx_scale` mode, tests/test_matmul.py:282-285), and bf16
activations split inside the library into two e4m3 terms, or (small token blocks) into four e2m1 terms for
tcgen05.mma.kind::mxf4."""
import pytest
import torch

import oracle
import triton_b200 as tb
from triton_b200.tensor import FP4, convert_layout, wrap_torch_tensor
from triton_b200.tensor_details.layout import B200BlockScaledScaleLayout, B200BlockScaledValueLayout

pytestmark = pytest.mark.gpu

MAXTOL_MX4 = 3e-2          # the reference's bound for MXFP4 weights (tests/test_matmul.py:649-650)


def quantised_weights(E, K, N, g, unit_scales=False, w_std=0.02):
    w = (torch.randn(E, K, N, generator=g) * w_std).bfloat16()
    wq, ws = oracle.downcast_to_mxfp_oracle(w, 1)
    if unit_scales:
        ws = torch.full_like(ws, 127)
    # K contiguous, as downcast_to_mxfp(axis=1) returns it
    wq = wq.contiguous().transpose(1, 2).contiguous().transpose(1, 2)
    ws = ws.contiguous().transpose(1, 2).contiguous().transpose(1, 2)
    return wq, ws, oracle.dequant_weight_oracle(wq, ws)


def to_block_scaled(wq, ws, device):
    tq = convert_layout(wrap_torch_tensor(wq.to(device), dtype=FP4), B200BlockScaledValueLayout())
    ts = convert_layout(wrap_torch_tensor(ws.to(device)), B200BlockScaledScaleLayout())
    return tq, ts


def test_block_scaled_layout_round_trip(device):
    g = torch.Generator().manual_seed(3)
    for E, K, N in [(2, 96, 40), (3, 2880, 200), (1, 128, 128)]:
        wq = torch.randint(0, 256, (E, N, K // 2), generator=g, dtype=torch.uint8).transpose(1, 2)   # [E, K/2, N], K contiguous
        ws = torch.randint(0, 255, (E, N, K // 32), generator=g, dtype=torch.uint8).transpose(1, 2)
        tq, ts = to_block_scaled(wq, ws, device)
        KT, NB = (K + 127) // 128, (N + 127) // 128
        assert tq.storage.data.numel() == E * KT * NB * 128 * 64 and ts.storage.data.numel() == E * KT * NB * 512
        # spot-check the documented positions on the host
        v = tq.storage.data.cpu().view(E, KT, NB, 128, 64)
        s = ts.storage.data.cpu().view(E, KT, NB, 32, 4, 4)
        for (e, n, k) in [(0, 0, 0), (E - 1, N - 1, K - 2), (0, min(N - 1, 33), min(K - 2, 70))]:
            assert int(v[e, k // 128, n // 128, n % 128, (k % 128) // 2]) == int(wq[e, k // 2, n])
            assert int(s[e, k // 128, n // 128, (n % 128) % 32, (n % 128) // 32, (k % 128) // 32]) == int(ws[e, k // 32, n])
        from triton_b200.tensor_details.layout import StridedLayout
        back_q = convert_layout(tq, StridedLayout(major_dim=-2))
        back_s = convert_layout(ts, StridedLayout(major_dim=-2))
        assert torch.equal(back_q.storage.data.cpu(), wq) and torch.equal(back_s.storage.data.cpu(), ws)


def run_mx(x, wq, ws, sizes, device, *, a_scale=None, bias=None, gather=None, scatter=None, gammas=None, betas=None,
           act=None, out_dtype=torch.bfloat16, block_m=None, block_n=None, kernel=None):
    dev = lambda t: None if t is None else t.to(device)
    tq, ts = to_block_scaled(wq, ws, device)
    M = int(sizes.sum())
    md = tb.make_ragged_tensor_metadata(dev(sizes), M)
    pc = tb.PrecisionConfig(b_mx_scale=ts, b_microblock_size=32, a_mx_scale=dev(a_scale), out_dtype=out_dtype)
    fa = None
    if act:
        fa = tb.FusedActivation(tb.FnSpecs("swiglu", tb.swiglu_fn, ("alpha", "limit"), reduction_n=2), act)
    cons = {}
    if block_m:
        cons["block_m"] = block_m
    if block_n:
        cons["block_n"] = block_n
    if kernel:
        cons["kernel"] = kernel
    with tb.scoped_opt_flags_constraints(cons):
        y = tb.matmul(dev(x), tq, dev(bias), md, None, dev(gather), dev(scatter), pc, betas=dev(betas), gammas=dev(gammas),
                      fused_activation=fa)
    tb.matmul_check_status()
    return y.cpu()


def dequant_act(x8, a_scale):
    xf = x8.float()
    if a_scale is not None:
        xf = (xf.view(x8.shape[0], -1, 32) * torch.exp2(a_scale.float() - 127.0)[:, :, None]).reshape(x8.shape)
    return xf


@pytest.mark.parametrize("stage", ["unit-scales", "weight-scales", "act-scales"])
@pytest.mark.parametrize("block_n", [128, 256, 384])
def test_block_scaled_dense_fp8_exact_products(stage, block_n, device):
    """One expert, e4m3 activations: every product is exact in the tensor core and the sum is fp32, so the result
    must match the fp32 oracle closely.  The three stages separate the value path (unit scales), the weight scales
    (per row and k group) and the activation scales."""
    g = torch.Generator().manual_seed(1)
    M, K, N = 48, 384, 384
    wq, ws, wdeq = quantised_weights(1, K, N, g, unit_scales=(stage == "unit-scales"), w_std=1.0)
    x8 = torch.randn(M, K, generator=g).to(torch.float8_e4m3fn)
    a_scale = None
    if stage == "act-scales":
        a_scale = torch.randint(120, 134, (M, K // 32), generator=g, dtype=torch.uint8)
    sizes = torch.tensor([M], dtype=torch.int32)
    y = run_mx(x8, wq, ws, sizes, device, a_scale=a_scale, out_dtype=torch.float32, block_n=block_n)
    ref = oracle.matmul_oracle(dequant_act(x8, a_scale), wdeq, None, sizes, out_dtype=torch.float32)
    err = (y - ref).abs().max().item() / ref.abs().max().item()
    assert err < 1e-5, f"{stage}: max error relative to max|ref| = {err}"


CASES = [
    # E, K, N, sizes, T
    (4, 96, 64, [13, 0, 29, 8], 50),
    (3, 512, 256, [130, 1, 64], 200),
    (8, 2880, 384, [0, 17, 128, 129, 3, 0, 64, 255], 300),
    (5, 320, 640, [60, 25, 7, 0, 51], 90),
]


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("mode", ["plain", "gather", "scatter_w", "swiglu", "all"])
@pytest.mark.parametrize("acts", ["bf16", "fp8", "mxfp8"])
def test_block_scaled_grouped_gemm(case, mode, acts, device):
    E, K, N, sizes, T = case
    g = torch.Generator().manual_seed(hash((E, K, N, mode)) % 1000)
    opts = dict(plain=dict(gather=False), gather=dict(gather=True),
                scatter_w=dict(gather=True, scatter=True, weights=True), swiglu=dict(gather=True, act=True),
                all=dict(gather=True, scatter=True, weights=True, act=True))[mode]
    sizes_t = torch.tensor(sizes, dtype=torch.int32)
    M = int(sizes_t.sum())
    rows_x = T if opts.get("gather") else M
    wq, ws, wdeq = quantised_weights(E, K, N, g)
    xb = torch.randn(rows_x, K, generator=g).bfloat16()
    a_scale = None
    if acts == "bf16":
        x, xref = xb, xb.float()
    else:
        x = xb.to(torch.float8_e4m3fn)
        if acts == "mxfp8":
            a_scale = torch.randint(122, 131, (rows_x, K // 32), generator=g, dtype=torch.uint8)
        xref = dequant_act(x, a_scale)
    bias = torch.randn(E, N, generator=g) * 0.1
    gather = torch.randint(0, T, (M,), generator=g, dtype=torch.int32) if opts.get("gather") else None
    scatter = torch.randperm(M, generator=g).int() if opts.get("scatter") else None
    gammas = torch.rand(M, generator=g) if opts.get("weights") else None
    betas = torch.rand(M, generator=g) if opts.get("weights") else None
    act = (1.702, 7.0) if opts.get("act") else None
    y = run_mx(x, wq, ws, sizes_t, device, a_scale=a_scale, bias=bias, gather=gather, scatter=scatter, gammas=gammas,
               betas=betas, act=act)
    ref = oracle.matmul_oracle(xref, wdeq, bias, sizes_t, gather, None, betas=betas, gammas=None if act else gammas,
                               out_dtype=torch.float32)
    if act:
        ref = oracle.swiglu_oracle(ref, *act)
        if gammas is not None:
            ref = ref * gammas[:, None]
    ref = ref.bfloat16()
    if scatter is not None:
        out = torch.zeros_like(ref)
        out[scatter.long()] = ref
        ref = out
    oracle.assert_close_oracle(ref, y, maxtol=MAXTOL_MX4, rmstol=None, what=f"block-scaled gemm {acts}")
    assert oracle.rel_l2(ref, y) < 1e-2


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("mode", ["plain", "scatter_w", "all"])
@pytest.mark.parametrize("kernel", ["mx-f8", "mx-f4"])
def test_block_scaled_bf16_token_forms(case, mode, kernel, device):
    """bf16 tokens in each of the two forms the kernel can split them into, pinned (the automatic choice depends on
    the block size): two e4m3 terms and four e2m1 terms."""
    E, K, N, sizes, T = case
    g = torch.Generator().manual_seed(hash((E, K, N, mode)) % 1000 + 1)
    opts = dict(plain={}, scatter_w=dict(gather=True, scatter=True, weights=True),
                all=dict(gather=True, scatter=True, weights=True, act=True))[mode]
    sizes_t = torch.tensor(sizes, dtype=torch.int32)
    M = int(sizes_t.sum())
    rows_x = T if opts.get("gather") else M
    wq, ws, wdeq = quantised_weights(E, K, N, g)
    x = torch.randn(rows_x, K, generator=g).bfloat16()
    bias = torch.randn(E, N, generator=g) * 0.1
    gather = torch.randint(0, T, (M,), generator=g, dtype=torch.int32) if opts.get("gather") else None
    scatter = torch.randperm(M, generator=g).int() if opts.get("scatter") else None
    gammas = torch.rand(M, generator=g) if opts.get("weights") else None
    betas = torch.rand(M, generator=g) if opts.get("weights") else None
    act = (1.702, 7.0) if opts.get("act") else None
    y = run_mx(x, wq, ws, sizes_t, device, bias=bias, gather=gather, scatter=scatter, gammas=gammas, betas=betas, act=act,
               out_dtype=torch.float32, kernel=kernel)
    ref = oracle.matmul_oracle(x.float(), wdeq, bias, sizes_t, gather, None, betas=betas, gammas=None if act else gammas,
                               out_dtype=torch.float32)
    if act:
        ref = oracle.swiglu_oracle(ref, *act)
        if gammas is not None:
            ref = ref * gammas[:, None]
    if scatter is not None:
        out = torch.zeros_like(ref)
        out[scatter.long()] = ref
        ref = out
    # fp32 output: what is left is the split of the tokens (two e4m3 terms hold a bf16 value exactly up to underflow;
    # four e2m1 terms leave about 2^-14 of a group's maximum) and the order of the fp32 sums
    assert oracle.rel_l2(ref, y) < (5e-4 if kernel == "mx-f4" else 2e-5)


@pytest.mark.parametrize("block_m, kernel", [(16, "mx"), (32, "mx"), (64, "mx"), (16, "mx-f8"), (16, "mx-f4"), (32, "mx-f4")])
def test_block_scaled_token_block_sizes(block_m, kernel, device):
    """bf16 activations with every token-block size: experts with more rows than a block take several blocks."""
    g = torch.Generator().manual_seed(7)
    E, K, N = 6, 640, 640           # five weight blocks in groups of three: the last group of the last expert is partial
    sizes = torch.tensor([70, 1, 0, 33, 16, 5], dtype=torch.int32)
    M = int(sizes.sum())
    wq, ws, wdeq = quantised_weights(E, K, N, g)
    x = torch.randn(M, K, generator=g).bfloat16()
    y = run_mx(x, wq, ws, sizes, device, block_m=block_m, block_n=384, kernel=kernel)
    ref = oracle.matmul_oracle(x.float(), wdeq, None, sizes, out_dtype=torch.float32).bfloat16()
    oracle.assert_close_oracle(ref, y, maxtol=MAXTOL_MX4, rmstol=None, what="block-scaled gemm")
    assert oracle.rel_l2(ref, y) < 1e-2


@pytest.mark.parametrize("acts, block_m", [("bf16", 16), ("bf16", 32), ("bf16", 64), ("fp8", 32), ("mxfp8", 16), ("mxfp8", 64), ("fp8", 128)])
@pytest.mark.parametrize("K, N, mode", [(96, 640, "plain"), (320, 129, "plain"), (640, 514, "scatter"), (416, 640, "swiglu"), (160, 768, "swiglu"), (128, 256, "e4m3")])
def test_block_scaled_tiles_of_two_weight_blocks(K, N, mode, acts, block_m, device):
    """The tiles that products of byte-expanded operands choose: odd and even counts of weight blocks, a last block of one row, widths without
    vector stores, experts of several token blocks, every output type.  fp32 outputs: products are exact and only the order of the sums differs."""
    g = torch.Generator().manual_seed(K + N + block_m)
    sizes = torch.tensor([70, 1, 0, 33, 16, 150], dtype=torch.int32)
    E, M = 6, int(sizes.sum())
    wq, ws, wdeq = quantised_weights(E, K, N, g)
    x = torch.randn(M, K, generator=g).bfloat16()
    a_scale = None
    if acts != "bf16":
        x = x.to(torch.float8_e4m3fn)
        if acts == "mxfp8":
            a_scale = torch.randint(122, 131, (M, K // 32), generator=g, dtype=torch.uint8)
    bias = torch.randn(E, N, generator=g) * 0.1
    scatter, gammas = (torch.randperm(M, generator=g).int(), torch.rand(M, generator=g)) if mode == "scatter" else (None, None)
    act = (1.702, 7.0) if mode == "swiglu" else None
    out_dtype = torch.float8_e4m3fn if mode == "e4m3" else torch.float32
    y = run_mx(x, wq, ws, sizes, device, a_scale=a_scale, bias=bias, scatter=scatter, gammas=gammas, act=act, out_dtype=out_dtype,
               kernel="mx-f8", block_m=block_m, block_n=256)
    ref = oracle.matmul_oracle(x.float() if acts == "bf16" else dequant_act(x, a_scale), wdeq, bias, sizes, gammas=gammas, out_dtype=torch.float32)
    if act:
        ref = oracle.swiglu_oracle(ref, *act)
    if scatter is not None:
        ref = torch.zeros_like(ref).index_copy_(0, scatter.long(), ref)
    if mode == "e4m3":                                               # one step of e4m3 where the sums differ at a rounding boundary
        ref8 = ref.to(torch.float8_e4m3fn).float()
        diff = (y.float() - ref8).abs()
        assert (diff <= ref8.abs().clamp_min(2.0 ** -6) * 0.125).all() and (diff > 0).float().mean() < 0.02
    else:
        assert oracle.rel_l2(ref, y) < 2e-5


@pytest.mark.parametrize("kernel", ["mx-f8", "mx-f4"])
def test_block_scaled_wide_dynamic_range_rows(kernel, device):
    """bf16 rows whose magnitudes span 2^40: each 32-group has its own scales, so small groups next to large ones keep
    their precision."""
    g = torch.Generator().manual_seed(9)
    E, K, N, M = 1, 512, 128, 20
    wq, ws, wdeq = quantised_weights(E, K, N, g)
    x = torch.randn(M, K, generator=g)
    x = (x * torch.exp2(torch.randint(-20, 20, (M, K // 32), generator=g).float()).repeat_interleave(32, dim=1)).bfloat16()
    sizes = torch.tensor([M], dtype=torch.int32)
    y = run_mx(x, wq, ws, sizes, device, out_dtype=torch.float32, kernel=kernel)
    ref = oracle.matmul_oracle(x.float(), wdeq, None, sizes, out_dtype=torch.float32)
    assert oracle.rel_l2(ref, y) < 1e-3


# each place of the four that a lane has, and of the eight; from 2.98e38 on a code times its scale is beyond the largest number
@pytest.mark.parametrize("k", [0, 1, 2, 3, 5, 255])
@pytest.mark.parametrize("value", [2.99e38, -3.38e38])
@pytest.mark.parametrize("kernel, block_m, bound", [("mx-f4", 16, 5e-4), ("mx-f8", 32, 2e-5)])
def test_block_scaled_values_near_the_largest(kernel, block_m, bound, value, k, device):
    """A bf16 value that is nearly the largest there is keeps its terms wherever it stands (the bounds are those of the forms)."""
    g = torch.Generator().manual_seed(k)
    wq, ws, wdeq = quantised_weights(1, 256, 128, g)
    x = torch.randn(12, 256, generator=g).bfloat16()
    x[3, k] = value
    sizes = torch.tensor([12], dtype=torch.int32)
    y = run_mx(x, wq, ws, sizes, device, out_dtype=torch.float32, kernel=kernel, block_m=block_m).double()
    ref = x.double() @ wdeq[0].double()
    assert oracle.rel_l2(ref[3] * 1e-38, y[3] * 1e-38) < bound
    rest = torch.arange(12) != 3
    assert oracle.rel_l2(ref[rest], y[rest]) < 5e-4


@pytest.mark.parametrize("k", [0, 1, 2, 3, 5, 255])
@pytest.mark.parametrize("value", [float("inf"), -float("inf"), float("nan")])
def test_four_terms_beside_a_value_that_is_not_finite(value, k, device):
    """The other values of its group of 32 keep three terms and more, wherever it stands: seen where its own weights are zero."""
    g = torch.Generator().manual_seed(k)
    wq, ws, _ = quantised_weights(1, 256, 128, g)
    low = wq[:, k // 2] & (0xF0 if k % 2 == 0 else 0x0F)             # the code of weight row k is zero for every output
    wq[:, k // 2] = low
    wdeq = oracle.dequant_weight_oracle(wq, ws)
    x = torch.randn(12, 256, generator=g).bfloat16()
    ref = x.double() @ wdeq[0].double()
    x[3, k] = value
    y = run_mx(x, wq, ws, torch.tensor([12], dtype=torch.int32), device, out_dtype=torch.float32, kernel="mx-f4", block_m=16).double()
    # three terms leave 1e-3 of the group's eighth of the row
    assert oracle.rel_l2(ref, y) < 5e-4 and oracle.rel_l2(ref[3], y[3]) < 1e-3


def test_block_scaled_e4m3_output(device):
    """fc1 of the fp8 mode: e4m3 rows in, SwiGLU, e4m3 rows out (saturating round to nearest)."""
    g = torch.Generator().manual_seed(21)
    E, K, N = 3, 512, 512
    sizes = torch.tensor([40, 0, 77], dtype=torch.int32)
    M = int(sizes.sum())
    wq, ws, wdeq = quantised_weights(E, K, N, g, w_std=0.05)
    x8 = torch.randn(M, K, generator=g).to(torch.float8_e4m3fn)
    bias = torch.randn(E, N, generator=g) * 0.1
    y = run_mx(x8, wq, ws, sizes, device, bias=bias, act=(1.702, 7.0), out_dtype=torch.float8_e4m3fn)
    assert y.dtype == torch.float8_e4m3fn
    ref32 = oracle.swiglu_oracle(oracle.matmul_oracle(x8.float(), wdeq, bias, sizes, out_dtype=torch.float32), 1.702, 7.0)
    ref8 = ref32.to(torch.float8_e4m3fn)
    # equal up to one e4m3 step where the fp32 sums differ in their last bits right at a rounding boundary
    diff = (y.float() - ref8.float()).abs()
    step = ref8.float().abs().clamp_min(2.0 ** -6) * 0.125
    assert (diff <= step).all()
    assert (diff > 0).float().mean() < 0.02


@pytest.mark.parametrize("tokens, E, kernel", [(64, 16, "gemm_mx_pair_kernel"), (2048, 16, "gemm_mx_pair_kernel"), (48, 16, "gemm_mx_kernel"),
                                               (8192, 32, "gemm_mx_pair_kernel")])
def test_layer_with_e4m3_activations_against_oracle(tokens, E, kernel, device):
    """The layer in fp8 mode (e4m3 tokens in, e4m3 between the GEMMs) against the oracle fed the same quantised rows: 16 rows per
    expert and prefill sizes on the pair kernel, fewer on the decode kernel."""
    from triton_b200.moe import moe_layer_forward
    from triton_b200.testing import make_synthetic_layer
    k = 4
    lw = make_synthetic_layer(E, 2880, 2880, device, seed=5, keep_canonical=True, block_scaled=True)
    g = torch.Generator(device=device).manual_seed(tokens)
    x8 = torch.randn(tokens, 2880, device=device, generator=g).to(torch.float8_e4m3fn)
    logits = torch.randn(tokens, E, device=device, generator=g)
    assert lw.kernels(tokens * k, torch.float8_e4m3fn) == (kernel,) * 2
    z = moe_layer_forward(x8, logits, lw, k)
    tb.matmul_check_status()
    assert z.dtype == torch.bfloat16
    rows = torch.linspace(0, tokens - 1, 6).round().long().unique()

    def expert_weights(e):
        w1 = oracle.dequant_weight_oracle(lw.w1_q[e:e + 1].cpu(), lw.w1_s[e:e + 1].cpu())[0]
        w2 = oracle.dequant_weight_oracle(lw.w2_q[e:e + 1].cpu(), lw.w2_s[e:e + 1].cpu())[0]
        return w1, lw.b1[e].cpu(), w2, lw.b2[e].cpu()

    ref = oracle.moe_layer_tokens_oracle(x8[rows.to(device)].cpu().float(), logits[rows.to(device)].cpu(), expert_weights, k,
                                         1.702, 7.0, h_dtype=torch.float8_e4m3fn, out_dtype=torch.bfloat16)
    got = z[rows.to(device)].cpu()
    oracle.assert_close_oracle(ref, got, maxtol=MAXTOL_MX4, rmstol=None, what="fp8 layer")
    assert oracle.rel_l2(ref, got) < 1e-2


@pytest.mark.parametrize("K", [384, 640, 2880])
@pytest.mark.parametrize("sizes", [[3, 0, 1, 16, 0, 7], [1], [16, 16, 5, 2], [20, 1, 0, 33]])
@pytest.mark.parametrize("act", [False, True])
def test_block_scaled_few_tiles_k_step_stages(K, sizes, act, device):
    """Decode-sized calls with so few tiles that a CTA gets single weight blocks: the kernel then puts three k steps of
    one block into a stage (K = 384: exactly one stage; 640: a full and a partial one; 2880: seven and a partial one)."""
    g = torch.Generator().manual_seed(K + len(sizes) * 7 + int(act))
    E, N = len(sizes), 640
    sizes_t = torch.tensor(sizes, dtype=torch.int32)
    M = int(sizes_t.sum())
    wq, ws, wdeq = quantised_weights(E, K, N, g)
    x = torch.randn(M, K, generator=g).bfloat16()
    bias = torch.randn(E, N, generator=g) * 0.1
    gammas = torch.rand(M, generator=g)
    scatter = torch.randperm(M, generator=g).int()
    a = (1.702, 7.0) if act else None
    ref = oracle.matmul_oracle(x.float(), wdeq, bias, sizes_t, None, None, gammas=None if act else gammas, out_dtype=torch.float32)
    if act:
        ref = oracle.swiglu_oracle(ref, *a) * gammas[:, None]
    out = torch.zeros_like(ref)
    out[scatter.long()] = ref
    y = run_mx(x, wq, ws, sizes_t, device, bias=bias, scatter=scatter, gammas=gammas, act=a, out_dtype=torch.float32,
               kernel="mx-f4", block_m=16)
    assert oracle.rel_l2(out, y) < 5e-4


@pytest.mark.parametrize("kernel", ["mx-f4", "mx-f8"])
@pytest.mark.parametrize("K", [128, 640])                   # one k step, and an odd number of them
@pytest.mark.parametrize("E, N", [(50, 1152), (50, 1280), (50, 1408), (50, 384), (7, 640)])
def test_block_scaled_last_round_by_blocks(E, N, K, kernel, device):
    """What does not fill a last round of the 148 CTAs is dealt out by single weight blocks, two k steps a stage: behind a whole round
    with 0, 1 and 2 blocks left over per token block, as all there is, and not where it would take two rounds."""
    g = torch.Generator().manual_seed(E + N + K)
    sizes = torch.randint(1, 17, (E,), generator=g).int()
    M = int(sizes.sum())
    wq, ws, wdeq = quantised_weights(E, K, N, g)
    x = torch.randn(M, K, generator=g).bfloat16()
    ref = oracle.matmul_oracle(x.float(), wdeq, None, sizes, out_dtype=torch.float32)
    y = run_mx(x, wq, ws, sizes, device, out_dtype=torch.float32, kernel=kernel, block_m=16, block_n=384)
    assert oracle.rel_l2(ref, y) < 5e-4


@pytest.mark.parametrize("acts", ["bf16", "fp8", "mxfp8"])
@pytest.mark.parametrize("K, N, sizes", [
    (32, 2, [1, 0, 33]),                            # one group of k, one column pair
    (128, 256, [192, 193, 224, 225]),               # one whole k step, one 256-row block, around the tile of either form
    (160, 129, [31, 32, 5, 449]),                   # k tail, odd width (scalar stores), an expert of several tiles
    (416, 514, [64, 1, 0, 97]),                     # ring longer than the k loop, a second tile of weight blocks
    (1024, 768, [300]),                             # three 256-row blocks: the last tile has one unit
    (160, 5129, [31, 32, 95, 40]),                  # enough tiles for two 256-row blocks each, the last has one row
    (96, 4866, [300, 2, 2, 700]),                   # the same with more rows per expert
    (96, 514, [225, 385]),                          # more rows per expert, one 256-row block each
])
@pytest.mark.parametrize("act", [False, True])
def test_pair_kernel_tile_edges(K, N, sizes, acts, act, device):
    """The pair form at the edges of its tiles, fp32 outputs.  e4m3 products and the two e4m3 terms of a bf16 value are
    exact, so only the order of an fp32 sum of K terms differs: 2e-5 of the norm is far above its error."""
    if act and N % 2:
        pytest.skip("SwiGLU needs an even width")
    g = torch.Generator().manual_seed(K + N + len(sizes))
    E, M = len(sizes), sum(sizes)
    sizes_t = torch.tensor(sizes, dtype=torch.int32)
    wq, ws, wdeq = quantised_weights(E, K, N, g)
    T = M + 7
    x = torch.randn(T, K, generator=g).bfloat16()
    a_scale = None
    if acts != "bf16":
        x = x.to(torch.float8_e4m3fn)
        if acts == "mxfp8":
            a_scale = torch.randint(122, 131, (T, K // 32), generator=g, dtype=torch.uint8)
    xref = x.float() if acts == "bf16" else dequant_act(x, a_scale)
    gather = torch.randint(0, T, (M,), generator=g, dtype=torch.int32)
    scatter, gammas, betas = torch.randperm(M, generator=g).int(), torch.rand(M, generator=g), torch.rand(M, generator=g)
    bias = torch.randn(E, N, generator=g) * 0.1
    ref = oracle.matmul_oracle(xref[gather.long()], wdeq, bias, sizes_t, None, None, betas=betas, out_dtype=torch.float32)
    if act:
        ref = oracle.swiglu_oracle(ref, 1.702, 7.0)
    out = torch.zeros_like(ref)
    out[scatter.long()] = ref * gammas[:, None]
    y = run_mx(x, wq, ws, sizes_t, device, a_scale=a_scale, bias=bias, gather=gather, scatter=scatter, gammas=gammas, betas=betas,
               act=(1.702, 7.0) if act else None, out_dtype=torch.float32, block_m=256)
    assert oracle.rel_l2(out, y) < 2e-5


@pytest.mark.parametrize("K, N, sizes", [
    (32, 2, [1, 0, 33]),                            # one group of k, one column pair
    (128, 256, [192, 193, 224, 225]),               # one whole k step, one 256-row block
    (160, 129, [31, 32, 5, 449]),                   # k tail, odd width, an expert of several tiles
    (416, 514, [64, 1, 0, 97]),                     # a second tile of weight blocks
    (1024, 768, [300, 2, 2]),                       # three 256-row blocks: the last tile has one
    (160, 5129, [31, 32, 95, 40]),                  # enough tiles for two 256-row blocks each, the last has one row
    (96, 4866, [300, 2, 2, 700]),                   # the same with more rows per expert
    (96, 514, [225, 385]),                          # more rows per expert, one 256-row block each
])
@pytest.mark.parametrize("act", [False, True])
def test_pair_kernel_on_default_weight_tiles(K, N, sizes, act, device):
    """The pair kernel fed from the default layout (rows of a weight block permuted, k permuted inside eight).  As above, only
    the order of an fp32 sum of exact products differs."""
    from triton_b200.tensor_details.layout import B200MXScaleLayout, B200MXValueLayout
    if act and N % 2:
        pytest.skip("SwiGLU needs an even width")
    g = torch.Generator().manual_seed(K + N + len(sizes))
    E, M = len(sizes), sum(sizes)
    sizes_t = torch.tensor(sizes, dtype=torch.int32)
    wq, ws, wdeq = quantised_weights(E, K, N, g)
    T = M + 7
    x = torch.randn(T, K, generator=g).bfloat16()
    gather = torch.randint(0, T, (M,), generator=g, dtype=torch.int32)
    scatter, gammas, betas = torch.randperm(M, generator=g).int(), torch.rand(M, generator=g), torch.rand(M, generator=g)
    bias = torch.randn(E, N, generator=g) * 0.1
    ref = oracle.matmul_oracle(x.float()[gather.long()], wdeq, bias, sizes_t, None, None, betas=betas, out_dtype=torch.float32)
    if act:
        ref = oracle.swiglu_oracle(ref, 1.702, 7.0)
    out = torch.zeros_like(ref)
    out[scatter.long()] = ref * gammas[:, None]
    dev = lambda t: t.to(device)
    pc = tb.PrecisionConfig(b_mx_scale=convert_layout(wrap_torch_tensor(dev(ws)), B200MXScaleLayout()), b_microblock_size=32,
                            out_dtype=torch.float32)
    fa = tb.FusedActivation(tb.FnSpecs("swiglu", tb.swiglu_fn, ("alpha", "limit"), reduction_n=2), (1.702, 7.0)) if act else None
    with tb.scoped_opt_flags_constraints({"kernel": "mx"}):
        y = tb.matmul(dev(x), convert_layout(wrap_torch_tensor(dev(wq), dtype=FP4), B200MXValueLayout()), dev(bias),
                      tb.make_ragged_tensor_metadata(dev(sizes_t), M), None, dev(gather), dev(scatter), pc, betas=dev(betas),
                      gammas=dev(gammas), fused_activation=fa)
    tb.matmul_check_status()
    assert oracle.rel_l2(out, y.cpu()) < 2e-5


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("tiled", [False, True])
def test_pair_kernel_non_finite_tokens(value, tiled, device):
    """A token row with a NaN or an infinity gives a row without finite values; the other rows are untouched."""
    from triton_b200.tensor_details.layout import B200MXScaleLayout, B200MXValueLayout
    g = torch.Generator().manual_seed(4)
    wq, ws, wdeq = quantised_weights(1, 256, 256, g)
    x = torch.randn(64, 256, generator=g).bfloat16()
    x[5, 77] = value
    sizes = torch.tensor([64], dtype=torch.int32)
    if tiled:
        pc = tb.PrecisionConfig(b_mx_scale=convert_layout(wrap_torch_tensor(ws.to(device)), B200MXScaleLayout()), b_microblock_size=32)
        with tb.scoped_opt_flags_constraints({"kernel": "mx"}):
            y = tb.matmul(x.to(device), convert_layout(wrap_torch_tensor(wq.to(device), dtype=FP4), B200MXValueLayout()), None,
                          tb.make_ragged_tensor_metadata(sizes.to(device), 64), precision_config=pc).cpu()
    else:
        y = run_mx(x, wq, ws, sizes, device, block_m=256)
    assert not torch.isfinite(y[5]).any()
    keep = torch.arange(64) != 5
    ref = oracle.matmul_oracle(x[keep].float(), wdeq, None, torch.tensor([63], dtype=torch.int32), out_dtype=torch.float32)
    assert oracle.rel_l2(ref, y[keep].float()) < 1e-2


@pytest.mark.parametrize("tiled", [True, False])
def test_pair_kernel_expert_of_more_rows_than_a_schedule_entry_counts(tiled, device):
    """An entry of the block schedule counts 65536 blocks of 16 rows inside an expert; the rows beyond are packed too.  (Two
    turns of the counter, with experts before and after; one group of k, so that the case is small.)"""
    from triton_b200.tensor_details.layout import B200MXScaleLayout, B200MXValueLayout
    g = torch.Generator().manual_seed(11)
    sizes = [40, 2 * 65536 * 16 + 50, 0, 33]
    E, K, N, M = len(sizes), 32, 64, sum(sizes)
    wq, ws, wdeq = quantised_weights(E, K, N, g)
    gd = torch.Generator(device=device).manual_seed(11)
    x = torch.randn(M, K, device=device, generator=gd).bfloat16()
    md = tb.make_ragged_tensor_metadata(torch.tensor(sizes, dtype=torch.int32, device=device), M)
    if tiled:
        w, s = (convert_layout(wrap_torch_tensor(wq.to(device), dtype=FP4), B200MXValueLayout()),
                convert_layout(wrap_torch_tensor(ws.to(device)), B200MXScaleLayout()))
    else:
        w, s = to_block_scaled(wq, ws, device)
    with tb.scoped_opt_flags_constraints({"kernel": "mx"} if tiled else {"block_m": 256}):
        y = tb.matmul(x, w, None, md, precision_config=tb.PrecisionConfig(b_mx_scale=s, b_microblock_size=32, out_dtype=torch.float32))
    tb.matmul_check_status()
    row = 0
    for e, n in enumerate(sizes):
        ref = x[row:row + n].double() @ wdeq[e].to(device).double()
        if n:
            # an fp32 sum of 32 exact products, the second term's underflow 2^-23 of the group's maximum
            assert ((y[row:row + n] - ref).norm(dim=1) <= 2e-5 * ref.norm(dim=1) + 1e-6).all(), e
        row += n


def test_expected_rows_choose_the_kernel(device):
    """A shard's metadata bounds its rows by those of all ranks; the rows it says to expect decide between the decode and the pair
    kernel (same bits as that kernel asked for by its block)."""
    g = torch.Generator().manual_seed(3)
    E, K, N, sizes = 16, 1024, 1536, [4, 3, 0, 5] * 4
    M = 512
    wq, ws, _ = quantised_weights(E, K, N, g)
    tq, ts = to_block_scaled(wq, ws, device)
    x = torch.randn(M, K, generator=g).bfloat16().to(device)
    y = {}
    for expected, cons in ((None, {}), (None, {"block_m": 256}), (4, {}), (None, {"block_m": 32})):
        md = tb.make_ragged_tensor_metadata(torch.tensor(sizes, dtype=torch.int32, device=device), M)
        md.expected_slice_size = expected
        with tb.scoped_opt_flags_constraints(cons):
            y[expected, tuple(cons.values())] = tb.matmul(x, tq, None, md, precision_config=tb.PrecisionConfig(b_mx_scale=ts, b_microblock_size=32),
                                                          c=torch.zeros(M, N, dtype=torch.bfloat16, device=device))
    tb.matmul_check_status()
    assert torch.equal(y[None, ()], y[None, (256,)]) and torch.equal(y[4, ()], y[None, (32,)])
    assert oracle.rel_l2(y[None, ()].cpu(), y[4, ()].cpu()) < 1e-2


@pytest.mark.parametrize("tiled", [True, False])
@pytest.mark.parametrize("sizes", [[20, 1, 0, 33], [70, 128, 0, 257]])       # terms side by side, and in two MMAs
@pytest.mark.parametrize("mode", ["plain", "scatter", "swiglu", "bf16 out"])
def test_pair_kernel_values_beyond_two_terms(tiled, sizes, mode, device):
    """Rows with an infinity, or a finite value that e4m3 rounds to 2^128, come out as the product of bf16 values gives them: infinite
    with the weight's sign, NaN where the weight is zero or infinities cancel, finite for the finite ones; other rows as ever.
    Against the exact sums in 64 bits, and under SwiGLU (whose limit makes infinities finite) against the bf16 kernel."""
    from triton_b200.tensor_details.layout import B200MXScaleLayout, B200MXValueLayout
    g = torch.Generator().manual_seed(sum(sizes))
    E, K, N, M = len(sizes), 416, 514, sum(sizes)
    sizes_t = torch.tensor(sizes, dtype=torch.int32)
    wq, ws, wdeq = quantised_weights(E, K, N, g)
    T = M + 5
    x = torch.randn(T, K, generator=g).bfloat16()
    gather = torch.randperm(T, generator=g)[:M].int()
    odd = {0: [(7, float("inf"))], sizes[0] - 1: [(415, float("-inf"))], sizes[0]: [(0, 3.3895e38)], M - 1: [(64, float("inf")), (65, float("-inf"))],
           M - 2: [(100, -3.3e38), (300, 1.0)], 3: [(5, float("nan")), (200, float("inf"))]}
    for m, values in odd.items():
        for k, v in values:
            x[gather[m].long(), k] = v
    scatter = torch.randperm(M, generator=g).int() if mode == "scatter" else None
    gammas, betas = (torch.rand(M, generator=g) + 0.5, torch.rand(M, generator=g)) if mode == "scatter" else (None, None)
    if mode == "scatter":
        scatter[0] = -1                                     # a dropped row, one of those with an infinity
    bias = torch.randn(E, N, generator=g) * 0.1
    dev = lambda t: None if t is None else t.to(device)
    dw = convert_layout(wrap_torch_tensor(dev(wq), dtype=FP4), B200MXValueLayout()), convert_layout(wrap_torch_tensor(dev(ws)), B200MXScaleLayout())
    bs = to_block_scaled(wq, ws, device)
    fa = tb.FusedActivation(tb.FnSpecs("swiglu", tb.swiglu_fn, ("alpha", "limit"), reduction_n=2), (1.702, 7.0)) if mode == "swiglu" else None
    out_dtype = torch.bfloat16 if mode == "bf16 out" else torch.float32

    def run(w, s, cons):
        with tb.scoped_opt_flags_constraints(cons):
            y = tb.matmul(dev(x), w, dev(bias), tb.make_ragged_tensor_metadata(dev(sizes_t), M), None, dev(gather), dev(scatter),
                          tb.PrecisionConfig(b_mx_scale=s, b_microblock_size=32, out_dtype=out_dtype), gammas=dev(gammas), betas=dev(betas),
                          fused_activation=fa, c=torch.zeros(M, N // 2 if fa else N, dtype=out_dtype, device=device))
        tb.matmul_check_status()
        return y.cpu()

    y = run(*dw, {"kernel": "mx"}) if tiled else run(*bs, {"block_m": 256})
    if mode == "swiglu":
        want = run(*dw, {"kernel": "tcgen05"}).double()
    else:
        want, row = torch.empty(M, N, dtype=torch.float64), 0
        for e, n in enumerate(sizes):
            beta = 1.0 if betas is None else betas[row:row + n, None].double()
            want[row:row + n] = x[gather[row:row + n].long()].double() @ wdeq[e].double() + bias[e].double() * beta
            row += n
        if mode == "scatter":
            out = torch.zeros_like(want)
            out[scatter[1:].long()] = (want * gammas[:, None].double())[1:]
            want = out
        assert torch.isinf(want).any() and torch.isnan(want).any()
    assert torch.equal(torch.isnan(y), torch.isnan(want)) and torch.equal(torch.isposinf(y), torch.isposinf(want))
    assert torch.equal(torch.isneginf(y), torch.isneginf(want))
    # rows without such values, and those with large finite ones: fp32 sums of exact products (SwiGLU passes them on), relative to
    # the row; 1e-4 leaves room for a gate at the edge of the limit, 2^-8 is bf16's rounding
    for got, ref in zip(y, want):
        keep = torch.isfinite(ref)
        assert (got.double() - ref)[keep].norm() <= (2.0 ** -8 if mode == "bf16 out" else 1e-4) * ref[keep].norm() + 1e-6


@pytest.mark.parametrize("per", [20, 24])
def test_infinities_in_products_of_twenty_rows_per_expert(per, device):
    """By the library's own choice of kernel: a token with an infinity gives infinities with the weight's sign, NaN where the weight is zero."""
    g = torch.Generator().manual_seed(per)
    E, K, N = 40, 448, 1024                                          # two tiles per expert: more than one round of the pairs
    wq, ws, wdeq = quantised_weights(E, K, N, g)
    x = torch.randn(E * per, K, generator=g).bfloat16()
    x[3, 5], x[7 * per, 440] = float("inf"), -float("inf")
    y = run_mx(x, wq, ws, torch.full((E,), per, dtype=torch.int32), device)
    for m, k in ((3, 5), (7 * per, 440)):
        w = wdeq[m // per][k].float() * x[m, k].float().sign()
        want = torch.where(w == 0, torch.nan, w * float("inf"))
        assert torch.equal(y[m].float().nan_to_num(7.0), want.nan_to_num(7.0))
    assert int(torch.isfinite(y).all(1).sum()) == E * per - 2


@pytest.mark.parametrize("form", ["tb16", "tb32", "tb64", "tb32 wide", "tb64 wide", "tb32 two", "tb64 two", "pair", "pair default tiles", "mixed"])
@pytest.mark.parametrize("T, ff", [(3, 320), (70, 736), (200, 320), (1300, 320)])
@pytest.mark.parametrize("kind", ["bf16", "e4m3", "no limit", "inf"])
def test_rows_handed_over_as_tokens(form, T, ff, kind, device):
    """fc1's rows written as fc2's tokens: the bits of the two products run apart.  Odd and even counts of weight blocks (5 and 11.5),
    k steps that are partly past K, one to many token blocks per expert, tiles of one, two and three weight
    blocks (there a chunk has the lines that its block's rows need), both kernels.  Without a limit on the activation the rows go
    through y; a token with an infinity is computed beside the pair kernel and joins the others there.  (1300 tokens: the pair kernel's
    token pass by token, in the operators by position.)"""
    from triton_b200 import _lib
    from triton_b200.moe import _NoTimer, moe_layer_forward
    from triton_b200.testing import make_synthetic_layer
    E, k, d = 6, 2, 512
    if kind == "e4m3" and form in ("tb64", "tb64 wide", "tb64 two", "pair default tiles"):
        pytest.skip("the same paths as with other blocks; e4m3 tokens have no kernel on the default tiles")
    lw = make_synthetic_layer(E, d, ff, device, seed=3, block_scaled=form != "pair default tiles")
    lw.limit = None if kind == "no limit" else 7.0
    g = torch.Generator(device=device).manual_seed(T)
    x = torch.randn(T, d, device=device, generator=g).bfloat16()
    if kind == "inf":
        x[T // 2, 5] = float("inf")
    x = x.to(torch.float8_e4m3fn) if kind == "e4m3" else x
    logits = torch.randn(T, E, device=device, generator=g) + torch.randn(E, device=device, generator=g)
    constraint = {"tb16": {"block_m": 16}, "tb32": {"block_m": 32}, "tb64": {"block_m": 64}, "tb32 wide": {"block_m": 32, "block_n": 384},
                  "tb64 wide": {"block_m": 64, "block_n": 384}, "tb32 two": {"block_m": 32, "block_n": 256},
                  "tb64 two": {"block_m": 64, "block_n": 256}, "pair": {"block_m": 256},
                  "pair default tiles": {"kernel": "mx"}, "mixed": {}}[form]
    lw.block_scaled_max_rows_per_expert = 10 ** 6
    with tb.scoped_opt_flags_constraints(constraint):
        count = _lib.load().moe_launch_count
        c0 = count()
        one = moe_layer_forward(x, logits, lw, k)
        c1 = count()
        many = moe_layer_forward(x, logits, lw, k, gemm_timer=_NoTimer)
        c2 = count()
    tb.matmul_check_status()
    assert torch.equal(one.view(torch.int16), many.view(torch.int16))
    if form != "mixed":
        # routing in one launch in either; the operators build index and weights of the positions by a launch of their own
        assert (c2 - c1) - (c1 - c0) == (1 if kind == "no limit" else 2)
