"""Host-side logic that needs no GPU: layouts (torch ops), block-count bounds, expert assignment, the
expert-parallel exchange plan (also across two gloo ranks), tuning constraints."""
import os

import pytest
import torch
import torch.distributed as dist
import torch.multiprocessing as mp

import oracle
import triton_b200
from triton_b200.distributed import make_exchange_plan, expert_owner
from triton_b200.tensor import FP4, RaggedTensorMetadata, convert_layout, wrap_torch_tensor
from triton_b200.tensor_details.layout import BlackwellMXScaleLayout, BlackwellMXValueLayout, StridedLayout


def test_n_blocks_bound_matches_oracle():
    for E in (1, 7, 128):
        for rows in (0, 1, 5, 127, 128, 129, 4096, 65536):
            for bs in (16, 32, 64, 128):
                assert RaggedTensorMetadata.n_blocks(E, rows, bs) == oracle.n_blocks(E, rows, bs)


def test_reference_layouts_round_trip_on_cpu(golden):
    g = golden("layout_bw")
    s = wrap_torch_tensor(g["scale"])
    sw = convert_layout(s, BlackwellMXScaleLayout())
    assert torch.equal(sw.storage.data, g["scale_swizzled"])
    assert torch.equal(convert_layout(sw, StridedLayout()).storage.data, g["scale"])
    v = wrap_torch_tensor(g["value"], dtype=FP4)                      # canonical: packed along N
    assert v.shape == [2, 96, 40]
    vw = convert_layout(v, BlackwellMXValueLayout())
    assert list(vw.storage.data.shape) == [2, 128, 40] and vw.storage.data.stride(-2) == 1
    assert torch.equal(vw.storage.data[:, :48], g["value_swizzled"][:, :48])
    back = convert_layout(vw, StridedLayout())
    assert torch.equal(back.storage.data, g["value"])
    # K-major strided layout (what downcast_to_mxfp produces for weights)
    km = convert_layout(v, StridedLayout(major_dim=-2))
    assert list(km.storage.data.shape) == [2, 48, 40] and km.storage.data.stride(-2) == 1
    assert torch.equal(km.storage.data, oracle.repack_fp4_oracle(g["value"], -1, -2))


def test_storage_shapes_of_reference_layouts():
    # values from the reference's tests/test_tensor.py:88-109 for the Blackwell layouts
    assert BlackwellMXValueLayout().storage_shape([3, 258, 514], True) == [3, 256, 514]
    assert BlackwellMXScaleLayout().storage_shape([3, 10, 200], False) == [1, 6, 4, 2, 256]


def test_expert_assignment():
    d = triton_b200.make_expt_dict_uniform(4, 128)
    a = triton_b200.make_expt_assignment(4, 128, d, "cpu")
    assert a.expt_boolmask.sum(0).eq(1).all() and a.n_expts_per_shard == [32] * 4
    assert a.expt_map[1, 32:64].tolist() == list(range(32)) and a.expt_map[1, 0] == -1
    assert (a.expt_bitmask[3, 3] & 0xFFFFFFFF) == 0xFFFFFFFF
    r = triton_b200.make_expt_dict_random(4, 37)
    assert sorted(sum(r.values(), [])) == list(range(37)) and all(len(v) for v in r.values())
    with pytest.raises(ValueError):
        triton_b200.make_expt_assignment(2, 4, {0: [0, 1], 1: [1, 2, 3]}, "cpu")
    assert expert_owner(a).tolist() == [e // 32 for e in range(128)]


def _plan_case(T_global=64, E=16, k=4, W=4, seed=0):
    g = torch.Generator().manual_seed(seed)
    logits = torch.randn(T_global, E, generator=g)
    _, indx, _ = oracle.topk_oracle(logits, k)
    _, col, row = oracle.bitmatrix_metadata_oracle(indx, E)
    assign = triton_b200.make_expt_assignment(W, E, triton_b200.make_expt_dict_random(W, E), "cpu")
    return indx, col, row, assign


def test_exchange_plan_is_a_consistent_permutation():
    W, k = 4, 4
    indx, col, row, assign = _plan_case(W=W, k=k)
    T_local = indx.shape[0] // W
    owner = expert_owner(assign)
    order, counts, flat = make_exchange_plan(indx, col, owner, W, T_local)
    assert sorted(order.tolist()) == list(range(indx.numel()))
    assert counts.sum() == indx.numel()
    starts = (torch.cumsum(counts.reshape(-1), 0) - counts.reshape(-1)).view(W, W)
    for s in range(W):
        for d in range(W):
            seg = order[starts[s, d]:starts[s, d] + counts[s, d]]
            assert (seg[1:] > seg[:-1]).all()
            f = col[seg].long()
            assert (f // (k * T_local) == s).all()
            assert (owner[indx.reshape(-1)[f].long()] == d).all()


def _gloo_worker(rank, W, port, ret):
    os.environ["MASTER_ADDR"], os.environ["MASTER_PORT"] = "127.0.0.1", str(port)
    dist.init_process_group("gloo", rank=rank, world_size=W)
    try:
        k, d_model = 2, 8
        indx, col, row, assign = _plan_case(T_global=32, E=8, k=k, W=W, seed=1)
        T_global = indx.shape[0]
        T_local = T_global // W
        x = torch.arange(T_global * d_model, dtype=torch.float32).view(T_global, d_model)
        owner = expert_owner(assign)
        order, counts, flat = make_exchange_plan(indx, col, owner, W, T_local)
        starts = (torch.cumsum(counts.reshape(-1), 0) - counts.reshape(-1)).view(W, W)
        # dispatch, the way convert_dp_to_ep does it, with torch indexing standing in for the CUDA row kernels
        lo, n_send = int(starts[rank, 0]), int(counts[rank].sum())
        tok = flat[lo:lo + n_send] // k
        send = x[tok]
        recv_counts = counts[:, rank].tolist()
        recv = torch.empty(sum(recv_counts), d_model)
        dist.all_to_all_single(recv, send, recv_counts, counts[rank].tolist())
        pos = torch.cat([order[int(starts[s, rank]):int(starts[s, rank]) + recv_counts[s]] for s in range(W)])
        y_ep = torch.full((T_global * k, d_model), float("nan"))
        y_ep[pos] = recv
        # what a single process would have: row p of the expert-sorted buffer is token col[p] // k
        full = x[col.long() // k]
        mine = owner[indx.reshape(-1)[col.long()].long()] == rank
        assert torch.equal(y_ep[mine], full[mine]) and torch.isnan(y_ep[~mine]).all()
        # combine back: every rank returns y_ep * 2 for the rows it owns
        send2 = (y_ep * 2)[pos]
        recv2 = torch.empty(n_send, d_model)
        dist.all_to_all_single(recv2, send2, counts[rank].tolist(), recv_counts)
        out = torch.zeros(T_local * k, d_model)
        out[flat[lo:lo + n_send] - rank * T_local * k] = recv2
        expect = (x[rank * T_local:(rank + 1) * T_local] * 2).repeat_interleave(k, 0)
        assert torch.equal(out, expect)
        ret[rank] = 1
    finally:
        dist.destroy_process_group()


def test_exchange_plan_across_two_gloo_ranks():
    W = 2
    port = 29500 + os.getpid() % 2000
    ctx = mp.get_context("spawn")
    ret = ctx.Manager().dict()
    procs = [ctx.Process(target=_gloo_worker, args=(r, W, port, ret)) for r in range(W)]
    for p in procs:
        p.start()
    for p in procs:
        p.join(120)
    assert all(p.exitcode == 0 for p in procs), [p.exitcode for p in procs]
    assert sorted(ret.keys()) == list(range(W))


def test_opt_flags_constraints_are_scoped():
    from triton_b200.matmul_details import opt_flags
    assert opt_flags.resolve_kernel_choice() == "auto"
    with triton_b200.scoped_opt_flags_constraints({"kernel": "simt", "block_m": 64}):
        assert opt_flags.resolve_kernel_choice() == "simt"
    assert opt_flags.resolve_kernel_choice() == "auto"
    with triton_b200.scoped_opt_flags_constraints({"split_k": 4}):
        with pytest.raises(triton_b200.InapplicableConstraint):
            opt_flags.resolve_kernel_choice()
    # a tile-shape key is honoured or refused, never dropped
    for bad in ({"block_m": 48}, {"block_k": 256}, {"is_persistent": False}, {"num_stages": 3}, {"epilogue_subtile": 2},
                {"no_such_key": 1}, {"idle_sms": -1}):
        with triton_b200.scoped_opt_flags_constraints(bad):
            with pytest.raises(triton_b200.InapplicableConstraint):
                opt_flags.resolve_kernel_choice()
    with triton_b200.scoped_opt_flags_constraints({"block_m": 32, "block_n": 384, "block_k": 128, "split_k": 1,
                                                   "is_persistent": True, "num_stages": None, "idle_sms": 8}):
        assert opt_flags.resolve_kernel_choice() == "auto"
        assert opt_flags.resolve_tile_m() == 32 and opt_flags.resolve_tile_n() == 384 and opt_flags.get_idle_sms() == 8
    assert opt_flags.get_idle_sms() == 0


def test_balanced_expert_placement():
    """Equal counts per shard, every expert placed once, and a far better balance than contiguous blocks on a skewed load."""
    import random
    from triton_b200.distributed import make_expt_dict_balanced, make_expt_dict_uniform
    rng = random.Random(0)
    load = [2.718 ** rng.gauss(0, 1) for _ in range(128)]
    for shards in (2, 4, 8):
        d = make_expt_dict_balanced(shards, 128, load)
        assert sorted(e for v in d.values() for e in v) == list(range(128))
        assert all(len(v) == 128 // shards for v in d.values())
        spread = lambda dd: max(sum(load[e] for e in v) for v in dd.values()) / (sum(load) / shards)
        assert spread(d) < 1.02 <= spread(make_expt_dict_uniform(shards, 128)) + 1e-9 or spread(d) < 1.02
        assert spread(d) <= spread(make_expt_dict_uniform(shards, 128))


def test_shuffled_value_layout_matches_reference_fixture(golden):
    """BlackwellMX4ValueShuffledLayout against the reference's own output (two tilings, K and N both padded)."""
    from triton_b200.tensor_details.layout import BlackwellMX4ValueShuffledLayout
    g = golden("layout_bw2")
    v = wrap_torch_tensor(g["value"], dtype=FP4)                      # canonical [E, K, N/2]
    assert v.shape == [2, 200, 300]
    for (bk, bn), key in (((128, 256), "value_shuffled_128_256"), ((64, 128), "value_shuffled_64_128")):
        lay = BlackwellMX4ValueShuffledLayout(block_k=bk, block_n=bn)
        sw = convert_layout(v, lay)
        assert list(sw.storage.data.shape) == list(g[key].shape)
        assert torch.equal(sw.storage.data, g[key])
        assert torch.equal(convert_layout(sw, StridedLayout()).storage.data, g["value"])
    # the reference's storage-shape known answers (tests/test_tensor.py:99-100, 103-105)
    from triton_b200.tensor_details.layout import BlackwellActMXScaleLayout
    assert BlackwellMX4ValueShuffledLayout().make_transformation([3, 258, 514], True).storage_shape == [3, 4, 3, 256, 64]
    assert BlackwellMX4ValueShuffledLayout().make_transformation([0, 64], True).storage_shape == [1, 0, 1, 256, 64]
    assert BlackwellActMXScaleLayout(None).make_transformation([130, 65], False).storage_shape == [1, 2, 18, 2, 256]
    assert BlackwellActMXScaleLayout(None).make_transformation([3, 130, 65], False).storage_shape == [1, 6, 18, 2, 256]
    assert BlackwellActMXScaleLayout(None).make_transformation([0, 64], False).storage_shape == [1, 0, 16, 2, 256]


def test_act_scale_layout_matches_reference_fixture_and_oracle(golden):
    from triton_b200.tensor_details.layout import BlackwellActMXScaleLayout
    g = golden("layout_bw2")
    a = wrap_torch_tensor(g["act_scale"])
    sw = convert_layout(a, BlackwellActMXScaleLayout(None))
    assert torch.equal(sw.storage.data, g["act_scale_swizzled"])
    assert torch.equal(convert_layout(sw, StridedLayout()).storage.data, g["act_scale"])
    # ragged: every slice starts at a new block of 128 rows; rows past the slices are dropped
    sizes = torch.tensor([130, 0, 5, 128, 20], dtype=torch.int32)
    M = int(sizes.sum()) + 17
    gen = torch.Generator().manual_seed(4)
    s = torch.randint(0, 255, (M, 12), generator=gen, dtype=torch.uint8)
    offs = torch.zeros(6, dtype=torch.int32)
    offs[1:] = torch.cumsum(sizes, 0)
    nb = [[0] * 6 for _ in range(4)]
    for b, bs in enumerate((16, 32, 64, 128)):
        run = 0
        for e in range(5):
            nb[b][e] = run
            run += (int(sizes[e]) + bs - 1) // bs
        nb[b][5] = run
    md = RaggedTensorMetadata(sizes, offs, torch.tensor(nb, dtype=torch.int32),
                              torch.zeros((4, RaggedTensorMetadata.max_n_blocks(5, M)), dtype=torch.int32))
    lay = BlackwellActMXScaleLayout(md)
    sw = convert_layout(wrap_torch_tensor(s), lay)
    assert torch.equal(sw.storage.data, oracle.swizzle_act_mx_scale_oracle(s, sizes.tolist()))
    back = convert_layout(sw, StridedLayout()).storage.data
    assert torch.equal(back[: int(sizes.sum())], s[: int(sizes.sum())]) and not back[int(sizes.sum()):].any()


def test_default_weight_layout_arguments():
    from triton_b200.tensor_details.layout import (B200MXScaleLayout, B200MXValueLayout, make_default_matmul_mxfp4_w_layout,
                                                   make_default_matmul_mxfp4_w_scale_layout)
    assert isinstance(make_default_matmul_mxfp4_w_layout(mx_axis=-2, allow_blackwell_value_shuffle=True), B200MXValueLayout)
    assert isinstance(make_default_matmul_mxfp4_w_scale_layout(mx_axis=1), B200MXScaleLayout)
    with pytest.raises(NotImplementedError):
        make_default_matmul_mxfp4_w_layout(mx_axis=-1)


def test_weight_file_round_trip_on_cpu(tmp_path):
    """save_layer_weights / load_layer_weights: every tensor comes back byte for byte, in the layout it was saved in."""
    from triton_b200.moe import MoeLayerWeights
    from triton_b200.tensor import Storage, Tensor
    from triton_b200.tensor_details.layout import (B200BlockScaledScaleLayout, B200BlockScaledValueLayout, B200MXScaleLayout,
                                                   B200MXValueLayout)
    from triton_b200.weights_io import load_layer_weights, read_header, save_layer_weights
    g = torch.Generator().manual_seed(0)
    E, K, N = 3, 256, 384

    def tiled(layout, logical, nbytes, fp4):
        data = torch.randint(0, 256, (nbytes,), generator=g, dtype=torch.uint8)
        return Tensor(Storage(data, layout), dtype=FP4 if fp4 else triton_b200.tensor.UINT8, shape=logical)

    nv, ns = E * 2 * 3 * 8192, E * 2 * 3 * 512
    lw = MoeLayerWeights(tiled(B200MXValueLayout(), [E, K, N], nv, True), tiled(B200MXScaleLayout(), [E, K // 32, N], ns, False),
                         torch.randn(E, N, generator=g).bfloat16(),
                         tiled(B200MXValueLayout(), [E, N // 2, K], E * 2 * 2 * 8192, True),
                         tiled(B200MXScaleLayout(), [E, N // 64, K], E * 2 * 2 * 512, False),
                         torch.randn(E, K, generator=g).bfloat16(), alpha=1.5, limit=None,
                         w1_bs=tiled(B200BlockScaledValueLayout(), [E, K, N], nv, True),
                         w1_bs_scale=tiled(B200BlockScaledScaleLayout(), [E, K // 32, N], ns, False))
    path = tmp_path / "layer.moeb200w"
    size = save_layer_weights(path, lw)
    assert path.stat().st_size == size and size % 4096 == 0
    hdr = read_header(path)
    assert all(e["offset"] % 4096 == 0 for e in hdr["tensors"].values()) and "w2_bs" not in hdr["tensors"]
    back = load_layer_weights(path, "cpu")
    assert back.alpha == 1.5 and back.limit is None and back.w2_bs is None
    for name in ("w1", "w1_scale", "w2", "w2_scale", "w1_bs", "w1_bs_scale"):
        a, b = getattr(lw, name), getattr(back, name)
        assert type(a.storage.layout) is type(b.storage.layout) and a.shape == b.shape and a.dtype == b.dtype
        assert torch.equal(a.storage.data, b.storage.data)
    assert torch.equal(lw.b1, back.b1) and torch.equal(lw.b2, back.b2)
    bad = tmp_path / "bad.bin"
    bad.write_bytes(b"not a weight file at all")
    with pytest.raises(ValueError):
        read_header(bad)


@pytest.mark.parametrize("T, E", [(50, 128), (1, 5), (33, 40), (32, 32)])
def test_bit_tensor_equals_the_checked_construction(T, E):
    """The mask every routing call makes without checks is the one `wrap_torch_tensor` returns."""
    from triton_b200.tensor import BIT, bit_tensor
    words, t_pad = (E + 31) // 32, (T + 31) // 32 * 32
    bm = torch.zeros(words, t_pad, dtype=torch.int32).transpose(0, 1)[:T]
    got, want = bit_tensor(bm, T, E), wrap_torch_tensor(bm, dtype=BIT, shape=[T, E], shape_max=[T, None])
    assert (got.shape, got.shape_max, got.dtype, got.storage.layout) == (want.shape, want.shape_max, want.dtype, want.storage.layout)
    assert got.storage.data is bm


def _layer_on_cpu(E=3, d=64, ff=96, block_scaled=True):
    from triton_b200.moe import MoeLayerWeights
    from triton_b200.tensor import UINT8, Storage, Tensor
    from triton_b200.tensor_details.layout import (B200BlockScaledScaleLayout, B200BlockScaledValueLayout, B200MXScaleLayout,
                                                   B200MXValueLayout)

    def pair(K, N, value, scale):
        n = E * ((K + 127) // 128) * ((N + 127) // 128)
        return (Tensor(Storage(torch.zeros(n * 8192, dtype=torch.uint8), value), dtype=FP4, shape=[E, K, N]),
                Tensor(Storage(torch.zeros(n * 512, dtype=torch.uint8), scale), dtype=UINT8, shape=[E, K // 32, N]))

    w1, s1 = pair(d, 2 * ff, B200MXValueLayout(), B200MXScaleLayout())
    w2, s2 = pair(ff, d, B200MXValueLayout(), B200MXScaleLayout())
    lw = MoeLayerWeights(w1, s1, torch.zeros(E, 2 * ff), w2, s2, torch.zeros(E, d))
    if block_scaled:
        lw.w1_bs, lw.w1_bs_scale = pair(d, 2 * ff, B200BlockScaledValueLayout(), B200BlockScaledScaleLayout())
        lw.w2_bs, lw.w2_bs_scale = pair(ff, d, B200BlockScaledValueLayout(), B200BlockScaledScaleLayout())
    return lw


@pytest.mark.parametrize("block_scaled", [False, True])
@pytest.mark.parametrize("fault", ["narrow b1", "narrow b2", "short b2", "width of w1", "depth of w2", "scale layout", "second scale layout"])
def test_layer_in_one_call_leaves_unfitting_weights_to_the_operators(block_scaled, fault):
    """The native layer step takes extents and layouts on trust, so only weights whose parts fit one another reach it; the
    operators, which check them, take the rest."""
    from triton_b200.moe import _one_call
    from triton_b200.tensor import Storage, Tensor
    from triton_b200.tensor_details.layout import StridedLayout
    lw, x, logits = _layer_on_cpu(block_scaled=block_scaled), torch.zeros(5, 64, dtype=torch.bfloat16), torch.zeros(5, 3)
    assert _one_call(x, logits, lw, 2)
    if block_scaled:
        assert _one_call(x.to(torch.float8_e4m3fn), logits, lw, 2)
    else:
        assert not _one_call(x.to(torch.float8_e4m3fn), logits, lw, 2)
    end = "_bs" if block_scaled else ""
    reshaped = lambda t, shape: Tensor(t.storage, dtype=t.dtype, shape=shape)
    if fault == "narrow b1":
        lw.b1 = lw.b1[:, :-1].contiguous()
    elif fault == "narrow b2":
        lw.b2 = lw.b2[:, :-1].contiguous()
    elif fault == "short b2":
        lw.b2 = lw.b2[:-1]
    elif fault == "width of w1":
        setattr(lw, "w1" + end, reshaped(getattr(lw, "w1" + end), [3, 64, 2 * 96 - 2]))
    elif fault == "depth of w2":
        setattr(lw, "w2" + end, reshaped(getattr(lw, "w2" + end), [3, 64, 64]))
    else:
        name = ("w1" if fault == "scale layout" else "w2") + end + "_scale"
        t = getattr(lw, name)
        setattr(lw, name, Tensor(Storage(t.storage.data, StridedLayout()), dtype=t.dtype, shape=t.shape))
    assert not _one_call(x, logits, lw, 2)


@pytest.mark.parametrize("block_scaled", [False, True])
def test_tiling_reads_storage_in_place_only_where_it_has_the_stated_shape(block_scaled):
    """A tensor may be stated larger than its storage (one expert's bytes standing for several): the kernel that reads the storage
    in place must not take it, the canonical form that broadcasts it does."""
    from triton_b200.tensor_details.layout import (B200BlockScaledScaleLayout, B200BlockScaledValueLayout, B200MXScaleLayout,
                                                   B200MXValueLayout)
    E, K, N = 3, 64, 40
    value, scale = (B200BlockScaledValueLayout(), B200BlockScaledScaleLayout()) if block_scaled else (B200MXValueLayout(), B200MXScaleLayout())
    tv, ts = value.make_transformation([E, K, N], True), scale.make_transformation([E, K // 32, N], False)
    q = torch.zeros(E, N, K // 2, dtype=torch.uint8).transpose(1, 2)
    s = torch.zeros(E, N, K // 32, dtype=torch.uint8).transpose(1, 2)
    order = StridedLayout(major_dim=-2).order(3)
    for bad in (q[:1], q[0], q[:, :16], q[:, :, :-1], q.to(torch.int16)):
        assert tv.swizzle_strided(bad, order) is None
    for bad in (s[:1], s[0], s[:, :1], s[:, :, :-1], s.float()):
        assert ts.swizzle_strided(bad, order) is None
    for good, t in ((q, tv), (s, ts)):
        with pytest.raises(ValueError, match="CUDA tensors only"):      # goes to the kernel
            t.swizzle_strided(good, order)


@pytest.mark.parametrize("limit", [0, 16, 47, 49, 100, 10000])
def test_block_scaled_row_limit_is_the_callers(limit):
    """A limit the caller sets decides alone, at any width; the default goes on by shape beyond its 48 rows per expert."""
    for ff, d in ((96, 64), (2880, 2880)):
        lw = _layer_on_cpu(E=3, d=d, ff=ff)
        for rows in (1, 48, 49, 64, 80, 81, 100, 300, 5000):
            assert lw.use_block_scaled(rows * 3) == (rows <= 80 or (ff == 2880 and rows >= 81))
        lw.block_scaled_max_rows_per_expert = limit
        for rows in (1, 16, 17, 47, 48, 49, 64, 80, 81, 100, 101, 300, 5000):
            assert lw.use_block_scaled(rows * 3) == (rows <= limit)
            assert (lw.fc_weights(rows * 3)[0] is lw.w1_bs) == (lw.fc_weights(rows * 3)[2] is lw.w2_bs) == (rows <= limit)


def test_weights_of_a_step_under_a_tuning_constraint():
    """Beyond the row limit a constraint that names a bf16 kernel or a tile keeps a step on the default copy; up to the limit, and
    under any other constraint, the choice is the one without it."""
    lw = _layer_on_cpu(E=3, d=2880, ff=2880)
    pinned = [{"kernel": k} for k in ("tcgen05", "tcgen05-pair", "stream", "simt")] + [{"block_m": 128}, {"block_m": 256}, {"block_n": 256}]
    free = [{}, {"kernel": "auto"}, {"idle_sms": 8}, {"kernel": "mx"}, {"block_m": None}]
    for cons in pinned + free:
        with triton_b200.scoped_opt_flags_constraints(cons):
            for rows in (1, 48, 49, 64, 300, 2048):
                assert lw.use_block_scaled(rows * 3) == (rows <= 48 or cons in free), (cons, rows)


def test_kernels_of_a_step():
    """The library names the kernel its dispatch takes: the figures beside the rules, on either weight copy."""
    both, default = _layer_on_cpu(E=3, d=2880, ff=2880), _layer_on_cpu(E=3, d=2880, ff=2880, block_scaled=False)
    decode, pair, tc = "gemm_mx_kernel", "gemm_mx_pair_kernel", "gemm_tc_kernel"
    assert both.kernels(3 * 8) == (decode,) * 2 and both.kernels(3 * 19) == (decode,) * 2
    assert both.kernels(3 * 20) == (pair,) * 2 and both.kernels(3 * 1000) == (pair,) * 2
    assert both.kernels(3 * 15, torch.float8_e4m3fn) == (decode,) * 2 and both.kernels(3 * 16, torch.float8_e4m3fn) == (pair,) * 2
    assert default.kernels(3 * 20) == (pair,) * 2 and default.kernels(3 * 1000) == (pair,) * 2
    small = _layer_on_cpu(E=3, d=512, ff=512, block_scaled=False)
    assert small.kernels(3 * 10) == ("gemm_stream_kernel",) * 2 and small.kernels(3 * 64) == (tc,) * 2
    narrow = _layer_on_cpu(E=3, d=2048, ff=2880, block_scaled=False)
    assert narrow.kernels(3 * 511) == (pair,) * 2 and narrow.kernels(3 * 512) == (pair, tc)
    with triton_b200.scoped_opt_flags_constraints({"kernel": "tcgen05"}):
        assert both.kernels(3 * 100) == (tc,) * 2
        with pytest.raises(triton_b200.InapplicableConstraint):
            both.kernels(3 * 8)


def test_kernel_of_a_shard_goes_by_its_own_rows(monkeypatch):
    """Eight ranks, 16 experts each, 512 routed rows in all: four rows per expert, not the 32 that the bound on the rows suggests."""
    from triton_b200 import _lib, moe
    kernel = lambda kind, M, rows: _lib.host().gemm_kernel(kind, 16, 2880, 5760, M, torch.bfloat16, torch.bfloat16, (0, 0, 0, 0), rows)
    mx, default = _lib.MOE_W_MX4_B200MX, _lib.MOE_W_MX4_B200
    assert kernel(mx, 512, 0) == "gemm_mx_pair_kernel" and kernel(mx, 512, 4) == kernel(mx, 64, 0) == "gemm_mx_kernel"
    assert kernel(mx, 512, 1000) == kernel(mx, 512, 0)                  # never above what the bound allows
    assert kernel(default, 8 * 512 * 16, 512) == kernel(default, 512 * 16, 0) == "gemm_mx_pair_kernel"
    md = triton_b200.RaggedTensorMetadata(*(torch.zeros(s, dtype=torch.int32) for s in ((2,), (3,), (4, 3), (4, 3))))
    monkeypatch.setattr(moe, "remap_ragged_tensor_metadata", lambda meta, table: md)
    assert moe._local_metadata(None, None, 512 // 8, 16).expected_slice_size == 4
    assert moe._local_metadata(None, None, 1, 16).expected_slice_size == 1


@pytest.mark.parametrize("E, K, N", [(32, 2880, 5760), (32, 2880, 2880), (64, 512, 1024), (64, 1440, 2880), (128, 2880, 5760)])
def test_infinities_are_kept_from_twenty_rows_per_expert_on(E, K, N):
    """Large bf16 products run from there on the kernel whose token pass holds rows with an infinity, however many rounds its tiles take."""
    from triton_b200 import _lib
    kernel = lambda per: _lib.host().gemm_kernel(_lib.MOE_W_MX4_B200MX, E, K, N, E * per, torch.bfloat16, torch.bfloat16, (0, 0, 0, 0))
    assert kernel(19) == "gemm_mx_kernel" and {kernel(per) for per in range(20, 48)} == {"gemm_mx_pair_kernel"}


def test_small_block_scaled_products_leave_the_decode_kernel_after_one_wave():
    """Below 2^24 elements the decode kernel keeps a product while its 32 x 128 tiles fit the SMs (148 of them where no GPU says
    otherwise): 32 experts of 512 x 512 up to some 16 rows per expert, 8 experts of 2048 x 512 to well beyond 96."""
    from triton_b200 import _lib
    if torch.cuda.is_available() and torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("sizes are those of 148 SMs")
    kernel = lambda E, K, N, per: _lib.host().gemm_kernel(_lib.MOE_W_MX4_B200MX, E, K, N, E * per, torch.bfloat16, torch.bfloat16, (0, 0, 0, 0))
    decode, pair = "gemm_mx_kernel", "gemm_mx_pair_kernel"
    assert kernel(32, 512, 512, 16) == decode and kernel(32, 512, 512, 32) == kernel(32, 512, 512, 64) == pair
    assert kernel(8, 512, 2048, 16) == decode and kernel(8, 512, 2048, 32) == kernel(8, 512, 2048, 80) == pair
    assert kernel(8, 2048, 512, 96) == kernel(8, 2048, 512, 128) == decode and kernel(8, 2048, 512, 160) == pair
    assert kernel(1, 512, 512, 1000) == decode and kernel(1, 512, 512, 1200) == pair


def test_wide_swiglu_product_over_few_k_stays_with_the_bf16_kernel():
    """From 512 rows per expert on, and only behind SwiGLU (fc1): a layer of 512 x 4096 with either weight copy."""
    for lw in (_layer_on_cpu(E=16, d=512, ff=2048, block_scaled=False), _layer_on_cpu(E=16, d=512, ff=2048)):
        assert lw.kernels(16 * 511)[0] == "gemm_mx_pair_kernel" and lw.kernels(16 * 512)[0] == "gemm_tc_kernel"
    wide = _layer_on_cpu(E=4, d=1024, ff=2048)
    assert wide.kernels(4 * 1024)[0] == "gemm_mx_pair_kernel"
    from triton_b200 import _lib
    plain = _lib.host().gemm_kernel(_lib.MOE_W_MX4_B200, 16, 512, 4096, 16 * 1024, torch.bfloat16, torch.bfloat16, (0, 0, 0, 0))
    assert plain == "gemm_mx_pair_kernel"


def test_kernels_read_nothing_of_the_chain_ahead_of_their_wait():
    """Memory that earlier kernels of the stream wrote is visible behind griddepcontrol.wait and not before.  Every kernel that waits does so
    with all its threads, in one place, and ahead of it touches neither metadata, operands nor weights, but for hints to L2."""
    import pathlib
    import re
    csrc = pathlib.Path(triton_b200.__file__).parent / "csrc"
    waiting, launched = set(), set()
    for path in sorted(csrc.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        launched |= set(re.findall(r"launch_pdl\(\s*(?:pack|(\w+))", text)) - {""}
        for m in re.finditer(r"__global__ void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\(", text):
            body = text[m.end():]
            body = body[:body.index("\n}\n")]
            if "pdl_" not in body:
                continue
            waiting.add(m.group(1))
            assert re.findall(r"\n( *)pdl_begin\(\);", body) == ["  "] and "pdl_wait" not in body, f"{path.name}: {m.group(1)}"
            ahead = body[body.index("{"):body.index("pdl_begin();")]
            reads = r"slice_sizes|slice_offs|block_offs|block_sched|p\.bias|gather|pair_prefix|map_block|map_ptile|elect_(tile|bulk|expect)|ld_?global|__ldg|cp_async"
            assert not re.search(reads, ahead), f"{path.name}: {m.group(1)}: {re.search(reads, ahead).group(0)}"
    assert launched <= waiting and {"gemm_mx_kernel", "gemm_mx_pair_kernel", "router_topk_kernel", "route_cluster_kernel"} <= waiting


def test_kernels_take_tensor_memory_before_they_let_the_next_one_go():
    """A kernel that lets its dependents go and then asks for tensor memory can find it taken by one of them, which waits for this kernel's end: all
    warps meet between the allocation and the release."""
    import pathlib
    import re
    csrc = pathlib.Path(triton_b200.__file__).parent / "csrc"
    found = set()
    for path in sorted(csrc.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__ void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\(", text):
            body = text[m.end():]
            body = body[:body.index("\n}\n")]
            if "tcgen05.alloc" not in body or "pdl_begin" not in body:
                continue
            found.add(m.group(1))
            assert body.count("tcgen05.alloc") == 1
            assert "__syncthreads();" in body[body.index("tcgen05.alloc"):].split("pdl_begin();")[0], m.group(1)
            assert body.index("tcgen05.alloc") < body.index("pdl_begin();"), m.group(1)
    assert {"gemm_tc_kernel", "gemm_mx_kernel", "gemm_mx_pair_kernel", "router_topk_kernel"} <= found
