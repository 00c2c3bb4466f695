"""Routing on the GPU (top-k + bitmatrix, histogram + expert-major sort, ragged metadata, remap),
bit-exact against the reference fixtures and the CPU oracle."""
import pytest
import torch

import oracle
from triton_b200 import _lib
from triton_b200 import (make_bitmatrix_metadata, make_ragged_tensor_metadata, remap_ragged_tensor_metadata, routing,
                         topk)
from triton_b200.tensor import BIT, RaggedTensorMetadata, wrap_torch_tensor

pytestmark = pytest.mark.gpu


def check_topk(logits_cpu, k, softmax, device, n_rows=None):
    sp = topk(logits_cpu.to(device), k, apply_softmax=softmax, n_rows=n_rows)
    vals, indx, bm = oracle.topk_oracle(logits_cpu, k, softmax, n_rows=n_rows)
    nr = logits_cpu.shape[0] if n_rows is None else n_rows
    assert sp.indx.dtype == torch.int16
    assert torch.equal(sp.indx[:nr].cpu().int(), indx[:nr])
    T, E = logits_cpu.shape
    data = sp.mask.storage.data
    assert data.shape == (T, (E + 31) // 32) and data.stride() == (1, (T + 31) // 32 * 32)
    assert torch.equal(data[:nr].cpu(), bm[:nr])
    if softmax:
        torch.testing.assert_close(sp.vals[:nr].cpu().float(), vals[:nr].float(), atol=2e-6, rtol=2e-5)
    else:
        assert torch.equal(sp.vals[:nr].cpu(), vals[:nr])
    return sp, indx


@pytest.mark.parametrize("name", ["topk_T7_E13_k4", "topk_T256_E128_k4", "topk_T300_E200_k8", "topk_T33_E32_k2"])
def test_against_reference_fixture(golden, name, device):
    g = golden(name)
    sp = topk(g["logits"].to(device), g["k"], apply_softmax=bool(g["softmax"]))
    assert torch.equal(sp.indx.cpu().int(), g["indx"].int())
    assert torch.equal(sp.mask.storage.data.cpu(), g["bitmatrix"])
    torch.testing.assert_close(sp.vals.cpu(), g["vals"], atol=2e-6, rtol=2e-5)
    md = sp.mask_metadata
    assert torch.equal(md.col_sum.cpu(), g["col_sum"].int())
    assert torch.equal(md.col_sorted_indx.cpu(), g["col_sorted"])
    assert torch.equal(md.row_sorted_indx.cpu(), g["row_sorted"])


@pytest.mark.parametrize("T", [1, 7, 256, 300])
@pytest.mark.parametrize("E", [13, 32, 128, 200])
@pytest.mark.parametrize("softmax", [True, False])
def test_topk_grid(T, E, softmax, device):
    # reference tests/test_topk.py:11-29 (k = 8)
    torch.manual_seed(T * 1000 + E)
    logits = torch.randn(T, E)
    logits[:, min(3, E - 1)] = logits[:, 0]              # ties
    check_topk(logits, 8, softmax, device)


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
def test_topk_low_precision_logits(dt, device):
    torch.manual_seed(1)
    logits = torch.randn(65, 64).to(dt)                  # many exact ties after rounding
    sp = topk(logits.to(device), 4, apply_softmax=False)
    vals, indx, bm = oracle.topk_oracle(logits, 4, False)
    assert torch.equal(sp.indx.cpu().int(), indx) and torch.equal(sp.vals.cpu(), vals)


def test_topk_n_rows_and_provided_indx(device):
    torch.manual_seed(2)
    logits = torch.randn(100, 40)
    sp, indx = check_topk(logits, 4, True, device, n_rows=61)
    md = sp.mask_metadata
    cs, col, row = oracle.bitmatrix_metadata_oracle(indx, 40)
    assert torch.equal(md.col_sum.cpu(), cs)
    assert torch.equal(md.col_sorted_indx.cpu(), col) and torch.equal(md.row_sorted_indx.cpu(), row)
    yi = torch.stack([torch.randperm(40)[:4] for _ in range(100)]).to(torch.int16)
    sp2 = topk(logits.to(device), 4, apply_softmax=True, y_indx=yi.to(device))
    vals, indx2, bm = oracle.topk_oracle(logits, 4, True, y_indx=yi)
    assert torch.equal(sp2.indx.cpu(), yi) and torch.equal(sp2.mask.storage.data.cpu(), bm)
    torch.testing.assert_close(sp2.vals.cpu(), vals, atol=2e-6, rtol=2e-5)


@pytest.mark.parametrize("T", [7, 256, 17111])
@pytest.mark.parametrize("E", [13, 32, 128, 811])
@pytest.mark.parametrize("k", [1, 4, 8])
def test_bitmatrix_metadata_grid(T, E, k, device):
    # reference tests/test_tensor.py:280-302
    torch.manual_seed(T + E + k)
    indx = torch.stack([torch.randperm(E)[:k] for _ in range(min(T, 512))])
    indx = indx.repeat((T + indx.shape[0] - 1) // indx.shape[0], 1)[:T]
    indx = indx[torch.randperm(T)].to(torch.int16)
    bm = wrap_torch_tensor(torch.empty((T, (E + 31) // 32), dtype=torch.int32, device=device), dtype=BIT, shape=[T, E])
    md = make_bitmatrix_metadata(indx.to(device), bm)
    cs, col, row = oracle.bitmatrix_metadata_oracle(indx.int(), E)
    assert torch.equal(md.col_sum.cpu(), cs)
    assert torch.equal(md.row_sorted_indx.cpu(), row)
    assert torch.equal(md.col_sorted_indx.cpu(), col)


@pytest.mark.parametrize("T, E, k", [(1, 1, 1), (600, 1024, 2), (300, 1025, 2), (700, 2500, 1), (33000, 128, 1), (20000, 3, 2)])
def test_expert_sort_at_the_segments_of_its_scan(T, E, k, device):
    # one block scans: experts 1024 at a time, the blocks of tokens in 1024 / E segments of up to (and past) sixteen
    torch.manual_seed(T + E)
    indx = torch.stack([torch.randperm(E)[:k] for _ in range(T)]).short()
    col_sum, col, row = _lib.host().bitmatrix_metadata(indx.to(device), E, None)
    o_sum, o_col, o_row = oracle.bitmatrix_metadata_oracle(indx, E)
    assert torch.equal(col_sum.cpu(), o_sum.int()) and torch.equal(col.cpu(), o_col.int()) and torch.equal(row.cpu(), o_row.int())


@pytest.mark.parametrize("T, E, k, n_rows", [(1, 1, 1, None), (7, 3, 2, 5), (9, 256, 1, None), (8192, 256, 4, None), (8193, 256, 4, None),
                                             (10922, 20, 3, 10000), (3000, 33, 5, 0)])
def test_expert_sort_in_one_launch(T, E, k, n_rows, device):
    # up to 32768 entries: whole and partial shares of 1024, dropped entries and rows past a device-side bound
    torch.manual_seed(T + E)
    indx = torch.randint(-1 if E > 3 else 0, E, (T, k)).short()
    bound = None if n_rows is None else torch.tensor([n_rows], dtype=torch.int32, device=device)
    col_sum, col, row = _lib.host().bitmatrix_metadata(indx.to(device), E, bound)
    kept = indx.clone()
    kept[T if n_rows is None else n_rows:] = -1
    o_sum, o_col, o_row = oracle.bitmatrix_metadata_oracle(kept, E)
    assert torch.equal(col_sum.cpu(), o_sum.int()) and torch.equal(col.cpu(), o_col.int()) and torch.equal(row.cpu(), o_row.int())


@pytest.mark.parametrize("n_slices", [1, 7, 33, 911, 1025])
def test_ragged_metadata_and_remap(n_slices, device):
    # reference tests/test_tensor.py:243-277
    torch.manual_seed(n_slices)
    sizes = torch.randint(0, 300, (n_slices,), dtype=torch.int32)
    sizes[torch.randint(0, n_slices, (1,))] = 0
    n_rows = int(sizes.sum()) + 100
    md = make_ragged_tensor_metadata(sizes.to(device), n_rows)
    so, bo, bs = oracle.ragged_metadata_oracle(sizes, n_rows)
    assert torch.equal(md.slice_offs.cpu(), so)
    assert torch.equal(md.block_offs_data.cpu(), bo)
    assert torch.equal(md.block_schedule_data.cpu(), bs)
    assert md.block_schedule_data.shape[1] == RaggedTensorMetadata.max_n_blocks(n_slices, n_rows)
    smap = torch.full((n_slices,), -1, dtype=torch.int32)
    keep = torch.randperm(n_slices)[: max(1, n_slices - 5)].sort().values
    smap[keep] = torch.randperm(keep.numel()).int()
    r = remap_ragged_tensor_metadata(md, smap.to(device))
    ro = oracle.remap_ragged_metadata_oracle(sizes, so, bo, bs, smap)
    assert torch.equal(r.slice_sizes.cpu(), ro[0]) and torch.equal(r.slice_offs.cpu(), ro[1])
    assert torch.equal(r.block_offs_data.cpu(), ro[2]) and torch.equal(r.block_schedule_data.cpu(), ro[3])


@pytest.mark.parametrize("name", ["ragged_E1", "ragged_E7", "ragged_E33", "ragged_E130"])
def test_ragged_against_reference_fixture(golden, name, device):
    g = golden(name)
    md = make_ragged_tensor_metadata(g["slice_sizes"].to(device), g["n_rows"])
    assert torch.equal(md.slice_offs.cpu(), g["slice_offs"])
    assert torch.equal(md.block_offs_data.cpu(), g["block_offs"])
    assert torch.equal(md.block_schedule_data.cpu(), g["block_schedule"])
    r = remap_ragged_tensor_metadata(md, g["slice_map"].to(device))
    assert torch.equal(r.slice_sizes.cpu(), g["r_slice_sizes"]) and torch.equal(r.slice_offs.cpu(), g["r_slice_offs"])
    assert torch.equal(r.block_offs_data.cpu(), g["r_block_offs"])
    assert torch.equal(r.block_schedule_data.cpu(), g["r_block_schedule"])


def test_routing_full_size(device):
    """fp32 logits [16384, 128], top-4 + softmax: indices, histogram and both index arrays equal the oracle's;
    the two index arrays are inverse permutations and the sort is expert-major and stable."""
    torch.manual_seed(0)
    logits = torch.randn(16384, 128)
    ragged, gather_idx, scatter_idx, sp = routing(logits.to(device), 4)
    vals, indx, bm = oracle.topk_oracle(logits, 4, True)
    assert torch.equal(sp.indx.cpu().int(), indx) and torch.equal(sp.mask.storage.data.cpu(), bm)
    cs, col, row = oracle.bitmatrix_metadata_oracle(indx, 128)
    md = sp.mask_metadata
    assert torch.equal(md.col_sum.cpu(), cs) and torch.equal(md.col_sorted_indx.cpu(), col)
    assert torch.equal(md.row_sorted_indx.cpu(), row)
    assert torch.equal(md.row_sorted_indx[md.col_sorted_indx.long()].cpu(), torch.arange(65536, dtype=torch.int32))
    e_sorted = sp.indx.reshape(-1)[md.col_sorted_indx.long()].int()
    assert (e_sorted[1:] >= e_sorted[:-1]).all()
    same = e_sorted[1:] == e_sorted[:-1]
    assert (md.col_sorted_indx[1:][same] > md.col_sorted_indx[:-1][same]).all()
    so, bo, bs = oracle.ragged_metadata_oracle(cs, 65536)
    assert torch.equal(ragged.slice_offs.cpu(), so) and torch.equal(ragged.block_offs_data.cpu(), bo)
    assert torch.equal(ragged.block_schedule_data.cpu(), bs)
    assert torch.equal(gather_idx.cpu(), col // 4) and torch.equal(scatter_idx.cpu(), col)


@pytest.mark.parametrize("T, E, k", [(1, 128, 4), (7, 13, 2), (255, 32, 4), (256, 128, 4), (257, 200, 8), (4099, 256, 4),
                                     (16384, 128, 4), (129, 48, 3), (1000, 128, 6), (300, 64, 16), (2500, 96, 1)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_fused_route_equals_separate_entry_points(T, E, k, dtype, device, monkeypatch):
    """`route` (three launches: top-k + histogram, scan + ragged metadata, rank) returns exactly what the five-launch
    composition topk -> make_bitmatrix_metadata -> make_ragged_tensor_metadata returns, and what the oracle computes."""
    import importlib
    routing_mod = importlib.import_module("triton_b200.routing")      # (the package exports a function of the same name)
    route = routing_mod.route
    monkeypatch.setattr(routing_mod, "FUSED_MAX_TOKENS", 1 << 30)      # the fused form at every size
    torch.manual_seed(T * 131 + E)
    logits = torch.randn(T, E, device=device).to(dtype)
    if T > 2:
        logits[1] = logits[0]                      # equal rows and ties inside a row
        logits[2, : E // 2] = logits[2, E // 2: 2 * (E // 2)]
    ragged, sp = route(logits, k)
    sp2 = topk(logits, k)
    md, md2 = sp.mask_metadata, sp2.mask_metadata
    rg2 = make_ragged_tensor_metadata(md2.col_sum, T * k)
    assert torch.equal(sp.indx, sp2.indx) and torch.equal(sp.vals, sp2.vals)
    assert torch.equal(sp.mask.storage.data[:T], sp2.mask.storage.data[:T])
    assert torch.equal(md.col_sum, md2.col_sum) and torch.equal(md.col_sorted_indx, md2.col_sorted_indx)
    assert torch.equal(md.row_sorted_indx, md2.row_sorted_indx)
    assert torch.equal(ragged.slice_offs, rg2.slice_offs) and torch.equal(ragged.block_offs_data, rg2.block_offs_data)
    assert torch.equal(ragged.block_schedule_data, rg2.block_schedule_data)
    # and the oracle
    vals_o, indx_o, _ = oracle.topk_oracle(logits.cpu(), k, apply_softmax=True)
    assert torch.equal(sp.indx.cpu().long(), indx_o.long())
    col_sum_o, col_sorted_o, row_sorted_o = oracle.bitmatrix_metadata_oracle(indx_o, E)
    assert torch.equal(md.col_sum.cpu().long(), col_sum_o.long())
    assert torch.equal(md.col_sorted_indx.cpu().long(), col_sorted_o.long())
    assert torch.equal(md.row_sorted_indx.cpu().long(), row_sorted_o.long())


@pytest.mark.parametrize("T", [2, 32, 33, 64, 65, 128, 129, 256])
@pytest.mark.parametrize("E, k", [(8, 8), (20, 1), (100, 2), (256, 16)])
def test_small_batch_routing_at_its_lane_splits(T, E, k, device):
    """Up to 256 tokens route in one launch with 32, 16, 8 or 4 lanes per token; whole numbers, so equal to the oracle."""
    g = torch.Generator().manual_seed(T * 1000 + E + k)
    # ties; + 0.0 leaves no negative zeros, which the selection has always ordered below zero and the oracle equal to it
    logits = (torch.randn(T, E, generator=g) * 4).round() / 4 + 0.0
    ragged, gather_idx, scatter_idx, sp = routing(logits.to(device), k)
    vals_o, indx_o, _ = oracle.topk_oracle(logits, k, apply_softmax=True)
    col_sum_o, col_sorted_o, row_sorted_o = oracle.bitmatrix_metadata_oracle(indx_o, E)
    assert torch.equal(sp.indx.cpu().long(), indx_o.long())
    # exps of 2 ulp, a sum of k terms, a division
    torch.testing.assert_close(sp.vals.cpu(), vals_o.float(), rtol=(k + 6) * 2 ** -23, atol=0)
    assert torch.equal(ragged.slice_sizes.cpu().long(), col_sum_o.long())
    assert torch.equal(scatter_idx.cpu().long(), col_sorted_o.long())
    assert torch.equal(sp.mask_metadata.row_sorted_indx.cpu().long(), row_sorted_o.long())
    assert torch.equal(gather_idx.cpu().long(), col_sorted_o.long() // k)
    ref = make_ragged_tensor_metadata(ragged.slice_sizes, T * k)
    assert torch.equal(ragged.block_offs_data, ref.block_offs_data) and torch.equal(ragged.block_schedule_data, ref.block_schedule_data)


@pytest.mark.parametrize("T", [24, 33, 64, 255, 257, 1000, 1025, 1536, 1537, 2041, 2048])
@pytest.mark.parametrize("E, k", [(8, 8), (20, 1), (100, 2), (128, 4), (256, 16)])
def test_routing_in_one_cluster(T, E, k, device):
    """Either side of where a cluster of eight blocks takes the step: shares of every size (empty and partial last ones among them), lanes per
    row, rounds of entries per warp, ties across the shares."""
    torch.manual_seed(T + E)
    logits = torch.randn(T, E)
    logits[:, min(3, E - 1)] = logits[:, 0]
    ragged, gather, scatter, sp = routing(logits.to(device), k)
    vals, indx, bm = oracle.topk_oracle(logits, k, True)
    col_sum, col, row = oracle.bitmatrix_metadata_oracle(indx, E)
    md = sp.mask_metadata
    assert torch.equal(sp.indx.cpu().int(), indx.int()) and torch.equal(sp.mask.storage.data.cpu(), bm)
    torch.testing.assert_close(sp.vals.cpu(), vals, atol=2e-6, rtol=2e-5)
    assert torch.equal(md.col_sum.cpu(), col_sum) and torch.equal(md.col_sorted_indx.cpu(), col) and torch.equal(md.row_sorted_indx.cpu(), row)
    offs, block_offs, sched = oracle.ragged_metadata_oracle(col_sum, T * k)
    assert torch.equal(ragged.slice_offs.cpu(), offs) and torch.equal(ragged.block_offs_data.cpu(), block_offs)
    assert torch.equal(ragged.block_schedule_data.cpu(), sched)
    assert torch.equal(gather.cpu().int(), (col // k).int())


@pytest.mark.parametrize("E, k, line", [(8, 1, 2048), (64, 2, 2048), (32, 4, 2048), (16, 8, 2048), (256, 1, 1536), (256, 2, 1536), (128, 4, 1536), (32, 8, 1536),
                                        (200, 4, 896), (64, 8, 896), (16, 16, 896), (256, 8, 1536)])
def test_lists_that_one_cluster_routes(E, k, line, device):
    """Launches of a call by itself on either side of the line between one cluster and two launches."""
    lib = _lib.load()
    for T, n in ((257, 1), (line, 1), (line + 1, 2)):
        logits = torch.randn(T, E, device=device)
        before = lib.moe_launch_count()
        sp = routing(logits, k)[3]
        assert lib.moe_launch_count() - before == n, (T, n)
        vals, indx, bm = oracle.topk_oracle(logits.cpu(), k, True)
        assert torch.equal(sp.indx.cpu().int(), indx.int())


@pytest.mark.parametrize("E, k, one, two", [(64, 1, 1024, 1025), (128, 2, 1024, 1025), (256, 1, 1024, 1025), (8, 1, 896, 897), (8, 2, 1025, 1024), (8, 1, 1536, 1537),
                                            (32, 2, 896, 897), (128, 4, 896, 897), (16, 8, 896, 897), (256, 8, 1536, 1537)])
def test_lists_that_one_cluster_routes_in_a_step(E, k, one, two, device):
    """The same of a layer step: one launch fewer with `one` tokens than with `two`, and the rows of the smaller step with either."""
    from triton_b200.moe import moe_layer_forward
    from triton_b200.testing import make_synthetic_layer
    lib, lw = _lib.load(), make_synthetic_layer(E, 256, 128, device, seed=1, chunk=E, block_scaled=True)
    x, logits = torch.randn(max(one, two), 256, device=device).bfloat16(), torch.randn(max(one, two), E, device=device)
    count, rows = [], []
    for T in (one, two):
        before = lib.moe_launch_count()
        rows.append(moe_layer_forward(x[:T], logits[:T], lw, k)[: min(one, two)])
        count.append(lib.moe_launch_count() - before)
    assert count[1] - count[0] == 1
    torch.testing.assert_close(rows[0], rows[1], rtol=2 ** -6, atol=1e-3)


@pytest.mark.parametrize("T, E, k", [(257, 20, 3), (2049, 128, 4), (8193, 200, 6), (8300, 256, 8), (8321, 256, 8), (18176, 32, 1), (18305, 32, 1), (300, 256, 40)])
def test_routing_in_two_launches(T, E, k, device):
    """Either side of where the blocks that rank also add up the counts (their number and the length of a block's list decide), k that the quad
    top-k does not take, entries of several rounds per warp, a last block of one token."""
    torch.manual_seed(T + E)
    logits = torch.randn(T, E)
    ragged, gather, scatter, sp = routing(logits.to(device), k)
    _, indx, _ = oracle.topk_oracle(logits, k, True)
    col_sum, col, row = oracle.bitmatrix_metadata_oracle(indx, E)
    md = sp.mask_metadata
    assert torch.equal(md.col_sum.cpu(), col_sum) and torch.equal(md.col_sorted_indx.cpu(), col) and torch.equal(md.row_sorted_indx.cpu(), row)
    offs, block_offs, sched = oracle.ragged_metadata_oracle(col_sum, T * k)
    assert torch.equal(ragged.slice_offs.cpu(), offs) and torch.equal(ragged.block_offs_data.cpu(), block_offs)
    assert torch.equal(ragged.block_schedule_data.cpu(), sched)


@pytest.mark.parametrize("call", ["row count", "reduce output", "router weight", "router bias"])
def test_host_tensors_are_refused(call, device):
    """A tensor in host memory beside device tensors is refused, not handed to a kernel."""
    from triton_b200 import reduce, router_topk
    x = torch.randn(64, 64, device=device).bfloat16()
    wg = torch.randn(8, 64).bfloat16().t()
    with pytest.raises(ValueError, match="CUDA tensors only"):
        if call == "row count":
            sp = topk(torch.randn(64, 8, device=device), 2)
            mask = wrap_torch_tensor(sp.mask.storage.data, dtype=BIT, shape=[torch.tensor(40, dtype=torch.int32), 8], shape_max=[64, 8])
            make_bitmatrix_metadata(sp.indx, mask)
        elif call == "reduce output":
            reduce(x.view(8, 8, 64), 1, y=torch.empty(8, 64, dtype=torch.bfloat16))
        elif call == "router weight":
            router_topk(x, wg, None, 2)
        else:
            router_topk(x, wg.to(device), torch.zeros(8), 2)


@pytest.mark.parametrize("T, E, k", [(3, 5, 4), (300, 128, 4), (40, 8, 6), (70, 32, 8)])
def test_rows_of_all_ones_bits_pick_experts_in_range(T, E, k, device):
    """Logits whose bytes are all 0xFF (memory that was never written, say) are NaN of the lowest order: their rows pick k different
    experts all the same, and nothing is counted outside the histogram."""
    logits = torch.randn(T, E, device=device)
    logits.view(torch.int32)[::2] = -1
    ragged, gather, scatter, sp = routing(logits, k)
    indx = sp.indx.cpu().long()
    assert (indx >= 0).all() and (indx < E).all()
    assert all(len(set(r.tolist())) == k for r in indx)
    assert torch.equal(sp.mask_metadata.col_sum.cpu(), torch.bincount(indx.reshape(-1), minlength=E).int())
    assert torch.equal(topk(logits, k).indx.cpu().long(), indx)
