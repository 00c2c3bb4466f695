"""Two products in a row through the C entry point: the same as the two products called one after the other, whatever the caller's buffers
look like.  The argument block is read from the header, so these tests call the library as a C program does."""
import ctypes as C
import re
from pathlib import Path

import pytest
import torch

from triton_b200 import _lib, make_ragged_tensor_metadata, routing
from triton_b200.testing import make_synthetic_layer

pytestmark = pytest.mark.gpu

HEADER = re.sub(r"/\*.*?\*/", "", (Path(__file__).resolve().parent.parent / "include" / "moe_b200.h").read_text(), flags=re.S)
CONST = {m[0]: int(m[1]) for m in re.findall(r"\b(MOE_[A-Z0-9_]+)\s*=?\s+(\d+)", HEADER)}


def _struct(name):
    body = re.search(r"typedef struct \{([^}]*)\} %s;" % name, HEADER).group(1)
    types = {"int": C.c_int, "int64_t": C.c_int64, "float": C.c_float}
    fields = []
    for decl in filter(None, (d.strip() for d in body.split(";"))):
        base, names = re.fullmatch(r"(?:const )?(\w+\s*\*?)\s*(.*)", decl, flags=re.S).groups()
        for n in names.split(","):
            array = re.fullmatch(r"\s*(\w+)\[(\w+)\]", n)
            t = C.c_void_p if "*" in base else types[base.strip()]
            fields.append((array.group(1), t * CONST[array.group(2)]) if array else (n.strip(), t))
    return type(name, (C.Structure,), {"_fields_": fields})


Args = _struct("MoeGemmArgs")
E, K, D, FF = 6, 2, 512, 320


class Problem:
    """fc1 + SwiGLU and fc2 of a layer as two argument blocks; `pitch1`, `pitch2`: row pitch of the rows between as the first writes and the
    second reads them."""

    def __init__(self, T, device, block=0, pitch1=FF, pitch2=FF, e4m3=False):
        g = torch.Generator(device=device).manual_seed(T)
        dt = torch.float8_e4m3fn if e4m3 else torch.bfloat16
        self.x = torch.randn(T, D, device=device, generator=g).bfloat16().to(dt)
        logits = torch.randn(T, E, device=device, generator=g) + torch.randn(E, device=device, generator=g)
        lw = make_synthetic_layer(E, D, FF, device, seed=3, block_scaled=True)
        ragged, self.gather, scatter, sp = routing(logits, K)
        self.M = M = T * K
        self.gather = self.gather.int().contiguous()
        self.h = torch.zeros(M + 1, max(pitch1, pitch2), device=device, dtype=torch.bfloat16).to(dt)
        self.y = torch.zeros(M, D, device=device, dtype=torch.bfloat16)
        self.status = torch.zeros(1, dtype=torch.int32, device=device)
        self.keep = [lw, ragged, scatter, sp, sp.mask_metadata]
        a, b = Args(), Args()
        code, size = (CONST["MOE_F8E4M3"], 1) if e4m3 else (CONST["MOE_BF16"], 2)
        for p, (w, ws, bias, k, n) in ((a, (lw.w1_bs, lw.w1_bs_scale, lw.b1, D, 2 * FF)), (b, (lw.w2_bs, lw.w2_bs_scale, lw.b2, FF, D))):
            p.w_kind, p.w, p.w_scale, p.E, p.K, p.N, p.M = _lib.MOE_W_MX4_B200MX, w.storage.data.data_ptr(), ws.storage.data.data_ptr(), E, k, n, M
            p.slice_sizes, p.slice_offs = ragged.slice_sizes.data_ptr(), ragged.slice_offs.data_ptr()
            p.block_offs_16, p.block_sched_16 = ragged.block_offs_data.data_ptr(), ragged.block_schedule_data.data_ptr()
            p.ld_block_offs, p.ld_block_sched = ragged.block_offs_data.stride(0), ragged.block_schedule_data.stride(0)
            p.bias, p.bias_dtype, p.ld_bias = bias.data_ptr(), CONST["MOE_F32"] if bias.dtype == torch.float32 else CONST["MOE_BF16"], bias.stride(0)
            p.tile_m, p.status = block, self.status.data_ptr()
            p.x_dtype = code
        a.x, a.ld_x, a.rows_x, a.gather_indx = self.x.data_ptr(), D, T, self.gather.data_ptr()
        a.activation, a.act_alpha, a.act_limit, a.act_has_limit = CONST["MOE_ACT_SWIGLU"], 1.702, 7.0, 1
        a.y, a.y_dtype, a.ld_y = self.h.data_ptr(), code, pitch1
        b.x, b.ld_x, b.rows_x = self.h.data_ptr(), pitch2, M
        b.y, b.y_dtype, b.ld_y = self.y.data_ptr(), CONST["MOE_BF16"], D
        lib = _lib.load()
        self.room = [int(lib.moe_gemm_mx_workspace_bytes(C.byref(p))) for p in (a, b)]
        self.ws = [torch.zeros(n + 4096, dtype=torch.uint8, device=device) for n in self.room]
        for p, n, ws in zip((a, b), self.room, self.ws):
            p.mx_workspace, p.mx_workspace_bytes = (ws.data_ptr() + 1023) // 1024 * 1024, n
        self.a, self.b = a, b

    def move(self, t, offset):
        """`t` into the second product's workspace, at `offset`; -> its address there."""
        raw = t.reshape(-1).view(torch.uint8)
        at = self.b.mx_workspace + offset
        lo = at - self.ws[1].data_ptr()
        assert lo + raw.numel() <= self.ws[1].numel()
        self.ws[1][lo:lo + raw.numel()].copy_(raw)
        return at

    def run(self, chain):
        """-> the second product's rows and the launches that took."""
        lib = _lib.load()
        self.h.view(torch.uint8).zero_()
        self.y.zero_()
        n0, st = lib.moe_launch_count(), torch.cuda.current_stream().cuda_stream
        if chain:
            _lib.check(lib.moe_grouped_gemm_chain(C.byref(self.a), C.byref(self.b), st), "chain")
        else:
            _lib.check(lib.moe_grouped_gemm(C.byref(self.a), st), "first")
            _lib.check(lib.moe_grouped_gemm(C.byref(self.b), st), "second")
        torch.cuda.synchronize()
        assert int(self.status) == 0
        return self.y.clone(), lib.moe_launch_count() - n0


# tokens and tile_m: four e2m1 terms, two e4m3 terms of 32 rows, the pair kernel
FORMS = [(20, 16), (70, 32), (300, 256)]


@pytest.mark.parametrize("T, block", FORMS)
@pytest.mark.parametrize("e4m3", [False, True])
def test_rows_are_handed_over(T, block, e4m3, device):
    p = Problem(T, device, block, e4m3=e4m3)
    (apart, n), (chain, m) = p.run(False), p.run(True)
    assert m == n - 1 and torch.equal(apart, chain) and bool(apart.abs().sum() > 0)


@pytest.mark.parametrize("T, block", FORMS)
@pytest.mark.parametrize("pitch1, pitch2", [(FF + 64, FF + 64), (FF, FF + 64), (FF + 64, FF)])
def test_pitches_of_the_rows_between(T, block, pitch1, pitch2, device):
    """The second product reads other rows than the first wrote where the pitches differ."""
    p = Problem(T, device, block, pitch1, pitch2)
    (apart, n), (chain, m) = p.run(False), p.run(True)
    assert torch.equal(apart, chain) and m == (n - 1 if pitch1 == pitch2 else n)


@pytest.mark.parametrize("T, block", FORMS)
def test_second_product_with_fewer_rows(T, block, device):
    """Rows past rows_x count as zero."""
    p = Problem(T, device, block)
    p.b.rows_x = p.M - 5
    (apart, n), (chain, m) = p.run(False), p.run(True)
    assert torch.equal(apart, chain) and m == n


@pytest.mark.parametrize("T, block", FORMS)
@pytest.mark.parametrize("operand", ["x", "gather"])
def test_operands_in_the_second_workspace(T, block, operand, device):
    """What the first product reads may lie in the workspace that the second one fills later."""
    p = Problem(T, device, block)
    want, n = p.run(False)
    if operand == "x":
        p.a.x = p.move(p.x, 0)
    else:
        p.a.gather_indx = p.move(p.gather, p.room[1] // 2 // 1024 * 1024)
    got, m = p.run(True)
    assert torch.equal(want, got) and m == n


@pytest.mark.parametrize("k", [2, 512, 513, 800])
def test_positions_of_a_row_beyond_a_block_of_shared_memory(k, device):
    """A row of x may go to any number of positions: the token pass by row holds those of eight rows, beyond that the pass goes by position."""
    p = Problem(20, device, 256)
    a, rows = p.a, 1184                                        # eight rows for each of 148 SMs: from there on by row
    g = torch.Generator(device=device).manual_seed(k)
    x = torch.randn(rows, D, device=device, generator=g).bfloat16()
    experts = torch.randint(0, E, (rows * k,), device=device, generator=g).short()
    order = torch.argsort(experts, stable=True)
    positions = torch.empty(rows * k, dtype=torch.int32, device=device)
    positions[order] = torch.arange(rows * k, dtype=torch.int32, device=device)
    gather = (order // k).int()
    ragged = make_ragged_tensor_metadata(torch.bincount(experts.long(), minlength=E).int(), rows * k)
    a.x, a.rows_x, a.M, a.gather_indx, a.N = x.data_ptr(), rows, rows * k, gather.data_ptr(), 128
    a.slice_sizes, a.slice_offs = ragged.slice_sizes.data_ptr(), ragged.slice_offs.data_ptr()
    a.block_offs_16, a.block_sched_16 = ragged.block_offs_data.data_ptr(), ragged.block_schedule_data.data_ptr()
    a.ld_block_offs, a.ld_block_sched = ragged.block_offs_data.stride(0), ragged.block_schedule_data.stride(0)
    lib, st = _lib.load(), torch.cuda.current_stream().cuda_stream
    ws = torch.empty(int(lib.moe_gemm_mx_workspace_bytes(C.byref(a))) + 1024, dtype=torch.uint8, device=device)
    a.mx_workspace, a.mx_workspace_bytes = (ws.data_ptr() + 1023) // 1024 * 1024, ws.numel() - 1024
    out = []
    for by_row in (False, True):
        y = torch.zeros(rows * k, 64, device=device, dtype=torch.bfloat16)
        a.y, a.ld_y = y.data_ptr(), 64
        if by_row:
            a.x_positions, a.x_experts, a.x_k = positions.data_ptr(), experts.data_ptr(), k
        assert lib.moe_gemm_kernel_name(C.byref(a)) == b"gemm_mx_pair_kernel"
        _lib.check(lib.moe_grouped_gemm(C.byref(a), st), "product")
        torch.cuda.synchronize()
        assert int(p.status) == 0
        out.append(y)
    assert torch.equal(*out) and bool(out[0].abs().sum() > 0)


class Passes:
    """One product over `rows` rows of x, each at k positions, to be called without and with the positions of every row."""

    def __init__(self, rows, k, depth, block, device, e4m3=False, dropped=False):
        g = torch.Generator(device=device).manual_seed(rows * k)
        x = torch.randn(rows, depth, device=device, generator=g).bfloat16()
        self.x = x.to(torch.float8_e4m3fn) if e4m3 else x
        lw = make_synthetic_layer(E, depth, 64, device, seed=3, block_scaled=True)
        experts = torch.randint(0, E, (rows * k,), device=device, generator=g).short()
        experts[: rows * k // 2] = 1                               # one expert of several blocks
        lost = torch.rand(rows * k, device=device, generator=g) < 0.3 if dropped else torch.zeros(rows * k, dtype=torch.bool, device=device)
        experts[lost] = E                                          # behind all others
        order = torch.argsort(experts, stable=True)
        positions = torch.empty(rows * k, dtype=torch.int32, device=device)
        positions[order] = torch.arange(rows * k, dtype=torch.int32, device=device)
        gather = (order // k).int()
        ragged = make_ragged_tensor_metadata(torch.bincount(experts.long(), minlength=E)[:E].int(), rows * k)
        self.live = int((~lost).sum())
        if dropped:                                                # no expert, none of the experts there are, no position, one past the expert's rows
            where = lost.nonzero().flatten()
            experts[where[0::4]], positions[where[0::4]] = -1, -1
            positions[where[1::4]] = 0
            experts[where[2::4]], positions[where[2::4]] = 0, -1
            experts[where[3::4]], positions[where[3::4]] = 0, ragged.slice_offs[1]
        self.status = torch.zeros(1, dtype=torch.int32, device=device)
        self.n, self.k, self.experts, self.positions = rows * k, k, experts, positions
        self.keep = [lw, gather, ragged]
        a = self.a = Args()
        a.w_kind, a.w, a.w_scale = _lib.MOE_W_MX4_B200MX, lw.w1_bs.storage.data.data_ptr(), lw.w1_bs_scale.storage.data.data_ptr()
        a.E, a.K, a.N, a.M = E, depth, 128, rows * k
        a.slice_sizes, a.slice_offs = ragged.slice_sizes.data_ptr(), ragged.slice_offs.data_ptr()
        a.block_offs_16, a.block_sched_16 = ragged.block_offs_data.data_ptr(), ragged.block_schedule_data.data_ptr()
        a.ld_block_offs, a.ld_block_sched = ragged.block_offs_data.stride(0), ragged.block_schedule_data.stride(0)
        a.x, a.ld_x, a.rows_x, a.gather_indx = self.x.data_ptr(), depth, rows, gather.data_ptr()
        a.x_dtype, a.y_dtype, a.ld_y = CONST["MOE_F8E4M3" if e4m3 else "MOE_BF16"], CONST["MOE_BF16"], 128
        a.tile_m, a.status = block, self.status.data_ptr()

    def run(self, by_row, kernel):
        lib, a = _lib.load(), self.a
        ws = torch.empty(int(lib.moe_gemm_mx_workspace_bytes(C.byref(a))) + 1024, dtype=torch.uint8, device=self.x.device)
        a.mx_workspace, a.mx_workspace_bytes = (ws.data_ptr() + 1023) // 1024 * 1024, ws.numel() - 1024
        y = torch.zeros(self.n, 128, device=self.x.device, dtype=torch.bfloat16)
        a.y = y.data_ptr()
        a.x_positions, a.x_experts, a.x_k = (self.positions.data_ptr(), self.experts.data_ptr(), self.k) if by_row else (None, None, 0)
        assert lib.moe_gemm_kernel_name(C.byref(a)) == kernel
        _lib.check(lib.moe_grouped_gemm(C.byref(a), torch.cuda.current_stream().cuda_stream), "product")
        torch.cuda.synchronize()
        assert int(self.status) == 0
        return y


# blocks of four e2m1 terms, of two e4m3 terms that fit their rows and that do not, e4m3 tokens; depths of whole and of cut k steps
@pytest.mark.parametrize("block, e4m3", [(16, False), (32, False), (64, False), (32, True)])
@pytest.mark.parametrize("rows, k, depth", [(1, 1, 96), (5, 3, 512), (17, 4, 736), (33, 2, 160), (3, 40, 128)])
def test_decode_tokens_by_row_are_those_by_position(block, e4m3, rows, k, depth, device):
    p = Passes(rows, k, depth, block, device, e4m3)
    by_position, by_row = p.run(False, b"gemm_mx_kernel"), p.run(True, b"gemm_mx_kernel")
    assert torch.equal(by_position, by_row) and bool(by_row.abs().sum() > 0)


# k steps in one part, two and four; an infinity in the first part, the last, or both; whole blocks from two and a half per SM on
@pytest.mark.parametrize("depth, rows", [(896, 1184), (1056, 1184), (1952, 1184), (2080, 1184), (2080, 2920), (2080, 2928), (1056, 4000)])
def test_pair_tokens_in_parts_are_those_by_row(depth, rows, device):
    p = Passes(rows, 2, depth, 256, device)                    # 1184, eight rows for each of 148 SMs: from there on by row with the positions
    p.x[3, 5] = p.x[40, depth - 1] = p.x[77, depth // 2] = float("inf")
    p.x[77, 0] = float("-inf")
    by_position, by_row = p.run(False, b"gemm_mx_pair_kernel"), p.run(True, b"gemm_mx_pair_kernel")
    assert torch.equal(by_position.nan_to_num(7.0, 9.0, -9.0), by_row.nan_to_num(7.0, 9.0, -9.0))
    assert bool(torch.isfinite(by_row).all(1).sum() > 2000) and not bool(torch.isfinite(by_row).all())


@pytest.mark.parametrize("rows, block, e4m3, kernel", [(40, 16, False, b"gemm_mx_kernel"), (40, 32, False, b"gemm_mx_kernel"), (40, 32, True, b"gemm_mx_kernel"),
                                                       (1184, 256, False, b"gemm_mx_pair_kernel"), (1184, 256, True, b"gemm_mx_pair_kernel")])
def test_entries_that_are_no_row_are_left_out(rows, block, e4m3, kernel, device):
    """Dropped picks and picks of experts or positions that there are not, among those of every token: the rows that there are come out as by position."""
    p = Passes(rows, 4, 512, block, device, e4m3, dropped=True)
    if block == 256 and not e4m3:
        p.x[7, 3] = float("inf")                                   # (a row that the token pass computes itself)
    by_position, by_row = (p.run(by, kernel)[:p.live].nan_to_num(7.0, 9.0, -9.0) for by in (False, True))
    assert torch.equal(by_position, by_row) and bool(by_row.abs().sum() > 0) and p.live < p.n


# blocks of four terms and of two
@pytest.mark.parametrize("block", [16, 32, 64])
@pytest.mark.parametrize("value", [float("inf"), float("nan"), 2.99e38, -3.38e38])
def test_decode_tokens_by_row_with_the_largest_values(block, value, device):
    p = Passes(40, 4, 512, block, device)
    for j in range(8):
        p.x[4 + j, 33 * j] = value                                 # at each of a lane's four places
    p.x[20, 64:72] = value                                         # a lane that has no other
    by_position, by_row = (p.run(by, b"gemm_mx_kernel").nan_to_num(7.0, 9.0, -9.0) for by in (False, True))
    assert torch.equal(by_position, by_row)
