"""Router product fused with the top-k selection: `topk(matmul(x, wg, bg), k)` in one kernel.

The reference computes the router logits with its general `matmul` and hands them to `topk`
(triton_kernels bench/bench_mlp.py:70, topk.py:106-141); here the logits stay in tensor memory and the selection,
the softmax over the selected logits and the expert bitmatrix happen in the GEMM's epilogue (`moe_router_topk`)."""
import torch

from . import _lib
from .matmul import _status_word
from .tensor import SparseMatrix, bit_tensor
from .topk import topk


def prepare_router_weight(wg: torch.Tensor) -> torch.Tensor:
    """-> Wg as the kernel reads it: logical shape [K, E] kept, memory [E, K] with K contiguous (stride(0) == 1).
    A weight that already has that memory order is returned as it is; do this once per layer, not per step."""
    assert wg.ndim == 2
    if wg.stride(0) == 1 and wg.stride(1) % 8 == 0 and wg.dtype == torch.bfloat16:
        return wg
    return wg.to(torch.bfloat16).t().contiguous().t()


def router_topk_supported(x, wg, k) -> bool:
    return (isinstance(x, torch.Tensor) and x.is_cuda and x.ndim == 2 and x.dtype == torch.bfloat16 and wg.dtype == torch.bfloat16
            and x.stride(1) == 1 and x.stride(0) % 8 == 0 and x.shape[1] % 8 == 0 and wg.stride(0) == 1 and wg.stride(1) % 8 == 0
            and wg.shape[1] <= 256 and k in (1, 2, 4, 8, 16) and k <= wg.shape[1] and x.data_ptr() % 16 == 0
            and wg.data_ptr() % 16 == 0)


def _two_steps(logits, k, apply_softmax, return_logits):
    sp = topk(logits, k, apply_softmax=apply_softmax)
    return (sp, logits.float()) if return_logits else sp


def router_topk(x: torch.Tensor, wg: torch.Tensor, bg, k: int, apply_softmax: bool = True, logits_dtype=None,
                return_logits: bool = False):
    """SparseMatrix of `topk(x @ wg + bg, k, apply_softmax)` (and the fp32 logits when `return_logits`).

    x [T, K] bf16; wg [K, E] bf16 -- in the memory order of `prepare_router_weight`, else it is re-laid-out on every
    call; bg [E] or None.  `logits_dtype` is the dtype the two-step form would give the logits (default x.dtype: bf16,
    i.e. every logit is rounded to bf16 before the selection, as `matmul` rounds its output); the routing weights come
    back in that dtype like `topk`'s.  Shapes the kernel does not take (more than 256 experts, k not a power of two up
    to 16, unaligned rows) run the two steps apart."""
    logits_dtype = x.dtype if logits_dtype is None else logits_dtype
    assert logits_dtype in (torch.bfloat16, torch.float32)
    wg = prepare_router_weight(wg)
    if not router_topk_supported(x, wg, k):
        logits = (x.float() @ wg.float() + (0 if bg is None else bg.float())).to(logits_dtype)
        return _two_steps(logits, k, apply_softmax, return_logits)
    T, E = x.shape[0], wg.shape[1]
    dev = x.device
    logits = torch.empty((T, E), dtype=torch.float32, device=dev) if return_logits else None
    if bg is not None and bg.dtype not in (torch.float32, torch.bfloat16):
        bg = bg.float()
    vals, indx, bm = _lib.host().router(x, wg, bg, k, bool(apply_softmax), logits_dtype == torch.bfloat16, logits, _status_word(dev))
    sp = SparseMatrix(indx=indx, vals=vals, mask=bit_tensor(bm, T, E))
    return (sp, logits) if return_logits else sp
