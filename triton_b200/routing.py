"""`routing()`: the composition the reference's earlier API exposed under this name, written out in
its tests today (python/triton_kernels/tests/test_distributed.py:203-210)."""
import torch

from . import _lib
from .tensor import BitmatrixMetadata, SparseMatrix, bit_tensor, make_ragged_tensor_metadata
from .tensor_details.ragged_tensor import ragged_from_kernel
from .topk import topk


FUSED_MAX_TOKENS = 1 << 22


def route(logits, n_expts_act, apply_softmax=True):
    """Top-k, expert histogram, expert-major sort and ragged metadata of one batch of logits in one launch (up to some 900
    tokens, 1536 or 2048 with short lists), two or three: -> (ragged_metadata, sparse_logits), the same objects `topk` + `make_ragged_tensor_metadata` return.
    More than 256 experts, more than FUSED_MAX_TOKENS tokens, or logits that are not a plain 2-D tensor take the
    five-launch composition of the separate entry points."""
    return _route(logits, n_expts_act, apply_softmax)[:2]


def _route(logits, n_expts_act, apply_softmax):
    """`route` and the token of every expert-sorted row where the same launches give it (float logits), else None"""
    if not (isinstance(logits, torch.Tensor) and logits.ndim == 2 and logits.shape[1] <= 256
            and 0 < logits.shape[0] <= FUSED_MAX_TOKENS and logits.stride(1) == 1):
        sparse = topk(logits, n_expts_act, apply_softmax=apply_softmax)
        md = sparse.mask_metadata
        return make_ragged_tensor_metadata(md.col_sum, md.row_sorted_indx.shape[0]), sparse, None
    T, E = logits.shape
    vals, indx, bm, col_sum, col_sorted, row_sorted, slice_offs, block_offs, sched, tokens = \
        _lib.host().route(logits, n_expts_act, bool(apply_softmax))
    sparse = SparseMatrix(indx=indx, vals=vals, mask=bit_tensor(bm, T, E),
                          mask_metadata=BitmatrixMetadata(col_sum=col_sum, col_sorted_indx=col_sorted, row_sorted_indx=row_sorted))
    return ragged_from_kernel(col_sum, slice_offs, block_offs, sched), sparse, tokens


def routing(logits, n_expts_act, all_gather=False, y_indx=None, symm_mem_pool=None, apply_softmax=True):
    """-> (ragged_metadata, gather_idx, scatter_idx, sparse_logits).

    gather_idx[p] is the token whose activations feed expert-sorted row p, scatter_idx[p] the flat
    (token * k + slot) row its output goes to; sparse_logits.vals holds the routing weights."""
    if not all_gather and y_indx is None:
        ragged, sparse, gather_idx = _route(logits, n_expts_act, apply_softmax)
        combine_indx = sparse.mask_metadata.col_sorted_indx
    else:
        gather_idx = None
        sparse = topk(logits, n_expts_act, apply_softmax=apply_softmax, all_gather=all_gather, y_indx=y_indx,
                      symm_mem_pool=symm_mem_pool)
        dispatch_indx = sparse.mask_metadata.row_sorted_indx
        combine_indx = sparse.mask_metadata.col_sorted_indx
        ragged = make_ragged_tensor_metadata(sparse.mask_metadata.col_sum, dispatch_indx.shape[0])
    if gather_idx is None:
        gather_idx = torch.div(combine_indx, n_expts_act, rounding_mode="trunc")
    scatter_idx = combine_indx
    return ragged, gather_idx, scatter_idx, sparse
