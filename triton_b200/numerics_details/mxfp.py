"""MXFP4 quantise / dequantise (triton_kernels/numerics_details/mxfp.py:25-176): e2m1 values packed two
per byte along `axis`, one e8m0 scale byte per 32 elements.  MXFP8 / NVFP4 variants of the reference
are outside the MoE path and raise NotImplementedError."""
from enum import Enum

import torch

from .. import _lib
from ..tensor import FP4, Tensor

MXFP_BLOCK_SIZE = 32
NVFP_BLOCK_SIZE = 16


class DequantScaleRoundingMode(Enum):
    ROUND_UP = 0      # scale = 2^ceil(log2(max / 6)): never clips the block maximum
    ROUND_DOWN = 1    # scale = 2^floor(log2(max / 4)): the OCP rule, may clip


def downcast_to_mxfp(x, out_dtype, axis: int, scale_dtype: torch.dtype = torch.uint8,
                     microblock_size: int = MXFP_BLOCK_SIZE,
                     DEQUANT_SCALE_ROUNDING_MODE: DequantScaleRoundingMode = DequantScaleRoundingMode.ROUND_UP):
    """-> (values uint8, scales uint8).  values.shape = x.shape with shape[axis] halved, scales.shape with
    shape[axis] // 32; both are contiguous along `axis` (StridedLayout(major_dim=axis), mxfp.py:61-64)."""
    if isinstance(x, Tensor):
        x = x.storage.data
    if out_dtype not in (torch.uint8, FP4):
        raise NotImplementedError("downcast_to_mxfp: only MXFP4 (torch.uint8) output is supported")
    if scale_dtype != torch.uint8 or microblock_size != MXFP_BLOCK_SIZE:
        raise NotImplementedError("downcast_to_mxfp: only e8m0 scales per 32 elements are supported")
    assert -x.ndim <= axis < x.ndim, f"Invalid axis {axis=}"
    axis %= x.ndim
    L = x.shape[axis]
    assert L % microblock_size == 0, f"axis dim must be divisible by {microblock_size}. Got {L}"
    # outputs: quantised axis innermost in memory, the other axes as in x.transpose(axis, -1)
    return _lib.host().downcast(x, axis, DEQUANT_SCALE_ROUNDING_MODE.value)


def upcast_from_mxfp(tensor: torch.Tensor, scale: torch.Tensor, target_dtype: torch.dtype, axis: int,
                     tensor_scale=None):
    """Packed e2m1 + e8m0 -> fp16 / bf16 / fp32, dequantised along `axis`; result is contiguous."""
    if tensor_scale is not None:
        raise NotImplementedError("upcast_from_mxfp: tensor_scale is not supported")
    if tensor.dtype != torch.uint8 or scale.dtype != torch.uint8:
        raise NotImplementedError("upcast_from_mxfp: only MXFP4 values with e8m0 scales are supported")
    assert target_dtype in (torch.float16, torch.bfloat16, torch.float32), f"Invalid output dtype {target_dtype=}"
    ndim = tensor.ndim
    assert -ndim <= axis < ndim and tensor.ndim == scale.ndim
    axis %= ndim
    return _lib.host().upcast(tensor, scale, target_dtype, axis)
