"""Blockwise linear absmax codec on CUDA tensors: the counterpart of
came_pytorch/blockwise_quantization.py (quantize_blockwise :66-82, dequantize_blockwise :108-124) and of
the tile layout of came2d_step, computed by libcame_b200 and bit-exact with the reference's fp32 formulas.
"""
from __future__ import annotations

import math

import torch

from . import _host

BLOCK = 256


def num_blocks(numel: int, block_size: int = BLOCK) -> int:
    if block_size <= 0:
        raise ValueError(f"block_size must be > 0, got {block_size}")
    return max(1, math.ceil(numel / block_size))


def _require(t: torch.Tensor, block_size: int) -> None:
    if block_size != BLOCK:
        raise ValueError("came_b200 supports block_size=256 only")
    if not t.is_cuda:
        raise RuntimeError("came_b200.quant works on CUDA tensors only (there is no CPU fallback)")


def quantize_blockwise(tensor: torch.Tensor, *, signed: bool, block_size: int = BLOCK):
    """-> (q, absmax): int8 (signed) or uint8 codes shaped like `tensor`, fp32 absmax per 256 flat elements."""
    _require(tensor, block_size)
    return _host.quantize(tensor, signed, False)


def dequantize_blockwise(q: torch.Tensor, absmax: torch.Tensor, *, signed: bool, block_size: int = BLOCK,
                         dtype: torch.dtype = torch.float32) -> torch.Tensor:
    _require(q, block_size)
    want = torch.int8 if signed else torch.uint8
    if q.dtype != want:
        raise RuntimeError(f"expected {want} codes, got {q.dtype}")
    need = num_blocks(q.numel())
    if absmax.numel() < need:
        raise RuntimeError(f"absmax has {absmax.numel()} entries, {need} needed")
    if absmax.device != q.device:
        raise RuntimeError(f"absmax is on {absmax.device}, the codes on {q.device}")
    out = _host.dequantize(q, absmax, signed, False)
    return out if dtype == torch.float32 else out.to(dtype)


def quantize_tile16(matrix: torch.Tensor):
    """-> (q int8 [R, C], absmax fp32 [ceil(R/16)*ceil(C/16)]): the exp_avg layout of CAME8bit / CAME8bit2D."""
    _require(matrix, BLOCK)
    if matrix.dim() != 2:
        raise RuntimeError("quantize_tile16 expects a 2-D tensor")
    return _host.quantize(matrix, True, True)


def dequantize_tile16(q: torch.Tensor, absmax: torch.Tensor) -> torch.Tensor:
    _require(q, BLOCK)
    if q.dim() != 2 or q.dtype != torch.int8:
        raise RuntimeError("dequantize_tile16 expects a 2-D int8 tensor")
    need = math.ceil(q.shape[0] / 16) * math.ceil(q.shape[1] / 16)
    if absmax.device != q.device:
        raise RuntimeError(f"absmax is on {absmax.device}, the codes on {q.device}")
    if absmax.numel() < need:
        raise RuntimeError(f"absmax has {absmax.numel()} entries, {need} needed")
    return _host.dequantize(q, absmax, True, True)
