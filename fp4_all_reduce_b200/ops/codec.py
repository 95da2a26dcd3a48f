"""Stand-alone codec and norm ops on CUDA tensors (hand-written sm_100a kernels, csrc/kernels/codec_ops.cu).

These are the building blocks of the fused AllReduce exposed one by one, the way the reference project
exposes them as benchmark kernels (bench/codec/codec_bench.cu:139-590).  All functions launch on the
current CUDA stream and never fall back to PyTorch: a missing library or a non-CUDA tensor is an error.  Checks,
output allocation and the launch are one C++ call (csrc/runtime/torch_front.cpp).
"""
from __future__ import annotations

import ctypes as C
from typing import Sequence

import torch

from .. import _native as N


def _stream() -> C.c_void_p:
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _req_layout(t: torch.Tensor, dtype, cols: int | None, name: str) -> torch.Tensor:
    """dtype, shape [rows, cols] and contiguity; the device is the caller's business."""
    if t.dtype != dtype:
        raise ValueError(f"{name} must be {dtype}, got {t.dtype}")
    if cols is not None and (t.dim() != 2 or t.shape[1] != cols):
        raise ValueError(f"{name} must have shape [rows, {cols}], got {tuple(t.shape)}")
    if not t.is_contiguous():
        raise ValueError(f"{name} must be contiguous")
    return t


def encode(x: torch.Tensor) -> tuple[torch.Tensor, torch.Tensor]:
    """BF16 [rows, 6144] -> (NVFP4 rows [rows, 3456] uint8: 3072 value bytes then 384 scale bytes,
    FP32 row scales [rows])."""
    return N.front().encode(x)


def encode_static(x: torch.Tensor, gs: float) -> torch.Tensor:
    """BF16 [rows, 6144] -> NVFP4 rows [rows, 3456] with the static per-tensor scale gs (no row scale)."""
    return N.front().encode_static(x, gs)


def decode_sum(qrows: Sequence[torch.Tensor], row_scales=None, gs=None) -> torch.Tensor:
    """FP32 decode-accumulate of the sources in list order, BF16 [rows, 6144] out."""
    return N.front().decode_sum(qrows, row_scales, gs)


def reduce_reencode(qrows: Sequence[torch.Tensor], row_scales=None, gs=None) -> tuple[torch.Tensor, torch.Tensor]:
    """The two-shot owner step: decode-sum, re-encode the FP32 sum with its own row scale, and output the
    decode of that re-encoding.  Returns (records [rows, 3584] uint8, BF16 [rows, 6144])."""
    return N.front().reduce_reencode(qrows, row_scales, gs)


def add_rmsnorm(x: torch.Tensor, residual: torch.Tensor, weight: torch.Tensor, eps: float = 1e-6,
                weight_bias: float = 1.0, epilogue: int = N.EPI_NORM_BF16, qscale: float = 1.0,
                inplace_residual: bool = False, out: torch.Tensor | None = None) -> tuple[torch.Tensor, torch.Tensor]:
    """z = x + residual; residual' = bf16(z); y = (bf16(z) * rinv) * (weight_bias + weight).
    Returns (y as BF16 [rows,6144] | NVFP4 rows [rows,3456] | MXFP8 rows [rows,6336], residual')."""
    return N.front().add_rmsnorm(x, residual, weight, eps, weight_bias, epilogue, qscale, inplace_residual, out)


def fill_sentinel(window: torch.Tensor, buffer_bytes: int, nbuffers: int = 2) -> None:
    """Overwrite a receive window with the not-yet-written patterns (0x88 values, 0xFF scales, -0.0 row scale)."""
    if window.dtype != torch.uint8 or not window.is_cuda or window.numel() < buffer_bytes * nbuffers:
        raise ValueError("window must be a CUDA uint8 tensor of at least buffer_bytes * nbuffers")
    with torch.cuda.device(window.device):
        N.check(N.cuda().fp4ar_fill_sentinel(window.data_ptr(), buffer_bytes, nbuffers, _stream()), "fp4ar_fill_sentinel")
