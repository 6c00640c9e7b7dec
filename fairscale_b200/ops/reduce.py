"""Column reductions (bias gradients) on ``csrc/norm.cu``'s strip-partial kernels."""

from __future__ import annotations

from typing import Optional

import torch

from . import _bind


def column_sum(x: torch.Tensor, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``x.sum(0)`` for a 2-D bf16 matrix, accumulated in fp32 without atomics.  ``out``: dense bf16 ``[H]`` that the kernel
    may write (a window of a flat gradient); other dtypes and sizes return a new tensor and leave it alone."""
    x2 = x.reshape(-1, x.shape[-1])
    rows, H = x2.shape
    if not _bind.use_native(x2) or x2.dtype != torch.bfloat16 or H % 8 or rows == 0:
        return x2.float().sum(0).to(x.dtype)
    x2 = _bind.dense16(x2)
    strips = _bind.fn("fsb_colsum_num_strips")(rows)
    partials = torch.empty((strips, H), dtype=torch.float32, device=x.device)
    if out is None:
        out = torch.empty((H,), dtype=torch.bfloat16, device=x.device)
    _bind.call("fsb_colsum", x2.data_ptr(), rows, H, partials.data_ptr(), out.data_ptr(), _bind.stream_ptr(x.device), launches=2)
    return out


def batched_column_sum(x: torch.Tensor) -> torch.Tensor:
    """``x.sum(1)`` for a 3-D tensor: the bias gradients of stacked experts, accumulated in fp32."""
    E, rows, H = x.shape
    if not _bind.use_native(x) or x.dtype != torch.bfloat16 or H % 8 or rows == 0:
        return x.float().sum(1).to(x.dtype)
    x = _bind.dense16(x)
    strips = _bind.fn("fsb_colsum_num_strips")(rows)
    partials = torch.empty((E, strips, H), dtype=torch.float32, device=x.device)
    out = torch.empty((E, H), dtype=torch.bfloat16, device=x.device)
    _bind.call("fsb_colsum_batched", x.data_ptr(), E, rows, H, partials.data_ptr(), out.data_ptr(), _bind.stream_ptr(x.device), launches=2)
    return out
