"""Causal multi-head self-attention.

``causal_attention(qkv, n_heads)`` takes the packed projection ``[B, S, 3*H*D]`` and returns ``[B, S, H*D]``.
CUDA bf16 inputs run the hand-written kernels of ``csrc/attention.cu`` when they are present in the
native library; otherwise (and on CPU) a PyTorch formulation is used and :data:`BACKEND` says so.
"""

from __future__ import annotations

import math
import warnings
from typing import Optional

import torch

from . import _bind

BACKEND = "unset"
_WARNED_LIBRARY_PATH = False  # the fall-back to the library kernel is announced once


def _reference(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, scale: float) -> torch.Tensor:
    """fp32 attention oracle on [B, H, S, D] tensors."""
    s = torch.matmul(q.float(), k.float().transpose(-1, -2)) * scale
    n = s.shape[-1]
    s = s.masked_fill(torch.ones(n, n, dtype=torch.bool, device=s.device).triu(1), float("-inf"))
    return torch.matmul(torch.softmax(s, dim=-1), v.float())


def _native_available() -> bool:
    from .. import _native

    try:
        return hasattr(_native.lib(), "fsb_attn_fwd")
    except Exception:
        return False


def _native_is_faster(B: int, S: int, H: int, inference: bool) -> bool:
    """For a length that is no multiple of 128: the kernels here or torch's operator, which needs q, k and v permuted and their
    gradients concatenated?  Forward + backward on B200 (us, torch / here): B4 S1543 H16 D128 540 / 292, B2 S4095 H16 D64 573 / 423,
    B4 S5000 H16 D64 1568 / 1286, B1 S8000 H2 D64 249 / 254, B1 S8000 H2 D128 316 / 368 - the backward here makes the scores twice, and
    few heads leave one long chain.  The lines at 5500 and 8 heads are those of a slower backward: beyond them the kernels here now
    take as long or less where there are heads enough (B4 S7000 H16 D64 2601 / 2430, B2 S7000 H16 D128 2048 / 1965, B1 S3000 H2 D64
    145 / 112).  The forward alone is up to 30 % faster in torch's operator from S 1500 on (B4 S1543 H16 D128 58 / 72, B2 S4095 H16
    D64 97 / 113, short ones are bound by the host, B1 S77 23 / 18, B4 S1000 H16 D64 27 / 26).  Only inference mode may go by that: a
    forward without gradients may be the first pass of a checkpointed block, whose repetition has to compute the same."""
    if inference:
        return S <= 1024 and B * H * S <= 65536
    return S <= 2048 or (S <= 5500 and B * H >= 8)


def _native_takes(qkv: torch.Tensor, n_heads: int, D: int, scale: float) -> bool:
    """Does this call run the tcgen05 kernels?  bf16 and head size 64 or 128; whole tiles (a length that is a multiple of 128)
    always, any other length where they are faster, unless the call asks for what only torch's own operator offers: a functorch transform, forward-mode
    differentiation, tracing, a softmax scale that is not positive, an empty tensor, autocast to another dtype."""
    if not (_bind.use_native(qkv) and qkv.dtype == torch.bfloat16 and D in (64, 128) and _native_available()):
        return False
    if qkv.shape[1] % 128 == 0:
        return True
    if qkv.numel() == 0 or qkv.shape[2] != 3 * n_heads * D or not (0.0 < scale < math.inf):
        return False
    if not _native_is_faster(qkv.shape[0], qkv.shape[1], n_heads, torch.is_inference_mode_enabled()):
        return False
    if torch.is_autocast_enabled("cuda") and torch.get_autocast_dtype("cuda") != qkv.dtype:
        return False
    return not (torch._C._are_functorch_transforms_active() or torch.autograd.forward_ad._current_level >= 0 or torch.compiler.is_compiling())


def causal_attention(qkv: torch.Tensor, n_heads: int, scale: Optional[float] = None) -> torch.Tensor:
    global BACKEND
    B, S, three_hd = qkv.shape
    D = three_hd // (3 * n_heads)
    scale = scale if scale is not None else 1.0 / math.sqrt(D)
    if _native_takes(qkv, n_heads, D, scale):
        from .attention_native import flash_attention_packed

        BACKEND = "tcgen05"
        return flash_attention_packed(qkv, n_heads, scale)
    q, k, v = qkv.view(B, S, 3, n_heads, D).permute(2, 0, 3, 1, 4)
    if qkv.is_cuda:
        global _WARNED_LIBRARY_PATH
        if not _WARNED_LIBRARY_PATH:
            _WARNED_LIBRARY_PATH = True
            warnings.warn(
                f"causal_attention: the tcgen05 kernels take bf16 with head size 64 or 128, and lengths that are no multiple of 128 where they "
                f"are faster (got {qkv.dtype}, head size {D}, length {S}); this call runs torch's scaled_dot_product_attention instead",
                stacklevel=2,
            )
        BACKEND = "torch-sdpa"
        o = torch.nn.functional.scaled_dot_product_attention(q, k, v, is_causal=True, scale=scale)
    else:
        BACKEND = "reference"
        o = _reference(q, k, v, scale).to(qkv.dtype)
    return o.transpose(1, 2).reshape(B, S, n_heads * D)
