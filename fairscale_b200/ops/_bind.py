"""ctypes signatures of the native library and small marshalling helpers."""

from __future__ import annotations

import ctypes
from ctypes import c_float, c_int, c_longlong, c_uint, c_ulonglong, c_void_p
from typing import Any, Optional

import torch

from .. import _native

_DTYPE_CODE = {torch.float32: 0, torch.float16: 1, torch.bfloat16: 2}

_SIGNATURES = {
    "fsb_gemm_bf16": [c_void_p] * 6 + [c_int] * 13 + [c_void_p, c_void_p],
    "fsb_gemm_bf16_streamed_a": [c_void_p] * 4 + [c_int] * 7 + [c_void_p, c_uint] + [c_int] * 4 + [c_longlong, c_void_p, c_void_p],
    "fsb_gemm_bf16_streamed_b": [c_void_p] * 4 + [c_int] * 6 + [c_void_p, c_uint, c_longlong, c_int, c_longlong, c_void_p, c_void_p],
    "fsb_adam_chunk_size": [],
    "fsb_multi_tensor_adam": [c_void_p, c_int, c_longlong, c_int, c_int, c_int, c_int] + [c_float] * 8 + [c_int, c_int, c_void_p, c_void_p, c_void_p, c_void_p],
    "fsb_multi_tensor_sumsq": [c_void_p, c_int, c_longlong, c_int, c_void_p, c_void_p],
    "fsb_multi_tensor_scale": [c_void_p, c_int, c_longlong, c_int, c_void_p, c_void_p, c_void_p],
    "fsb_norm_fwd": [c_void_p] * 6 + [c_longlong, c_int, c_float, c_int, c_void_p],
    "fsb_norm_bwd_res": [c_void_p] * 10 + [c_longlong, c_int, c_int, c_void_p],
    "fsb_norm_bwd_num_strips": [c_longlong],
    "fsb_colsum_num_strips": [c_longlong],
    "fsb_colsum": [c_void_p, c_longlong, c_int, c_void_p, c_void_p, c_void_p],
    "fsb_colsum_batched": [c_void_p, c_int, c_longlong, c_int, c_void_p, c_void_p, c_void_p],
    "fsb_ce_fwd_dtype": [c_void_p, c_int] + [c_void_p] * 4 + [c_longlong, c_int, c_longlong, c_longlong, c_longlong, c_void_p],
    "fsb_ce_bwd_dtype": [c_void_p, c_int] + [c_void_p] * 3 + [c_int, c_float, c_void_p, c_longlong, c_int, c_longlong, c_longlong, c_longlong, c_void_p],
    "fsb_moe_claim_rows": [c_void_p] * 3 + [c_longlong] * 3 + [c_void_p] * 3,
    "fsb_moe_scatter_local": [c_void_p, c_int, c_void_p, c_void_p, c_longlong, c_int, c_void_p, c_void_p, c_longlong, c_void_p],
    "fsb_moe_gather_local": [c_void_p, c_int, c_void_p, c_void_p, c_longlong, c_int] + [c_void_p] * 5,
    "fsb_embedding_fwd": [c_void_p] * 4 + [c_longlong, c_int, c_int, c_longlong, c_longlong, c_float, c_void_p],
    "fsb_embedding_bwd": [c_void_p] * 4 + [c_longlong, c_int, c_int, c_longlong, c_longlong, c_float, c_void_p],
    "fsb_cast": [c_void_p, c_int, c_void_p, c_int, c_longlong, c_float, c_void_p],
    "fsb_accum_bf16_into_f32": [c_void_p, c_void_p, c_longlong, c_float, c_int, c_void_p],
    "fsb_gelu": [c_void_p, c_void_p, c_void_p, c_longlong, c_int, c_void_p],
    "fsb_swiglu_fwd": [c_void_p, c_void_p, c_longlong, c_int, c_void_p],
    "fsb_swiglu_bwd": [c_void_p, c_void_p, c_void_p, c_longlong, c_int, c_void_p],
    "fsb_add_bf16": [c_void_p, c_void_p, c_void_p, c_longlong, c_void_p],
    "fsb_rope": [c_void_p, c_void_p, c_longlong, c_int, c_int, c_int, c_float, c_int, c_int, c_void_p],
    "fsb_dropout": [c_void_p, c_void_p, c_longlong, c_float, c_ulonglong, c_ulonglong, c_void_p],
    "fsb_delay": [c_ulonglong, c_void_p],
    "fsb_softmax": [c_void_p, c_void_p, c_longlong, c_int, c_int, c_float, c_int, c_int, c_void_p],
}

_bound: dict = {}
_launch_count = 0


def fn(name: str) -> Any:
    """Bound native function with argtypes set (cached)."""
    f = _bound.get(name)
    if f is None:
        f = getattr(_native.lib(), name)
        if name in _SIGNATURES:
            f.argtypes = _SIGNATURES[name]
        f.restype = c_int
        _bound[name] = f
    return f


def call(name: str, *args: Any, launches: int = 1) -> None:
    """Invoke a native entry point and raise on a non-zero return code."""
    global _launch_count
    code = fn(name)(*args)
    if code != 0:
        raise RuntimeError(f"{name} failed with code {code}")
    _launch_count += launches


def launch_count() -> int:
    """Number of kernels of this library launched so far by this process."""
    return _launch_count


def add_launches(n: int) -> None:
    global _launch_count
    _launch_count += n


def ptr(t: Optional[torch.Tensor]) -> Optional[int]:
    return None if t is None else t.data_ptr()


def dense16(t: torch.Tensor) -> torch.Tensor:
    """``t`` contiguous and starting on a 16-byte boundary, as kernels with 16-byte accesses and TMA tensor maps need it (a view
    may start at any element)."""
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


def _device_index(device: Any) -> int:
    index = device.index if isinstance(device, torch.device) else (device if isinstance(device, int) else None)
    if index is None:
        index = torch.device(device).index if device is not None and not isinstance(device, torch.device) else None
    return torch.cuda.current_device() if index is None else index


def stream_ptr(device: Any = None) -> int:
    """Raw handle of the current stream (without building a ``torch.cuda.Stream`` around it for every launch)."""
    return torch._C._cuda_getCurrentRawStream(_device_index(device))


def dtype_code(dt: torch.dtype) -> int:
    return _DTYPE_CODE[dt]


def use_native(*tensors: Any) -> bool:
    return _native.use_native(*tensors)


_status_ptrs: dict = {}  # device index -> address of its status word (allocated once per process)


def status_ptr(device: Any) -> int:
    index = _device_index(device)
    ptr_ = _status_ptrs.get(index)
    if ptr_ is None:
        ptr_ = _status_ptrs[index] = _native.status_word(index).data_ptr()
    return ptr_


def no_graph() -> bool:
    """True when an operation may run without its autograd node: gradients are off, and nothing else (forward-mode
    differentiation, a functorch transform, a tracer) has to see the node either."""
    return not (torch.is_grad_enabled() or torch.autograd.forward_ad._current_level >= 0 or torch._C._are_functorch_transforms_active()
                or torch.compiler.is_compiling())
