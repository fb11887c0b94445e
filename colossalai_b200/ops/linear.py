"""Projections of a few token rows: what a decode step spends most of its time on.

A plain `torch.nn.Linear` without bias on up to ROWS_MAX 16-bit rows, outside autograd, runs on the framework's own kernel
(`kernel/csrc/gemm_rows_tcgen05.cu`: weights streamed once, fp32 sums, residual added before the rounding); every other call is
the module's own.
"""
from __future__ import annotations

import functools
from typing import Optional

import torch
from torch import nn
from torch.nn.modules import module as _module

from ..kernel import loader
from ._dispatch import plain_call, use_native
from .activation import glu

__all__ = ["linear_rows", "gated_rows", "embed_rows", "unwatched", "ROWS_MAX"]

ROWS_MAX = 32         # what the kernel takes; figures there
_LINEAR, _EMBEDDING = nn.Linear.forward, nn.Embedding.forward


def unwatched(m: nn.Module, forward) -> bool:
    """A call of the module runs `forward`, what its class came with, and nothing else: it is replaced neither on the instance (as
    `convert_linear_to_fp8` and adapters do) nor on the class, not compiled, and no hook sees the call."""
    if type(m).forward is not forward or "forward" in m.__dict__ or m._compiled_call_impl is not None:
        return False
    return not (m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks
                or _module._global_forward_hooks or _module._global_forward_pre_hooks
                or _module._global_backward_hooks or _module._global_backward_pre_hooks)


@functools.lru_cache(maxsize=None)
def _sm100(device: torch.device) -> bool:
    return torch.cuda.get_device_capability(device)[0] == 10


def _native(linear: nn.Module, x: torch.Tensor, residual: Optional[torch.Tensor]) -> bool:
    if type(linear) is not nn.Linear or torch.is_grad_enabled() or not use_native(x) or x.dim() != 2 or not 0 < x.shape[0] <= ROWS_MAX:
        return False
    w = linear.weight
    if linear.bias is not None or w.dtype != x.dtype or x.dtype not in (torch.bfloat16, torch.float16) or w.device != x.device:
        return False
    # (before strides and pointers are looked at: what vmap, tracing or a mode hands in may have neither)
    if not plain_call(x, w, residual) or not unwatched(linear, _LINEAR) or torch.is_autocast_enabled("cuda"):
        return False
    n, k = w.shape
    # one contiguous weight, rows that TMA can address
    if x.shape[1] != k or k % 8 or k == 0 or n == 0 or not w.is_contiguous() or x.stride(1) != 1 or x.stride(0) % 8 or x.stride(0) < k \
            or (x.data_ptr() | w.data_ptr()) % 16:
        return False
    if residual is not None and (residual.shape != (x.shape[0], n) or residual.dtype != x.dtype or residual.device != x.device
                                 or residual.stride(1) != 1):
        return False
    return _sm100(x.device)


def linear_rows(linear: nn.Module, x: torch.Tensor, residual: Optional[torch.Tensor] = None) -> torch.Tensor:
    """linear(x), plus `residual` if there is one."""
    if _native(linear, x, residual) and (host := loader.host()) is not None:
        return host.linear_rows(x, linear.weight, residual)
    y = linear(x)
    return y if residual is None else residual + y


_GATED = {"silu": 0, "swiglu": 0, "gelu_tanh": 1, "gelu_new": 1, "gelu_pytorch_tanh": 1, "gelu": 2, "geglu": 2}


def gated_rows(linear: nn.Module, x: torch.Tensor, act: str) -> torch.Tensor:
    """glu(linear(x), act), the unit in the projection's epilogue where that is the framework's own kernel: a decode step then has one launch
    less a layer, with the same roundings."""
    if act in _GATED and _native(linear, x, None) and linear.weight.shape[0] % 16 == 0 and (host := loader.host()) is not None:
        return host.gated_rows(x, linear.weight, _GATED[act])
    return glu(linear_rows(linear, x), act)


def _native_lookup(embedding: nn.Module, ids: torch.Tensor) -> bool:
    if type(embedding) is not nn.Embedding or embedding.max_norm is not None or torch.is_grad_enabled() or not use_native(ids):
        return False
    w = embedding.weight
    if not plain_call(ids, w) or not unwatched(embedding, _EMBEDDING):
        return False
    return (ids.dim() == 1 and ids.dtype == torch.int64 and ids.is_contiguous() and ids.numel() > 0 and w.device == ids.device
            and w.dtype in (torch.bfloat16, torch.float16, torch.float32) and w.is_contiguous()
            and w.shape[1] * w.element_size() % 16 == 0 and w.shape[1] > 0 and w.data_ptr() % 16 == 0)


def embed_rows(embedding: nn.Module, ids: torch.Tensor) -> torch.Tensor:
    """embedding(ids).  Outside autograd the rows of a plain table come through a kernel with a block per id (16 rows of 4096: 2.6 us,
    torch's index kernel 14); an id outside the table ends in a device assertion there too."""
    if _native_lookup(embedding, ids) and (host := loader.host()) is not None:
        return host.embed_rows(ids, embedding.weight)
    return embedding(ids)
