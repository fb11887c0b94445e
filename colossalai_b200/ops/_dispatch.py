"""Native-vs-reference dispatch policy shared by every op.

Rule: CUDA tensors -> the sm_100a kernel (hard error if its library is missing on a GPU box);
CPU tensors -> the plain PyTorch reference (CPU plumbing tier).  `CB200_FORCE_TORCH=1` forces the reference
path on GPU too (used by the numerics tests and by the "baseline mode" of the benchmarks).
"""
from __future__ import annotations

import os
from contextlib import contextmanager

import torch
from torch.autograd import forward_ad

_force_torch = os.environ.get("CB200_FORCE_TORCH", "0") == "1"


def use_native(*tensors: torch.Tensor) -> bool:
    if _force_torch:
        return False
    for t in tensors:
        if t is not None:
            return t.is_cuda
    return False


_functorch_level = torch._C._functorch.peek_interpreter_stack
_tracing = torch._C._get_tracing_state
_dispatch_modes, _function_modes = torch._C._len_torch_dispatch_stack, torch._C._len_torch_function_stack
_compiling = torch.compiler.is_compiling


def plain_call(*tensors) -> bool:
    """True when nothing but autograd watches a call: tensors of no subclass, no tracing or compilation, no functorch level,
    no forward-mode level, no dispatch or function mode.  Such calls may take the native host module (`kernel.loader.host`);
    the others keep the python autograd functions, which behave under all of these as they always did."""
    for t in tensors:
        if t is not None and type(t) is not torch.Tensor and type(t) is not torch.nn.Parameter:
            return False
    return not (_dispatch_modes() or _function_modes() or forward_ad._current_level >= 0 or _functorch_level() is not None
                or _tracing() is not None or _compiling())


@contextmanager
def force_torch(enabled: bool = True):
    """Context manager: run ops through their PyTorch reference implementation."""
    global _force_torch
    prev = _force_torch
    _force_torch = enabled
    try:
        yield
    finally:
        _force_torch = prev


def is_forced_torch() -> bool:
    return _force_torch
