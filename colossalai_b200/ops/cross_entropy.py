"""Building blocks of the (vocab-parallel) cross entropy: row statistics (max, sum-exp, target logit) in one pass over the
logits, the loss from them, softmax gradient.

Native path: `kernel/csrc/cross_entropy.cu`.  Reference path: PyTorch fp32.
Parity: the math of reference `DistCrossEntropy` (`colossalai/shardformer/layer/loss.py:25-127`).
"""
from __future__ import annotations

import ctypes
from typing import Optional

import torch

from ..kernel import loader
from ._dispatch import use_native
from ._dtypes import code

_lib = None


def _get_lib():
    global _lib
    if _lib is None:
        _lib = loader.load("cb200_loss")
    return _lib


def _ok(logits: torch.Tensor) -> bool:
    vec = 4 if logits.dtype == torch.float32 else 8
    return (use_native(logits) and logits.dtype in (torch.float32, torch.float16, torch.bfloat16)
            and logits.shape[-1] % vec == 0 and logits.is_contiguous())


def row_stats(logits: torch.Tensor, target: torch.Tensor, vocab_start: int, ignore_index: int,
              valid_cols: Optional[int] = None) -> torch.Tensor:
    """Returns fp32 [3, T]: row 0 = max_j x_j; row 1 = sum_j exp(x_j - max); row 2 = x_target if this rank owns the target
    else 0.  The logits are read once.  Without columns: -inf, 0, 0."""
    T, V = logits.shape
    Vv = V if valid_cols is None else valid_cols
    if _ok(logits):
        lib = _get_lib()
        out = torch.empty(3, T, dtype=torch.float32, device=logits.device)
        tgt = target if target.dtype == torch.int64 else target.long()
        loader.check(lib.cb_ce_row_stats(loader.ptr(logits), loader.ptr(tgt.contiguous()), loader.ptr(out), T, V, Vv,
                                         ctypes.c_int64(vocab_start), ctypes.c_int64(ignore_index), code(logits.dtype),
                                         loader.stream_ptr()), "ce_row_stats")
        loader.launch_counter.add("ce_row_stats")
        return out
    if Vv <= 0:
        zero = torch.zeros(T, dtype=torch.float32, device=logits.device)
        return torch.stack([zero - float("inf"), zero, zero], 0)
    xf = logits[:, :Vv].float()
    gmax = xf.max(dim=-1).values
    local = target - vocab_start
    own = (local >= 0) & (local < Vv) & (target != ignore_index)
    tl = xf.gather(-1, local.clamp(0, Vv - 1).unsqueeze(-1)).squeeze(-1)
    ref = torch.where(torch.isneginf(gmax), torch.zeros_like(gmax), gmax)    # a row of -inf sums to 0, as in the kernel
    return torch.stack([gmax, torch.exp(xf - ref.unsqueeze(-1)).sum(-1), torch.where(own, tl, torch.zeros_like(tl))], 0)


def rescale(stats: torch.Tensor, gmax: torch.Tensor) -> torch.Tensor:
    """Rows 1, 2 of `row_stats` with the sums taken against `gmax` (the maximum over all shards) instead of the shard's own:
    fp32 [2, T].  A shard without columns contributes nothing."""
    s = stats[1] * torch.exp(stats[0] - gmax)
    return torch.stack([torch.where(stats[1] == 0, torch.zeros_like(s), s), stats[2]], 0)


def row_max(logits: torch.Tensor, valid_cols: Optional[int] = None) -> torch.Tensor:
    return row_stats(logits, torch.zeros(logits.shape[0], dtype=torch.int64, device=logits.device), 0, 0, valid_cols)[0]


def sumexp_and_target(logits: torch.Tensor, target: torch.Tensor, gmax: torch.Tensor, vocab_start: int,
                      ignore_index: int, valid_cols: Optional[int] = None) -> torch.Tensor:
    """Returns fp32 [2, T]: row 0 = sum_j exp(x_j - gmax); row 1 = x_target if this rank owns the target else 0."""
    return rescale(row_stats(logits, target, vocab_start, ignore_index, valid_cols), gmax)


def loss_from_stats(stats: torch.Tensor, target: torch.Tensor, ignore_index: int, mean: bool):
    """(loss fp32 scalar, number of labels int64 scalar) from `row_stats` over the whole vocabulary: the sum over the rows
    with a label of log(sum-exp) + max - target logit, with `mean` divided by their number (at least 1)."""
    if use_native(stats):
        loss = torch.empty((), dtype=torch.float32, device=stats.device)
        n_valid = torch.empty((), dtype=torch.int64, device=stats.device)
        tgt = target if target.dtype == torch.int64 else target.long()
        blocks = _get_lib().cb_ce_loss_blocks(stats.shape[1])
        parts = torch.empty(2 * blocks, dtype=torch.float64, device=stats.device) if blocks > 1 else None
        loader.check(_get_lib().cb_ce_loss(loader.ptr(stats), loader.ptr(tgt.contiguous()), loader.ptr(loss),
                                           loader.ptr(n_valid), loader.ptr(parts), stats.shape[1], ctypes.c_int64(ignore_index),
                                           int(mean), loader.stream_ptr()), "ce_loss")
        loader.launch_counter.add("ce_loss", 1 + (blocks > 1))
        return loss, n_valid
    valid = target != ignore_index
    n_valid = valid.sum()
    loss = torch.where(valid, torch.log(stats[1]) + stats[0] - stats[2], torch.zeros_like(stats[0])).sum()
    return (loss / n_valid.clamp(min=1) if mean else loss), n_valid


def softmax_grad(logits: torch.Tensor, target: torch.Tensor, gmax: torch.Tensor, sumexp: torch.Tensor,
                 scale: Optional[torch.Tensor], vocab_start: int, ignore_index: int,
                 row_scale: Optional[torch.Tensor] = None, valid_cols: Optional[int] = None,
                 n_valid: Optional[torch.Tensor] = None) -> torch.Tensor:
    """grad[t, j] = s_t * (softmax(x)[t, j] - 1[j == target_t])  with s_t = row_scale[t], or scale (scalar tensor; divided by
    max(n_valid, 1), an int64 scalar tensor, when that is given); rows whose target == ignore_index get zero."""
    T, V = logits.shape
    Vv = V if valid_cols is None else valid_cols
    if _ok(logits):
        lib = _get_lib()
        out = torch.empty_like(logits)
        tgt = target if target.dtype == torch.int64 else target.long()
        rs = None if row_scale is None else row_scale.contiguous()
        one = None if rs is not None else scale.reshape(1).float()
        loader.check(lib.cb_ce_softmax_grad(loader.ptr(logits), loader.ptr(tgt.contiguous()), loader.ptr(gmax.contiguous()),
                                            loader.ptr(sumexp.contiguous()), loader.ptr(rs), loader.ptr(one),
                                            loader.ptr(None if rs is not None else n_valid), loader.ptr(out),
                                            T, V, Vv, ctypes.c_int64(vocab_start), ctypes.c_int64(ignore_index),
                                            code(logits.dtype), loader.stream_ptr()), "ce_softmax_grad")
        loader.launch_counter.add("ce_softmax_grad")
        return out
    if row_scale is None:
        scale = scale if n_valid is None else scale / n_valid.clamp(min=1)
        row_scale = scale.reshape(1).expand(T).float()
    xf = logits[:, :Vv].float()
    p = torch.exp(xf - gmax.unsqueeze(-1)) / sumexp.unsqueeze(-1)
    local = target - vocab_start
    own = (local >= 0) & (local < Vv)
    idx = local.clamp(0, Vv - 1)
    onehot = torch.zeros_like(p)
    onehot.scatter_(-1, idx.unsqueeze(-1), own.float().unsqueeze(-1))
    g = (p - onehot) * row_scale.unsqueeze(-1)
    g = torch.where((target != ignore_index).unsqueeze(-1), g, torch.zeros_like(g))
    if Vv < V:
        g = torch.cat([g, g.new_zeros(T, V - Vv)], dim=-1)
    return g.to(logits.dtype)
