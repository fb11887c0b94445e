"""The native host module against the python autograd functions that calls under tracing, modes and subclasses keep: the same
kernels on the same values, so every result is the same bit for bit - except where atomics order a sum (dQ of attention)."""
import importlib

import pytest
import torch

from colossalai_b200 import ops
from colossalai_b200.kernel import loader
from colossalai_b200.ops import inference
from colossalai_b200.shardformer.layer import loss as loss_mod

MODULES = [importlib.import_module("colossalai_b200.ops." + m) for m in ("norm", "activation", "attention", "inference", "rope")] + [loss_mod]


def test_plain_call_sees_what_watches():
    from torch.autograd import forward_ad
    from torch.utils._python_dispatch import TorchDispatchMode

    from colossalai_b200.ops._dispatch import plain_call
    from colossalai_b200.tensor import ColoParameter

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, f, types, args=(), kwargs=None):
            return f(*args, **(kwargs or {}))

    x, seen = torch.randn(3), []
    assert plain_call(x, None, torch.nn.Parameter(x))
    assert not plain_call(x, ColoParameter(x.clone()))
    look = lambda t: (seen.append(plain_call(t)), t + 1)[1]      # noqa: E731
    torch.func.vmap(look)(x)
    torch.func.grad(lambda t: look(t).sum())(x)
    with forward_ad.dual_level():
        look(x)
    with Mode():
        look(x)
    torch.jit.trace(look, x, check_trace=False)
    assert seen == [False] * 5 and plain_call(x)


@pytest.mark.parametrize("why", ["no rebuild", "build fails", "does not load"])
def test_a_host_module_of_other_sources_is_not_taken(monkeypatch, tmp_path, why):
    """One built for another torch or other launchers, whatever lies in the build folder: the python functions remain."""
    def build(name, **kw):
        if why == "build fails":
            raise RuntimeError("no compiler here")

    (tmp_path / "libcb200_host.so").write_bytes(b"of another torch")
    monkeypatch.setattr(loader, "BUILD", tmp_path)
    monkeypatch.setattr(loader, "build", build)
    monkeypatch.setattr(loader, "load", lambda name: None)
    monkeypatch.setattr(loader, "_host", None)
    monkeypatch.setattr(loader, "_host_asked", False, raising=False)
    monkeypatch.setenv("CB200_NO_REBUILD", "1" if why == "no rebuild" else "0")
    with pytest.warns(UserWarning, match="host module is not used"):
        assert loader.host() is None
    assert loader.host() is None


@pytest.mark.gpu
def test_calls_without_a_host_module(monkeypatch):
    monkeypatch.setattr(loader, "_host", None)
    monkeypatch.setattr(loader, "_host_asked", True)
    x = torch.randn(6, 64, device="cuda", dtype=torch.bfloat16)
    cu = torch.tensor([0, 6], device="cuda", dtype=torch.int32)
    cache = torch.randn(2, 16, 1, 64, device="cuda", dtype=torch.bfloat16)
    pages = torch.tensor([[0], [1]], device="cuda", dtype=torch.int32)
    calls = [lambda: ops.rms_norm(x, x[0]), lambda: ops.rms_norm(x, x[0], 1e-6, x), lambda: ops.glu(x),
             lambda: ops.rope_qkv(x, None, *ops.build_rope_cache(8, 16, 1e4, device="cuda"), 2, 1, 16),
             lambda: ops.attention(x.view(6, 1, 64), x.view(6, 1, 64), x.view(6, 1, 64), cu_seqlens_q=cu),
             lambda: inference.paged_decode_attention(x[:2].view(2, 1, 64), cache, cache, pages, torch.full_like(cu, 6)),
             lambda: loss_mod.cross_entropy_1d(x, torch.zeros(6, dtype=torch.int64, device="cuda"), process_group="local")]
    for call in calls:
        before = loader.launch_counter.count
        call()
        assert loader.launch_counter.count > before


def _both(monkeypatch, fn):
    """fn() on the host module and on the python functions; how many launches each made."""
    out = []
    for plain in (None, lambda *a: False):
        with monkeypatch.context() as m:
            if plain is not None:
                for mod in MODULES:
                    m.setattr(mod, "plain_call", plain)
            else:
                loader.host()
            loader.launch_counter.reset()
            out.append(fn())
            torch.cuda.synchronize()
            out.append(loader.launch_counter.count)
    assert out[1] == out[3] > 0, "the same kernels on both ways"
    return out[0], out[2]


def _same(a, b):
    assert len(a) == len(b)
    for x, y in zip(a, b):
        assert (x is None) == (y is None)
        if x is not None:
            assert x.dtype == y.dtype and x.shape == y.shape and torch.equal(x, y)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shape", [(1, 8), (3, 5, 64), (300, 4096)])
@pytest.mark.parametrize("use", ["both", "norm", "sum", "no_residual"])
def test_rms_norm(monkeypatch, dtype, shape, use):
    def fn():
        torch.manual_seed(0)
        x = torch.randn(shape[-1:] + shape[:-1], device="cuda", dtype=dtype).movedim(0, -1).requires_grad_()     # strided rows
        r = torch.randn(shape, device="cuda", dtype=dtype, requires_grad=True)
        w = torch.nn.Parameter(torch.rand(shape[-1], device="cuda", dtype=dtype))
        if use == "no_residual":
            y = ops.rms_norm(x, w, 1e-5)
            y.backward(torch.randn_like(y))
            return y.detach(), x.grad, w.grad
        y, h = ops.rms_norm(x, w, 1e-5, r)
        outs = {"both": (y, h), "norm": (y,), "sum": (h,)}[use]
        torch.autograd.backward(outs, [torch.randn(shape, device="cuda").to(dtype) for _ in outs])
        return y.detach(), h.detach(), x.grad, r.grad, w.grad

    _same(*_both(monkeypatch, fn))


@pytest.mark.gpu
@pytest.mark.parametrize("act", ["silu", "gelu_tanh", "gelu"])
def test_glu_saved_tensor_hooks_and_checkpoint(monkeypatch, act):
    from torch.autograd.graph import saved_tensors_hooks
    from torch.utils.checkpoint import checkpoint

    def fn():
        torch.manual_seed(0)
        gu = torch.randn(2, 7, 48, device="cuda", dtype=torch.bfloat16, requires_grad=True)
        packed = []
        with saved_tensors_hooks(lambda t: (packed.append(t.shape), t.cpu())[1], lambda t: t.cuda()):
            y = ops.glu(gu, act)
        assert packed
        (g1,) = torch.autograd.grad(y, gu, torch.ones_like(y))
        z = checkpoint(lambda t: ops.glu(t, act), gu, use_reentrant=False)
        (g2,) = torch.autograd.grad(z, gu, torch.ones_like(z))
        return y.detach(), g1, z.detach(), g2

    _same(*_both(monkeypatch, fn))


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(0, 24 * 16), (3, 24 * 16), (3, 24, 16)])
def test_rope(monkeypatch, shape):
    def fn():
        torch.manual_seed(0)
        x = torch.randn(shape, device="cuda", requires_grad=True)
        pos = torch.arange(shape[0], device="cuda")
        y = ops.rope_qkv(x, pos, *ops.build_rope_cache(8, 16, 1e4, device="cuda"), 16, 4, 16)
        return y.detach(), torch.autograd.grad(y, x, torch.ones((), device="cuda").expand(shape))[0]

    _same(*_both(monkeypatch, fn))


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["mean", "sum"])
@pytest.mark.parametrize("vocab", [1000, 1024])
@pytest.mark.parametrize("labels", [torch.int64, torch.int32])
def test_cross_entropy(monkeypatch, mode, vocab, labels):
    def fn():
        torch.manual_seed(0)
        x = torch.randn(33, 1024, device="cuda", dtype=torch.bfloat16, requires_grad=True)
        t = torch.randint(0, vocab, (33,), device="cuda")
        t[::5] = -100
        out = loss_mod.cross_entropy_1d(x, t.to(labels), process_group="local", vocab_size=vocab, mode=mode)
        (g,) = torch.autograd.grad(out * 3, x)
        return out.detach(), g

    _same(*_both(monkeypatch, fn))


@pytest.mark.gpu
@pytest.mark.parametrize("D,grad", [(128, True), (128, False), (64, False)])
def test_packed_attention(monkeypatch, D, grad):
    def fn():
        torch.manual_seed(0)
        q, k, v = (torch.randn(300, h, D, device="cuda", dtype=torch.bfloat16, requires_grad=grad) for h in (8, 2, 2))
        cu = torch.tensor([0, 7, 7, 200, 300], device="cuda")
        o = ops.attention(q, k, v, causal=True, cu_seqlens_q=cu, cu_seqlens_k=cu)
        return (o.detach(),) + (torch.autograd.grad(o, (q, k, v), torch.ones(300, 8, 1, device="cuda").bfloat16().expand(300, 8, D))
                                if grad else ())

    a, b = _both(monkeypatch, fn)
    _same(a[:1] + a[2:], b[:1] + b[2:])
    if grad:
        torch.testing.assert_close(a[1], b[1], rtol=2 ** -7, atol=2e-3)      # fp32 sums in the order of the reductions


@pytest.mark.gpu
def test_packed_attention_boundaries_refilled(monkeypatch):
    """A static buffer of boundaries that is written again between forward and backward (the same contents here), and what
    saved-tensor hooks get to see."""
    from torch.autograd.graph import saved_tensors_hooks

    def fn():
        torch.manual_seed(0)
        q, k, v = (torch.randn(150, h, 128, device="cuda", dtype=torch.bfloat16, requires_grad=True) for h in (4, 2, 2))
        cu = torch.tensor([0, 40, 150], device="cuda", dtype=torch.int32)
        seen = []
        with saved_tensors_hooks(lambda t: (seen.append(t.dtype), t)[1], lambda t: t):
            o = ops.attention(q, k, v, causal=True, cu_seqlens_q=cu, cu_seqlens_k=cu)
        cu.copy_(torch.tensor([0, 40, 150], dtype=torch.int32))
        grads = torch.autograd.grad(o, (q, k, v), torch.ones_like(o))
        assert seen == [torch.bfloat16] * 4 + [torch.float32]
        return (o.detach(),) + grads[1:]                                     # (dQ is summed in the order of its reductions)

    _same(*_both(monkeypatch, fn))


@pytest.mark.gpu
@pytest.mark.parametrize("D", [64, 256])
def test_paged_decode(monkeypatch, D):
    def fn():
        torch.manual_seed(0)
        qkv = torch.randn(5, (8 + 4) * D, device="cuda", dtype=torch.float16)
        kc, vc = (torch.randn(40, 16, 2, D, device="cuda", dtype=torch.float16) for _ in range(2))
        tables = torch.randperm(40, device="cuda")[:40].view(5, 8).int()
        lens = torch.tensor([1, 16, 100, 128, 77], device="cuda", dtype=torch.int32)
        q = qkv[:, : 8 * D].view(5, 8, D)                                         # rows of a wider projection
        return inference.paged_decode_attention(q, kc, vc, tables, lens, window=50),

    _same(*_both(monkeypatch, fn))


@pytest.mark.gpu
@pytest.mark.parametrize("T,E,k,H,inter", [(1, 8, 2, 64, 64), (37, 16, 4, 256, 192), (700, 64, 6, 128, 64), (300, 5, 1, 512, 40)])
@pytest.mark.parametrize("mode", ["grad", "no_grad", "inference", "frozen"])
def test_local_experts(monkeypatch, T, E, k, H, inter, mode):
    """A layer of local experts (outputs of no multiple of 128 included, whose input gradient is not this module's): the same bits and
    products without the module, with weights that need no gradient, and with choices of no expert."""
    from colossalai_b200.models import get_config
    from colossalai_b200.models.moe import GroupedExperts
    from colossalai_b200.moe.dispatch_combine import moe_forward

    g = torch.Generator(device="cuda").manual_seed(T)
    experts = GroupedExperts(get_config("deepseek-moe-16b", hidden_size=H), E, inter).cuda().bfloat16()
    for p in experts.parameters():
        p.requires_grad_(mode != "frozen")
    x0 = torch.randn(T, H, device="cuda", generator=g).bfloat16()
    score = torch.rand(T, E, device="cuda", generator=g)
    dy = torch.randn(T, H, device="cuda", generator=g).bfloat16()

    def fn():
        x = x0.clone().requires_grad_(mode in ("grad", "frozen"))
        w, idx = score.topk(k, dim=-1)
        idx[T // 2, 0] = E                                        # its token's sum is NaN
        w = w.detach().requires_grad_(mode == "grad")
        with torch.inference_mode() if mode == "inference" else torch.set_grad_enabled(mode != "no_grad"):
            y = moe_forward(x, w, idx, experts, E, None)
        if not y.requires_grad:
            return [y]
        ins = [t for t in (x, w, *experts.parameters()) if t.requires_grad]
        return [y, *torch.autograd.grad(y, ins, dy)]

    out = []
    for without in (False, True):
        with monkeypatch.context() as m:
            if without:
                m.setattr(loader, "_host", None)
                m.setattr(loader, "_host_asked", True)
            else:
                loader.host()
            loader.launch_counter.reset()
            out.append([t.nan_to_num(nan=7.0) for t in fn()])
            out.append(dict(loader.launch_counter.by_name))
    _same(out[0], out[2])
    without_unit = [{name: n for name, n in o.items() if "glu" not in name} for o in (out[1], out[3])]      # (in the products, with the module)
    assert without_unit[0] == without_unit[1] and out[1]["grouped_gemm"] >= 2


@pytest.mark.gpu
def test_counts_written_to_after_the_sort():
    """The running sums that the sort wrote beside the counts are not taken for counts that changed since."""
    from colossalai_b200.moe.grouped_gemm import rows_of
    from colossalai_b200.ops.moe import expert_ends, sort_choices

    idx = torch.tensor([[0, 2], [2, 5]], device="cuda")
    _, _, counts = sort_choices(idx, 6, 16)
    ends, total = expert_ends(counts)
    assert counts.tolist() == [16, 0, 16, 0, 0, 16] and ends.tolist() == [16, 16, 32, 32, 32, 48] and int(total) == int(rows_of(counts)) == 48
    counts[1] += 16
    assert expert_ends(counts) == (None, None) and int(rows_of(counts)) == 64 and expert_ends(counts + 0) == (None, None)
