"""Projections of a few rows and the embedding lookup of a decode step, against 64-bit products of the same 16-bit numbers."""
import pytest
import torch
from torch import nn

# CTAs that share a reduction, on 148 SMs: 1, 1, 1, 4 (the last with less), 8, 4, 1, 8; 2, 8 (the last with nothing), the same with a
# tile that ends inside the width, 4 (17 k-blocks)
SIZES = [(8, 8), (128, 64), (136, 200), (264, 1096), (1000, 2048), (6144, 1024), (18944, 256), (512, 14336),
         (8, 512), (1024, 2112), (1000, 2112), (1536, 1088)]


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 15, 16, 17, 32])
@pytest.mark.parametrize("N,K", SIZES)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_rows_match_64_bits(rows, N, K, dtype):
    """Widths and depths that end inside a tile and a k-block, every number of splits of the reduction, with a residual and from
    rows that are a part of wider ones.  A row's bits do not depend on how many rows there are."""
    from colossalai_b200 import ops
    from colossalai_b200.kernel import launch_counter

    g = torch.Generator(device="cuda").manual_seed(N + K)
    lin = nn.Linear(K, N, bias=False, device="cuda", dtype=dtype)
    wide = torch.randn(rows, K + 24, device="cuda", generator=g).to(dtype)
    x = wide[:, 8:8 + K]
    res = torch.randn(rows, N, device="cuda", generator=g).to(dtype)
    ref = x.double() @ lin.weight.detach().double().t()
    # half a unit of the result's rounding, and fp32 sums of K products
    unit = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    slack = 1e-6 * (x.double().abs() @ lin.weight.detach().double().abs().t()) + 1e-7
    with torch.no_grad():
        before = launch_counter.by_name.get("gemm_rows", 0)
        y, z = ops.linear_rows(lin, x), ops.linear_rows(lin, x, res)
        alone = ops.linear_rows(lin, x[rows - 1:])
    assert launch_counter.by_name["gemm_rows"] == before + 3
    assert ((y.double() - ref).abs() <= unit * 1.01 * ref.abs() + slack).all()
    assert ((z.double() - (ref + res.double())).abs() <= unit * 1.01 * (ref + res.double()).abs() + slack).all()
    assert torch.equal(alone[0], y[-1])


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 16, 17, 32])
@pytest.mark.parametrize("I,K", [(8, 8), (64, 64), (72, 200), (704, 1096), (1408, 2048), (9472, 256), (256, 14336), (9536, 512), (512, 2112)])
@pytest.mark.parametrize("dtype,act", [(torch.bfloat16, "silu"), (torch.float16, "gelu_tanh"), (torch.bfloat16, "gelu")])
def test_gated_rows(rows, I, K, dtype, act):
    """The unit in the projection's epilogue against projection and unit one after the other: the same bits where both cut the matrix into
    the same tiles (multiples of 64), otherwise up to the order of fp32 sums, which may turn a rounding of either factor."""
    from colossalai_b200 import ops
    from colossalai_b200.kernel import launch_counter

    g = torch.Generator(device="cuda").manual_seed(I + K)
    lin = nn.Linear(K, 2 * I, bias=False, device="cuda", dtype=dtype)
    x = torch.randn(rows, K + 24, device="cuda", generator=g).to(dtype)[:, 8:8 + K]
    with torch.no_grad():
        want = ops.glu(ops.linear_rows(lin, x), act)
        launch_counter.reset()
        y = ops.gated_rows(lin, x, act)
        assert dict(launch_counter.by_name) == {"gemm_rows": 1}
        assert torch.equal(ops.gated_rows(lin, x[rows - 1:], act)[0], y[-1])
    assert y.shape == want.shape and y.dtype == dtype
    if I % 64 == 0:
        assert torch.equal(y, want)
    else:
        unit = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
        assert ((y - want).abs() <= 6 * unit * want.abs() + 1e-6).all()       # a unit of each factor and of the result, twice over
    y = ops.gated_rows(lin, x, act)                                           # autograd: the module and the unit
    assert y.requires_grad


@pytest.mark.gpu
def test_calls_that_stay_with_the_module():
    """Autograd, hooks, a bias, many rows, other types and subclasses, rows that TMA cannot address: the module's own result."""
    from colossalai_b200.ops import linear as L

    lin = nn.Linear(64, 32, bias=False, device="cuda", dtype=torch.bfloat16)
    x = torch.randn(4, 64, device="cuda").bfloat16()
    assert not L._native(lin, x, None)                                       # gradients on
    with torch.no_grad():
        assert L._native(lin, x, None) and L._native(lin, x, torch.zeros(4, 32, device="cuda", dtype=torch.bfloat16))
        assert not L._native(lin, x, torch.zeros(4, 32, device="cuda"))
        assert not L._native(nn.Linear(64, 32, device="cuda", dtype=torch.bfloat16), x, None)
        assert not L._native(lin, x.float(), None) and not L._native(lin, x[None], None) and not L._native(lin, x[:0], None)
        assert not L._native(lin, torch.randn(33, 64, device="cuda").bfloat16(), None)
        assert not L._native(lin, torch.randn(4, 65, device="cuda").bfloat16()[:, 1:], None)
        assert not L._native(lin, torch.randn(64, 4, device="cuda").bfloat16().t(), None)
        with torch.autocast("cuda", dtype=torch.float16):
            assert not L._native(lin, x, None)
        seen = []
        hook = lin.register_forward_hook(lambda m, a, o: seen.append(o))
        y = L.linear_rows(lin, x, torch.ones(4, 32, device="cuda", dtype=torch.bfloat16))
        hook.remove()
        assert len(seen) == 1 and torch.equal(y, seen[0] + 1)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,H", [(torch.bfloat16, 8), (torch.float16, 264), (torch.float32, 4100), (torch.bfloat16, 12)])
def test_embed_rows(dtype, H):
    from colossalai_b200 import ops

    emb = nn.Embedding(50, H, device="cuda", dtype=dtype)
    ids = torch.tensor([0, 49, 7, 7, 3], device="cuda")
    with torch.no_grad():
        assert torch.equal(ops.embed_rows(emb, ids), emb.weight[ids])
    assert ops.embed_rows(emb, ids).requires_grad


def test_on_the_cpu_the_module_is_called():
    from colossalai_b200 import ops

    lin, emb = nn.Linear(8, 4), nn.Embedding(5, 8)
    ids = torch.tensor([4, 0])
    with torch.no_grad():
        x = ops.embed_rows(emb, ids)
        assert torch.equal(x, emb(ids)) and torch.equal(ops.linear_rows(lin, x, x[:, :4]), x[:, :4] + lin(x))


def test_graph_inputs_of_one_type_are_copied_together():
    """Copies of alike tensors go together, other types and layouts one by one: the static inputs end up equal."""
    from colossalai_b200.inference.graph_runner import CUDAGraphRunner

    r = CUDAGraphRunner(None)
    r.static_inputs = {"a": torch.zeros(3), "b": torch.zeros(2, 2), "c": torch.zeros(4, dtype=torch.int64), "d": torch.zeros(2, 3)}
    r.graph = type("G", (), {"replay": lambda self: None})()
    new = {"a": torch.randn(3), "b": torch.randn(1, 2).expand(2, 2), "c": torch.arange(4, dtype=torch.int32), "d": torch.randn(3, 2).t()}
    r(**new)
    for k, v in new.items():
        assert torch.equal(r.static_inputs[k], v.to(r.static_inputs[k].dtype))


def _replaced():
    """Modules whose call is not what their class came with, on the instance and on the class."""
    from types import MethodType

    from colossalai_b200.quantization.fp8_hook import convert_linear_to_fp8

    lin, emb = nn.Linear(16, 16, bias=False), nn.Embedding(5, 16)
    lin.forward = MethodType(lambda self, x: x + 1, lin)
    emb.forward = MethodType(lambda self, ids: ids + 1, emb)
    fp8 = nn.Linear(16, 16, bias=False)
    convert_linear_to_fp8(fp8)
    compiled = nn.Linear(16, 16, bias=False)
    compiled._compiled_call_impl = lambda x: x + 1
    return [(lin, nn.Linear), (emb, nn.Embedding), (fp8, nn.Linear), (compiled, nn.Linear)]


def test_a_replaced_forward_is_seen(monkeypatch):
    from colossalai_b200.ops import linear as L

    lin, emb = nn.Linear(16, 16, bias=False), nn.Embedding(5, 16)
    assert L.unwatched(lin, L._LINEAR) and L.unwatched(emb, L._EMBEDDING)
    for m, kind in _replaced():
        assert not L.unwatched(m, L._LINEAR if kind is nn.Linear else L._EMBEDDING)
    monkeypatch.setattr(nn.Linear, "forward", lambda self, x: x + 1)
    assert not L.unwatched(lin, L._LINEAR)


@pytest.mark.parametrize("where", ["instance", "class"])
def test_a_replaced_feed_forward_gets_one_argument(where, monkeypatch):
    from colossalai_b200.models.config import ModelConfig
    from colossalai_b200.models.transformer import MLP, TransformerLMHeadModel

    cfg = ModelConfig(vocab_size=32, hidden_size=32, intermediate_size=64, num_hidden_layers=1, num_attention_heads=2,
                      num_key_value_heads=2)
    model = TransformerLMHeadModel(cfg)
    mlp = next(m for m in model.modules() if isinstance(m, MLP))
    if where == "instance":
        mlp.forward = lambda x: torch.zeros_like(x)
    else:
        monkeypatch.setattr(MLP, "forward", lambda self, x: torch.zeros_like(x))
    ids = torch.arange(6)[None]
    want = model(ids)["logits"]
    with torch.no_grad():
        assert torch.equal(model(ids)["logits"], want)


@pytest.mark.gpu
def test_a_replaced_forward_is_called():
    from colossalai_b200 import ops
    from colossalai_b200.kernel import launch_counter

    x, ids = torch.randn(4, 16, device="cuda").bfloat16(), torch.tensor([4, 0], device="cuda")
    before = {k: launch_counter.by_name.get(k, 0) for k in ("gemm_rows", "embed_rows")}
    for m, kind in _replaced():
        m = m.to("cuda", torch.bfloat16)
        a = x if kind is nn.Linear else ids
        with torch.no_grad():
            got = ops.linear_rows(m, a) if kind is nn.Linear else ops.embed_rows(m, a)
            assert torch.equal(got, m(a))
    assert before == {k: launch_counter.by_name.get(k, 0) for k in before}


@pytest.mark.parametrize("what", ["linear", "embedding"])
def test_watched_calls_are_not_asked_for_pointers(what):
    """Under vmap and fake tensors there is none to be had: the module is called."""
    import warnings

    from torch._subclasses.fake_tensor import FakeTensorMode

    from colossalai_b200 import ops

    with FakeTensorMode(), torch.no_grad(), warnings.catch_warnings():
        warnings.simplefilter("error")
        if what == "linear":
            m, f, one = nn.Linear(64, 32, bias=False, device="cuda", dtype=torch.bfloat16), ops.linear_rows, (4, 64)
            x = torch.empty(3, *one, device="cuda", dtype=torch.bfloat16)
        else:
            m, f, one = nn.Embedding(50, 32, device="cuda", dtype=torch.bfloat16), ops.embed_rows, (4,)
            x = torch.zeros(3, *one, device="cuda", dtype=torch.int64)
        assert f(m, x[0]).shape == (4, 32)
        assert torch.func.vmap(lambda a: f(m, a))(x).shape == (3, 4, 32)


@pytest.mark.gpu
def test_vmap_calls_the_module():
    from colossalai_b200 import ops

    lin, emb = nn.Linear(64, 32, bias=False, device="cuda", dtype=torch.bfloat16), nn.Embedding(50, 32, device="cuda", dtype=torch.bfloat16)
    x, ids = torch.randn(3, 4, 64, device="cuda").bfloat16(), torch.randint(0, 50, (3, 4), device="cuda")
    with torch.no_grad():
        assert torch.equal(torch.func.vmap(lambda a: ops.linear_rows(lin, a))(x), torch.func.vmap(lin)(x))
        assert torch.equal(torch.func.vmap(lambda a: ops.embed_rows(emb, a))(ids), emb(ids))


@pytest.mark.parametrize("id_,entries,refused", [(0, 1, False), (49, 50, False), (2**40, 2**41, False), (-1, 50, True), (50, 50, True),
                                                 (2**32, 50, True), (0, 0, True)])
def test_an_id_outside_the_table_is_refused(id_, entries, refused, tmp_path):
    """The rule that the lookup kernel applies to every id, run on the host: it ends the program, as torch's own lookup does."""
    import subprocess

    from colossalai_b200.kernel.loader import CSRC

    assert "cb_checked_id(ids[blockIdx.x], entries)" in (CSRC / "gemm_rows_tcgen05.cu").read_text()
    src, exe = tmp_path / "id.cpp", tmp_path / "id"
    src.write_text('#include "checked_id.h"\n#include <stdlib.h>\n'
                   "int main(int, char** a) { return cb_checked_id(atoll(a[1]), atoll(a[2])) == atoll(a[1]) ? 0 : 1; }\n")
    subprocess.run(["g++", "-O2", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe), str(id_), str(entries)], capture_output=True, text=True)
    assert r.returncode == (-6 if refused else 0) and ("outside the table" in r.stderr) == refused
