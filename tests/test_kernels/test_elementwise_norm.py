"""Numerics of the sm_100a norm / activation / rope / CE kernels against plain PyTorch fp32 references."""
import math

import pytest
import torch

from colossalai_b200 import ops
from colossalai_b200.ops import cross_entropy as ce

pytestmark = pytest.mark.gpu

DTYPES = [torch.bfloat16, torch.float16, torch.float32]


def _tol(dtype):
    return dict(atol=3e-2, rtol=3e-2) if dtype != torch.float32 else dict(atol=1e-4, rtol=1e-3)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("shape", [(37, 1024), (512, 4096), (8, 8192), (5, 16384)])
@pytest.mark.parametrize("with_res", [False, True])
def test_rmsnorm_fwd_bwd(dtype, shape, with_res):
    torch.manual_seed(0)
    x = torch.randn(*shape, device="cuda", dtype=dtype, requires_grad=True)
    w = (1 + 0.1 * torch.randn(shape[1], device="cuda")).to(dtype).requires_grad_(True)
    res = torch.randn(*shape, device="cuda", dtype=dtype, requires_grad=True) if with_res else None
    xr, wr = x.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
    rr = res.detach().float().requires_grad_(True) if with_res else None
    out = ops.rms_norm(x, w, 1e-5, res)
    ref = ops.rms_norm_ref(xr, wr, 1e-5, rr)
    if with_res:
        y, h = out
        yr, hr = ref
        g1, g2 = torch.randn_like(yr), torch.randn_like(hr)
        (y.float() * g1).sum().backward(retain_graph=True)
        (h.float() * g2).sum().backward()
        ((yr * g1).sum() + (hr * g2).sum()).backward()
        torch.testing.assert_close(h.float(), hr, **_tol(dtype))
        torch.testing.assert_close(res.grad.float(), rr.grad, **_tol(dtype))
    else:
        y, yr = out, ref
        g1 = torch.randn_like(yr)
        (y.float() * g1).sum().backward()
        (yr * g1).sum().backward()
    torch.testing.assert_close(y.float(), yr, **_tol(dtype))
    torch.testing.assert_close(x.grad.float(), xr.grad, **_tol(dtype))
    wt = dict(atol=0.5, rtol=5e-2) if dtype != torch.float32 else dict(atol=1e-3, rtol=1e-3)
    torch.testing.assert_close(w.grad.float(), wr.grad, **wt)


@pytest.mark.parametrize("norm", ["rms", "layer", "layer_bias"])
def test_norm_of_no_rows(norm):
    """The gradients of the parameters are zero, not what the allocator's memory held."""
    ps = [torch.ones(1024, device="cuda", requires_grad=True) for _ in range(2 if norm == "layer_bias" else 1)]
    x = torch.zeros(0, 1024, device="cuda", requires_grad=True)
    y = ops.rms_norm(x, ps[0]) if norm == "rms" else ops.layer_norm(x, *ps)
    held = [torch.full((1024,), 7.0, device="cuda") for _ in range(8)]
    del held
    grads = torch.autograd.grad(y, [x] + ps, torch.zeros_like(y))
    assert grads[0].shape == (0, 1024) and not any(g.any() for g in grads[1:])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("bias", [True, False])
def test_layernorm_fwd_bwd(dtype, bias):
    torch.manual_seed(0)
    x = torch.randn(300, 2048, device="cuda", dtype=dtype, requires_grad=True)
    w = (1 + 0.1 * torch.randn(2048, device="cuda")).to(dtype).requires_grad_(True)
    b = (0.1 * torch.randn(2048, device="cuda")).to(dtype).requires_grad_(True) if bias else None
    xr, wr = x.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
    br = b.detach().float().requires_grad_(True) if bias else None
    y = ops.layer_norm(x, w, b, 1e-5)
    yr = torch.nn.functional.layer_norm(xr, (2048,), wr, br, 1e-5)
    g = torch.randn_like(yr)
    (y.float() * g).sum().backward()
    (yr * g).sum().backward()
    torch.testing.assert_close(y.float(), yr, **_tol(dtype))
    torch.testing.assert_close(x.grad.float(), xr.grad, **_tol(dtype))
    wt = dict(atol=0.5, rtol=5e-2) if dtype != torch.float32 else dict(atol=1e-3, rtol=1e-3)
    torch.testing.assert_close(w.grad.float(), wr.grad, **wt)
    if bias:
        torch.testing.assert_close(b.grad.float(), br.grad, **wt)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("act", ["silu", "gelu_tanh", "gelu"])
def test_glu_fwd_bwd(dtype, act):
    torch.manual_seed(0)
    gu = torch.randn(333, 2 * 1792, device="cuda", dtype=dtype, requires_grad=True)
    gr = gu.detach().float().requires_grad_(True)
    y = ops.glu(gu, act)
    yr = ops.glu_ref(gr, act)
    g = torch.randn_like(yr)
    (y.float() * g).sum().backward()
    (yr * g).sum().backward()
    torch.testing.assert_close(y.float(), yr, **_tol(dtype))
    torch.testing.assert_close(gu.grad.float(), gr.grad, **_tol(dtype))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_bias_act(dtype):
    x = torch.randn(100, 512, device="cuda", dtype=dtype, requires_grad=True)
    b = torch.randn(512, device="cuda", dtype=dtype, requires_grad=True)
    xr, br = x.detach().float().requires_grad_(True), b.detach().float().requires_grad_(True)
    y = ops.bias_act(x, b, "gelu")
    yr = torch.nn.functional.gelu(xr + br)
    y.float().sum().backward()
    yr.sum().backward()
    torch.testing.assert_close(y.float(), yr, **_tol(dtype))
    torch.testing.assert_close(x.grad.float(), xr.grad, **_tol(dtype))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("interleaved,rot", [(False, 128), (False, 64), (True, 64)])
def test_rope_qkv(dtype, interleaved, rot):
    torch.manual_seed(0)
    T, hq, hkv, D = 200, 8, 2, 128
    qkv = torch.randn(T, (hq + 2 * hkv) * D, device="cuda", dtype=dtype, requires_grad=True)
    pos = torch.randint(0, 4096, (T,), device="cuda")
    cos, sin = ops.build_rope_cache(4096, rot, 10000.0, device="cuda")
    out = ops.rope_qkv(qkv, pos, cos, sin, hq, hkv, D, rot_dim=rot, interleaved=interleaved)
    qr = qkv.detach().float().requires_grad_(True)
    x = qr.view(T, hq + 2 * hkv, D)
    ref = torch.cat([ops.rope_ref(x[:, : hq + hkv], pos, cos, sin, rot, interleaved), x[:, hq + hkv:]], 1).reshape(T, -1)
    g = torch.randn_like(ref)
    (out.float() * g).sum().backward()
    (ref * g).sum().backward()
    torch.testing.assert_close(out.float(), ref, **_tol(dtype))
    torch.testing.assert_close(qkv.grad.float(), qr.grad, **_tol(dtype))


@pytest.mark.parametrize("layout", ["packed", "strided", "odd_offset", "expanded_grad"])
@pytest.mark.parametrize("T,hq,hkv,D,rot,interleaved", [(1, 1, 1, 16, 16, False), (3, 5, 1, 24, 16, True),
                                                        (2, 33, 3, 96, 64, False), (5, 64, 8, 128, 128, False)])
def test_rope_row_layouts(layout, T, hq, hkv, D, rot, interleaved):
    """The rows the one-pass kernel reads where they lie and those it packs first, with an odd number of pass-through
    vectors and more items than a block has threads: both directions equal the reference's rounding of fp32 values."""
    torch.manual_seed(1)
    W = (hq + 2 * hkv) * D
    base = torch.randn(T * (W + 16) + 8, device="cuda").bfloat16()
    x = {"strided": base[: T * (W + 16)].view(T, W + 16)[:, 8: 8 + W], "odd_offset": base[3: 3 + T * W].view(T, W)}.get(
        layout, base[: T * W].view(T, W))
    x = x.detach().requires_grad_(True)
    pos = torch.randint(0, 64, (T,), device="cuda")
    cos, sin = ops.build_rope_cache(64, rot, 10000.0, device="cuda")
    out = ops.rope_qkv(x, pos, cos, sin, hq, hkv, D, rot_dim=rot, interleaved=interleaved)
    g = torch.randn(1, 1, device="cuda").bfloat16().expand(T, W) if layout == "expanded_grad" else torch.randn(T, W, device="cuda").bfloat16()
    out.backward(g)

    def turned(z, sign):
        z = z.detach().reshape(T, -1, D)
        return torch.cat([ops.rope_ref(z[:, : hq + hkv], pos, cos, sin * sign, rot, interleaved), z[:, hq + hkv:]], 1).reshape(T, -1)

    # two roundings of the same fp32 value (contracted or not) differ by one step of 2^-8 at most
    torch.testing.assert_close(out, turned(x, 1), rtol=2 ** -7, atol=1e-6)
    torch.testing.assert_close(x.grad, turned(g, -1), rtol=2 ** -7, atol=1e-6)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("V,valid,start", [(32000, 32000, 0), (16064, 16000, 16064), (4096, 4096, 8192)])
def test_cross_entropy_blocks(dtype, V, valid, start):
    torch.manual_seed(0)
    T = 257
    logits = (3 * torch.randn(T, V, device="cuda")).to(dtype)
    target = torch.randint(start, start + valid, (T,), device="cuda")
    target[::7] = -100
    target[1::11] = 3   # owned by another rank (unless start == 0)
    with ops.force_torch():
        m_ref = ce.row_max(logits, valid)
        s_ref = ce.sumexp_and_target(logits, target, m_ref, start, -100, valid)
        scale = torch.rand(T, device="cuda")
        g_ref = ce.softmax_grad(logits, target, m_ref, s_ref[0], None, start, -100, row_scale=scale, valid_cols=valid)
    m = ce.row_max(logits, valid)
    s = ce.sumexp_and_target(logits, target, m, start, -100, valid)
    g = ce.softmax_grad(logits, target, m, s[0], None, start, -100, row_scale=scale, valid_cols=valid)
    torch.testing.assert_close(m, m_ref)
    torch.testing.assert_close(s, s_ref, atol=1e-3, rtol=1e-4)
    torch.testing.assert_close(g.float(), g_ref.float(), atol=2e-3 if dtype != torch.float32 else 1e-6, rtol=2e-2)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("V,valid", [(8, 8), (16384, 16384), (16392, 16385), (50304, 50257), (4096, 1), (4096, 0)])
def test_cross_entropy_one_pass_stats(dtype, V, valid):
    """Row maximum and sum in one pass at the ends of a thread's share, with rows of the type's lowest value, of -inf in
    front, of one finite entry, and sorted rows whose running maximum moves at every vector."""
    torch.manual_seed(V)
    x = 3 * torch.randn(9, V, device="cuda")
    x[1] = torch.finfo(dtype).min
    x[2] = float("-inf")
    x[2, -1] = x[2, max(valid - 1, 0)] = 1.0
    x[3] = torch.linspace(-40, 40, V, device="cuda")
    x[4] = torch.linspace(40, -40, V, device="cuda")
    x[5] = float("-inf")
    x[6, V // 2] = float("nan")
    x = x.to(dtype)
    t = torch.full((9,), 5, device="cuda")
    t[7], t[8] = -100, 5 + V
    m, s, tl = ce.row_stats(x, t, 5, -100, valid)
    x64 = x[:, :valid].double()
    if valid == 0:
        assert torch.isneginf(m).all() and not s.any() and not tl.any()
        return
    rows = [r for r in range(9) if r not in (5, 6)]
    assert torch.equal(m[rows].double(), x64.max(-1).values[rows])
    # approximate exponentials of 2^-21 each and fp32 sums of at most V / 512 + 40 terms in a row
    ref = (x64 - x64.max(-1, keepdim=True).values).exp().sum(-1)
    assert ((s.double() - ref).abs() <= 2e-5 * ref)[rows].all()
    assert torch.isneginf(m[5]) and s[5] == 0 and (valid <= V // 2 or torch.isnan(s[6]))
    assert torch.equal(tl[rows[:5]], x[rows[:5], 0].float()) and tl[7] == 0 and tl[8] == 0


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("vecs", [1, 31, 33, 127, 128, 129, 385, 1000, 2047, 2048, 2049])
@pytest.mark.parametrize("short", [0, 1])
def test_cross_entropy_stats_by_width(dtype, vecs, short):
    """Every block size that a row's width asks for, with and without a last column that does not count."""
    g = torch.Generator(device="cuda").manual_seed(vecs)
    V = vecs * (4 if dtype == torch.float32 else 8)
    x = (3 * torch.randn(5, V, device="cuda", generator=g)).to(dtype)
    x[:, -1] = 30.0
    t = torch.randint(0, V - short, (5,), device="cuda", generator=g)
    m, s, tl = ce.row_stats(x, t, 0, -100, V - short)
    x64 = x[:, : V - short].double()
    assert torch.equal(m.double(), x64.max(-1).values) and torch.equal(tl, x[torch.arange(5), t].float())
    ref = (x64 - x64.max(-1, keepdim=True).values).exp().sum(-1)
    assert ((s.double() - ref).abs() <= 2e-5 * ref).all()        # approximate exponentials of 2^-21 each, fp32 sums


@pytest.mark.parametrize("mean", [True, False])
@pytest.mark.parametrize("rows", [0, 1, 31, 1025, 2 ** 24 + 77])
def test_cross_entropy_counts_labels(rows, mean):
    """The number of labels is a whole number, also past 2^24."""
    stats = torch.zeros(3, rows, device="cuda")
    stats[1] = 2.0
    t = torch.zeros(rows, dtype=torch.int64, device="cuda")
    t[: rows // 1000] = -100
    n = rows - rows // 1000
    loss, n_valid = ce.loss_from_stats(stats, t, -100, mean)
    assert int(n_valid) == n
    want = (n / max(n, 1) if mean else n) * math.log(2.0)
    assert abs(float(loss) - want) <= 2.0 ** -23 * want                       # summed in 64 bits, rounded once


@pytest.mark.parametrize("mean", [True, False])
@pytest.mark.parametrize("rows", [2049, 4096, 4097, 5000, 8 * 1024, 128 * 1024 + 1, 300000])
def test_cross_entropy_loss_of_many_rows(rows, mean):
    """One block and several: the sum over the rows in 64 bits, rounded once, the same whenever it is taken."""
    g = torch.Generator(device="cuda").manual_seed(rows)
    stats = torch.rand(3, rows, device="cuda", generator=g) + 0.5
    t = torch.randint(-1, 3, (rows,), device="cuda", generator=g)
    loss, n = ce.loss_from_stats(stats, t, -1, mean)
    ok = t != -1
    assert int(n) == int(ok.sum())
    s = stats.double()
    terms = (s[1].log() + s[0] - s[2])[ok]
    want = terms.sum() / (int(n) if mean else 1)
    # one rounding of the result, and 64-bit sums of at most 300000 terms in another order
    assert abs(float(loss) - float(want)) <= 2.0 ** -24 * abs(float(want)) + 1e-11 * float(terms.abs().sum()) / (int(n) if mean else 1)
    assert torch.equal(loss, ce.loss_from_stats(stats, t, -1, mean)[0])


def test_dist_cross_entropy_matches_torch():
    from colossalai_b200.shardformer.layer.loss import cross_entropy_1d

    torch.manual_seed(0)
    logits = torch.randn(512, 32000, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    tgt = torch.randint(0, 32000, (512,), device="cuda")
    tgt[:17] = -100
    lr = logits.detach().float().requires_grad_(True)
    loss = cross_entropy_1d(logits, tgt, process_group="local", vocab_size=32000)
    ref = torch.nn.functional.cross_entropy(lr, tgt, ignore_index=-100)
    loss.backward()
    ref.backward()
    torch.testing.assert_close(loss, ref, atol=2e-3, rtol=1e-3)
    torch.testing.assert_close(logits.grad.float(), lr.grad, atol=1e-5, rtol=5e-2)


@pytest.mark.parametrize("I", [8, 24, 1408, 4096, 4104, 14336])
@pytest.mark.parametrize("act", ["silu", "gelu"])
def test_glu_row_parts(I, act):
    """Rows narrower than a block, of one part exactly, of one vector more, of several: forward and both gradients."""
    torch.manual_seed(I)
    x = torch.randn(3, 2 * I, device="cuda").bfloat16().requires_grad_(True)
    xr = x.detach().float().requires_grad_(True)
    a, b = xr.chunk(2, -1)
    ref = (torch.nn.functional.silu(a) if act == "silu" else torch.nn.functional.gelu(a)) * b
    y, g = ops.glu(x, act), torch.randn(3, I, device="cuda").bfloat16()
    y.backward(g)
    ref.backward(g.float())
    torch.testing.assert_close(y.float(), ref, rtol=2 ** -7, atol=1e-5)      # one rounding to bf16, fast exponentials
    torch.testing.assert_close(x.grad.float(), xr.grad, rtol=2 ** -7, atol=1e-5)


def test_glu_row_limit():
    """`valid_rows`: rows past the device-side limit are neither read nor written, forward and backward."""
    import torch

    from colossalai_b200 import ops

    torch.manual_seed(0)
    x = torch.randn(512, 2 * 256, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    n = torch.tensor(300, device="cuda")
    y = ops.glu(x, "silu", valid_rows=n)
    ref = ops.glu(x.detach()[:300], "silu")
    torch.testing.assert_close(y[:300], ref, atol=0, rtol=0)
    dy = torch.randn(512, 256, device="cuda", dtype=torch.bfloat16)
    (g,) = torch.autograd.grad(y, x, dy)
    xr = x.detach()[:300].clone().requires_grad_(True)
    (gr,) = torch.autograd.grad(ops.glu(xr, "silu"), xr, dy[:300])
    torch.testing.assert_close(g[:300], gr, atol=0, rtol=0)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("heads,kv,D,rot,interleaved", [(1, 1, 16, 16, False), (2, 1, 32, 16, True), (1, 0, 16, 16, False), (12, 5, 32, 32, False),
                                                       (16, 0, 32, 32, False), (32, 0, 32, 32, False), (33, 0, 32, 32, False)])
@pytest.mark.parametrize("T", [1, 7, 1000])
def test_rope_of_narrow_rows(dtype, heads, kv, D, rot, interleaved, T):
    """Rows of which several share a block, up to and past the widest of them, with a last block that is not full."""
    torch.manual_seed(T)
    width = (heads + 2 * kv) * D
    x = torch.randn(T, width, device="cuda").to(dtype).requires_grad_()
    pos = torch.randint(0, 50, (T,), device="cuda")
    cos, sin = ops.build_rope_cache(50, rot, 1e4, device="cuda")
    y = ops.rope_qkv(x, pos, cos, sin, heads, kv, D, rot_dim=rot, interleaved=interleaved)
    g = torch.randn_like(y)
    dx, = torch.autograd.grad(y, x, g)

    def turn(z, sign):
        z = z.double().view(T, -1, D)
        c, s = cos[pos].double()[:, None], sign * sin[pos].double()[:, None]
        h = z[:, : heads + kv]
        a, b = (h[..., 0:rot:2], h[..., 1:rot:2]) if interleaved else (h[..., : rot // 2], h[..., rot // 2: rot])
        u, w = a * c - b * s, b * c + a * s
        r = torch.stack([u, w], -1).flatten(-2) if interleaved else torch.cat([u, w], -1)
        return torch.cat([torch.cat([r, h[..., rot:]], -1), z[:, heads + kv:]], 1).flatten(1)

    eps = torch.finfo(dtype).eps
    for got, src, sign in ((y, x, 1), (dx, g, -1)):
        # two products of at most the largest entry each, rounded to fp32, and one rounding to the type
        assert (got.double() - turn(src.detach(), sign)).abs().max() <= (0.51 * eps + 3 * 2.0 ** -24) * 1.5 * src.detach().abs().max()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("vecs", [1, 2, 3, 33, 64, 127, 128, 129])
@pytest.mark.parametrize("rows,limit", [(1, None), (300, None), (300, 257)])
def test_glu_of_narrow_rows(dtype, vecs, rows, limit):
    """Rows of which several share a block, up to and past the widest of them; a last block that is not full; only the first
    rows live."""
    torch.manual_seed(vecs)
    I = vecs * (4 if dtype == torch.float32 else 8)
    gu = torch.randn(rows, 2 * I, device="cuda").to(dtype).requires_grad_()
    g = torch.randn(rows, I, device="cuda").to(dtype)
    valid = None if limit is None else torch.tensor([limit], device="cuda")
    y = ops.glu(gu, "silu", valid_rows=valid)
    dgu, = torch.autograd.grad(y, gu, g)
    n = limit or rows
    ref = gu.detach().double()[:n].requires_grad_()
    a, b = ref.chunk(2, -1)
    want = torch.nn.functional.silu(a) * b
    dwant, = torch.autograd.grad(want, ref, g.double()[:n])
    eps = max(torch.finfo(dtype).eps, 1e-5)                 # 32 bits: an approximate exponential and division
    assert (y[:n].double() - want).abs().le(eps * want.abs() + 1e-6).all()
    assert (dgu[:n].double() - dwant).abs().le(eps * dwant.abs() + 2e-5).all()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("hq,hkv,D,rot,interleaved", [(32, 8, 128, 128, False), (33, 3, 96, 64, False), (7, 1, 128, 64, True), (64, 8, 256, 64, False)])
@pytest.mark.parametrize("per_sm", [5, 30])
def test_rope_of_many_rows(dtype, hq, hkv, D, rot, interleaved, per_sm):
    """A thread's several items in calls of many tokens: the bits of the same rows a few at a time, with items that are no multiple of what
    a thread or a block takes."""
    T = per_sm * torch.cuda.get_device_properties(0).multi_processor_count
    g = torch.Generator(device="cuda").manual_seed(hq)
    x = torch.randn(T, (hq + 2 * hkv) * D, device="cuda", generator=g).to(dtype)
    pos = torch.randint(0, 64, (T,), device="cuda", generator=g)
    cos, sin = ops.build_rope_cache(64, rot, 10000.0, device="cuda")
    f = lambda z, p: ops.rope_qkv(z, p, cos, sin, hq, hkv, D, rot_dim=rot, interleaved=interleaved)      # noqa: E731
    assert torch.equal(f(x, pos), torch.cat([f(a, b) for a, b in zip(x.split(100), pos.split(100))]))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("H", [64, 4096, 8200])
@pytest.mark.parametrize("odd", [0, 1])
@pytest.mark.parametrize("with_res", [False, True])
@pytest.mark.parametrize("per_sm", [8, 17])
def test_rmsnorm_of_many_rows(dtype, H, odd, with_res, per_sm):
    """Two rows a block in calls of many rows, the last block's second one missing: the bits of the same rows a few at a time."""
    rows = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + 2 + odd
    g = torch.Generator(device="cuda").manual_seed(H)
    x, r = (torch.randn(rows, H, device="cuda", generator=g).to(dtype) for _ in "xr")
    w = torch.randn(H, device="cuda", generator=g).to(dtype)
    f = lambda a, b: ops.rms_norm(a, w, 1e-5, b) if with_res else (ops.rms_norm(a, w, 1e-5),)      # noqa: E731
    few = [f(a, b) for a, b in zip(x.split(500), r.split(500))]
    for i, y in enumerate(f(x, r)):
        assert torch.equal(y, torch.cat([p[i] for p in few]))
