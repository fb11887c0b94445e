"""tcgen05 grouped (per-expert) GEMM: forward / dgrad with variable rows per expert and wgrad with variable reduction
length, against fp32 per-expert matmuls.  Expert sizes include 0, 1, non-multiples of the tile and of the k-block."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(x, w, counts):
    out = torch.empty(x.shape[0], w.shape[1], dtype=torch.float32, device=x.device)
    s = 0
    for e, n in enumerate(counts.tolist()):
        out[s:s + n] = x[s:s + n].float() @ w[e].float().t()
        s += n
    return out


CASES = [
    ([300, 0, 1, 255, 256, 257, 700, 131], 512, 768),          # ragged groups, an empty one
    ([2048] * 8, 4096, 2816),                                  # balanced, Mixtral-like aspect
    ([5, 9000, 17, 3], 1024, 1408),                            # one dominant expert, output width not a tile multiple
    ([128 * i for i in range(1, 17)], 2048, 2816),             # 16 experts, every size a k-block multiple
]


@pytest.mark.parametrize("counts,K,N", CASES)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_grouped_forward(counts, K, N, dtype):
    from colossalai_b200.moe import grouped_gemm as gg

    torch.manual_seed(0)
    c = torch.tensor(counts, device="cuda")
    rows = int(sum(counts))
    x = (torch.randn(rows, K, device="cuda") * 0.5).to(dtype)
    w = (torch.randn(len(counts), N, K, device="cuda") * 0.05).to(dtype)
    assert gg.native_ok(x, w)
    y = gg.grouped_linear(x, w, c)
    ref = _ref(x, w, c)
    torch.testing.assert_close(y.float(), ref, atol=2e-2 + 2e-3 * K ** 0.5 * 0.05, rtol=1.6e-2)


@pytest.mark.parametrize("counts,K,N", CASES)
@pytest.mark.parametrize("aligned", [False, True])
def test_grouped_backward(counts, K, N, aligned):
    """dX (variable-M NN kernel) and dW (variable-K TN kernel; padded on the device when the layout is not aligned)."""
    from colossalai_b200.moe import grouped_gemm as gg

    if N % 128 != 0:
        pytest.skip("dgrad kernel needs the expert output width to be a multiple of 128")
    if aligned and any(n % 128 for n in counts):
        pytest.skip("layout is not aligned")
    torch.manual_seed(1)
    c = torch.tensor(counts, device="cuda")
    rows = int(sum(counts))
    x = (torch.randn(rows, K, device="cuda") * 0.5).bfloat16().requires_grad_(True)
    w = (torch.randn(len(counts), N, K, device="cuda") * 0.05).bfloat16().requires_grad_(True)
    dy = (torch.randn(rows, N, device="cuda") * 0.1).bfloat16()
    gg.grouped_linear(x, w, c, aligned=aligned).backward(dy)
    xf, wf = x.detach().float().requires_grad_(True), w.detach().float().requires_grad_(True)
    out = torch.empty(rows, N, device="cuda")
    s, parts = 0, []
    for e, n in enumerate(counts):
        parts.append(xf[s:s + n] @ wf[e].t())
        s += n
    torch.cat(parts, 0).backward(dy.float())
    dxe = (x.grad.float() - xf.grad).abs().max().item()
    assert dxe <= 1.6e-2 * xf.grad.abs().max().item() + 1e-3, dxe
    for e, n in enumerate(counts):
        ref = wf.grad[e]
        err = (w.grad[e].float() - ref).abs().max().item()
        assert err <= 1.6e-2 * ref.abs().max().item() + 2e-3 * max(n, 1) ** 0.5 * 0.05 + 1e-3, (e, n, err)


def test_grouped_gemm_counts_stay_on_device():
    """No host synchronisation: the group sizes are only ever read by the kernel."""
    from colossalai_b200.moe import grouped_gemm as gg

    c = torch.tensor([100, 200, 300, 424], device="cuda")
    x = torch.randn(1024, 512, device="cuda", dtype=torch.bfloat16)
    w = torch.randn(4, 256, 512, device="cuda", dtype=torch.bfloat16)
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        torch.cuda.set_sync_debug_mode("error")
        try:
            y = gg.grouped_linear(x, w, c)
        finally:
            torch.cuda.set_sync_debug_mode("default")
    torch.cuda.synchronize()
    torch.testing.assert_close(y.float(), _ref(x, w, c), atol=0.5, rtol=2e-2)


@pytest.mark.parametrize("counts,K,N", [([16, 0, 256, 272, 496, 512, 528, 16], 256, 384), ([48] * 40 + [144], 128, 264), ([4880], 72, 128)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_groups_of_sixteen_rows(counts, K, N, dtype):
    """Groups on and beside the edges of one, two and many row tiles (up to 256 rows, multiples of 16), of a 32- and a 64-row box and of a
    k-block; output widths that end inside a tile.  Rows behind the last group belong to nobody."""
    from colossalai_b200.moe import grouped_gemm as gg

    g = torch.Generator(device="cuda").manual_seed(len(counts))
    c = torch.tensor(counts, device="cuda")
    rows, E = int(sum(counts)), len(counts)
    x, dy = (torch.randn(rows + 40, n, device="cuda", generator=g).to(dtype) for n in (K, N))
    w = (torch.randn(E, N, K, device="cuda", generator=g) * K ** -0.5).to(dtype)
    offs = gg._offs(c, x.device)
    y = gg._native_fwd(x, w, offs, True)
    dw = gg._native_wgrad(dy, x, offs, E, dtype)
    dw32 = gg._native_wgrad(dy, x, offs, E, torch.float32)
    dx = gg._native_fwd(dy, w, offs, False) if N % gg.K_BLOCK == 0 else None
    eps = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)                # half a unit of the results' rounding, and fp32 sums
    s = 0
    for e, n in enumerate(counts):
        xe, de, we = x[s:s + n].double(), dy[s:s + n].double(), w[e].double()
        for got, ref in ((y[s:s + n], xe @ we.t()), (dw[e], de.t() @ xe)) + (((dx[s:s + n], de @ we),) if dx is not None else ()):
            assert ref.numel() == 0 or (got.double() - ref).abs().max() <= eps * ref.abs().max()
        assert (dw32[e].double() - de.t() @ xe).norm() <= 1e-5 * (de.t() @ xe).norm()
        s += n


@pytest.mark.parametrize("act", ["silu", "gelu_tanh", "gelu"])
@pytest.mark.parametrize("counts,H,inter,dtype", [
    ([16, 0, 48, 272, 256], 128, 64, torch.bfloat16),         # half a block of columns, an empty group, a tile and a little more
    ([240, 16, 528], 256, 192, torch.float16),                # a block and a half
    ([0] * 30 + [16] * 34, 512, 1408, torch.bfloat16),        # the smallest groups
    ([4096, 16, 1024, 2000], 1024, 704, torch.bfloat16),
])
def test_gated_experts(counts, H, inter, dtype, act):
    """The unit in the epilogues of the products before and behind it: the bits of one operator after the other, rows behind the last group left
    alone."""
    from colossalai_b200.kernel import loader
    from colossalai_b200.moe import grouped_gemm as gg
    from colossalai_b200.ops import glu

    g = torch.Generator(device="cuda").manual_seed(inter)
    rows, E = sum(counts), len(counts)
    c = torch.tensor(counts, device="cuda")
    c.cb200_aligned = True
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=g)
    ins = [rand(rows + 80, H), rand(E, 2 * inter, H) * H ** -0.5, rand(E, H, inter) * inter ** -0.5]
    ins = [t.to(dtype).requires_grad_(True) for t in ins]
    dy = rand(rows + 80, H).to(dtype)
    out = []
    for fused in (True, False):
        loader.launch_counter.reset()
        if fused:
            y = gg.gated_experts(*ins, c, act)
        else:
            y = gg.grouped_linear(glu(gg.grouped_linear(ins[0], ins[1], c), act, valid_rows=gg.rows_of(c)), ins[2], c)
        dx, d_up, d_down = torch.autograd.grad(y, ins, dy)
        out.append([y[:rows], dx[:rows], d_up, d_down])
        assert any("glu" in name for name in loader.launch_counter.by_name) != fused
    for a, b in zip(*out):
        assert torch.equal(a, b)


@pytest.mark.parametrize("form", ["gated", "linear", "python"])
@pytest.mark.parametrize("frozen", [False, True])
def test_expert_gradients_that_are_differentiated_again(form, frozen, monkeypatch):
    """Gradients under `create_graph` carry a graph: their own gradients against 64 bits, for all inputs or for the rows alone."""
    from colossalai_b200.kernel import loader
    from colossalai_b200.moe import grouped_gemm as gg

    if form == "python":
        loader.host()
        monkeypatch.setattr(loader, "_host", None)
    counts, H, inter = [16, 0, 48, 32], 128, 64
    rows = sum(counts)
    g = torch.Generator(device="cuda").manual_seed(3)
    c = torch.tensor(counts, device="cuda")
    c.cb200_aligned = True
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=g)
    ins = [rand(rows + 16, H), rand(4, 2 * inter, H) * H ** -0.5] + ([rand(4, H, inter) * inter ** -0.5] if form == "gated" else [])
    ins = [t.bfloat16().requires_grad_(i == 0 or not frozen) for i, t in enumerate(ins)]
    dy = rand(rows + 16, H if form == "gated" else 2 * inter).bfloat16().requires_grad_()

    def second(fn, tensors, dy):
        live = [t for t in tensors if t.requires_grad]
        first = torch.autograd.grad(fn(*tensors), live, dy, create_graph=True)
        total = sum((t[:rows] if t.dim() == 2 else t).double().square().sum() for t in first)
        return [t.double() for t in torch.autograd.grad(total, live + [dy], allow_unused=True) if t is not None]

    def exact(x, w_up, w_down=None):
        parts, out = x[:rows].split(counts), []
        for e, part in enumerate(parts):
            h = part @ w_up[e].t()
            if w_down is not None:
                gate, up = h.chunk(2, -1)
                h = (torch.nn.functional.silu(gate) * up) @ w_down[e].t()
            out.append(h)
        return torch.cat(out + [torch.zeros(16, out[0].shape[1], dtype=x.dtype, device=x.device)])

    fn = (lambda *t: gg.gated_experts(*t, c, "silu")) if form == "gated" else (lambda *t: gg.grouped_linear(*t, c))
    got = second(fn, ins, dy)
    wide = [t.detach().double().requires_grad_(t.requires_grad) for t in ins]
    want = second(exact, wide, dy.detach().double().requires_grad_())
    assert len(got) == len(want) >= 1
    for a, b in zip(got, want):                     # 16-bit operands and results throughout: some roundings of 2^-9
        assert (a - b).norm() <= 2e-2 * b.norm()
