"""Kernels that take their place while the one before them runs wait for what it writes."""
import pytest
import torch

pytestmark = pytest.mark.gpu
R, W = 148, 4096


class Step:
    """What the kernels read and write besides the rows that come from the kernel before them."""

    def __init__(self):
        from colossalai_b200.ops import build_rope_cache

        g = torch.Generator(device="cuda").manual_seed(3)
        rand = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
        self.w, self.res, self.down = rand(W), rand(R, W), torch.nn.Linear(W, 256, bias=False, device="cuda", dtype=torch.bfloat16)
        self.pos = torch.arange(R, device="cuda")
        self.cos, self.sin = (t.cuda() for t in build_rope_cache(R, 128))
        self.kc, self.vc = rand(64, 16, 8, 128), rand(64, 16, 8, 128)
        self.written = torch.zeros_like(self.kc), torch.zeros_like(self.vc)
        self.tables = torch.arange(64, device="cuda", dtype=torch.int32).view(2, 32)
        self.seq, self.at = torch.zeros(R, device="cuda", dtype=torch.int32), torch.arange(R, device="cuda", dtype=torch.int32)
        self.lens = torch.tensor([512, 300], device="cuda", dtype=torch.int32)
        self.long = torch.tensor([4097], device="cuda", dtype=torch.int32)
        self.long_table = torch.arange(257, device="cuda", dtype=torch.int32).view(1, 257) % 64
        self.ids = torch.tensor([0, R - 1, 5, 77], device="cuda")

    def norm(self, y):
        from colossalai_b200 import ops
        return ops.rms_norm(y, self.w, 1e-5)

    def norm_residual(self, y):
        from colossalai_b200 import ops
        return ops.rms_norm(self.res, self.w, 1e-5, y)

    def glu(self, y):
        from colossalai_b200 import ops
        return ops.glu(y, "silu")

    def rope(self, y):
        from colossalai_b200 import ops
        return ops.rope_qkv(y, self.pos, self.cos, self.sin, 16, 8, 128)

    def cache_write(self, y):
        from colossalai_b200.ops import inference as iops
        y = y.view(R, 4, 8, 128)
        iops.kv_cache_write(y[:, 0], y[:, 1], *self.written, self.tables, self.seq, self.at)
        return self.written

    def decode(self, y):
        from colossalai_b200.ops import inference as iops
        return iops.paged_decode_attention(y[:2].view(2, 32, 128), self.kc, self.vc, self.tables, self.lens)

    def decode_long(self, y):
        from colossalai_b200.ops import inference as iops
        return iops.paged_decode_attention(y[:1].view(1, 32, 128), self.kc, self.vc, self.long_table, self.long)

    def linear(self, y):
        from colossalai_b200 import ops
        return ops.linear_rows(self.down, y[:32])

    def linear_residual(self, y):
        from colossalai_b200 import ops
        return ops.linear_rows(self.down, self.res[:32], y[:32, :256])

    def embedding(self, y):
        from colossalai_b200 import ops
        emb = torch.nn.Embedding(R, W, device="meta")
        emb.weight = torch.nn.Parameter(y, requires_grad=False)
        return ops.embed_rows(emb, self.ids)


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("name", [n for n in vars(Step) if not n.startswith("_")])
def test_the_rows_of_the_kernel_before_are_complete(name, graph):
    """A projection of 90 us, whose CTAs are all on the chip from its beginning and which writes its rows at its end, over NaN; the
    kernel behind it, launched meanwhile, gives the bits that it gives when everything is done."""
    from colossalai_b200 import ops

    step = Step()
    call = getattr(step, name)
    g = torch.Generator(device="cuda").manual_seed(5)
    first = torch.nn.Linear(14336, R * W // 32, bias=False, device="cuda", dtype=torch.bfloat16)
    x = torch.randn(32, 14336, device="cuda", generator=g).bfloat16()
    with torch.no_grad():
        y = ops.linear_rows(first, x)
        torch.cuda.synchronize()
        want = call(y.view(R, W))
        want = [t.clone() for t in (want if isinstance(want, tuple) else (want,))]
        assert all(torch.isfinite(t).all() for t in want)
        for t in step.written:
            t.zero_()

        def both():
            y = ops.linear_rows(first, x)
            return y, call(y.view(R, W))

        if graph:
            pool = torch.cuda.CUDAGraph()
            with torch.cuda.graph(pool):
                y, got = both()
            y.fill_(float("nan"))
            pool.replay()
        else:
            del y
            torch.cuda.empty_cache()
            y = torch.full((32, R * W // 32), float("nan"), device="cuda", dtype=torch.bfloat16)
            at = y.data_ptr()
            del y
            y, got = both()
            assert y.data_ptr() == at                                           # over the NaN
        for a, b in zip(got if isinstance(got, tuple) else (got,), want):
            assert torch.equal(a, b)
