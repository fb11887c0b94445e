"""Paged-KV inference kernels vs fp32 PyTorch references (reference: tests/test_infer/test_kernels/cuda/
test_{kv_cache_memcpy,flash_decoding_attention,convert_fp8}.py)."""
import pytest
import torch

from colossalai_b200.ops import inference as iops

pytestmark = pytest.mark.gpu


def _mk_cache(n_seqs, max_len, bs, Hkv, D, dtype, dev):
    max_blocks = (max_len + bs - 1) // bs
    nb = n_seqs * max_blocks + 3
    perm = torch.randperm(nb, device=dev)[: n_seqs * max_blocks].to(torch.int32)
    tables = perm.view(n_seqs, max_blocks).contiguous()
    kc = torch.randn(nb, bs, Hkv, D, device=dev, dtype=dtype)
    vc = torch.randn(nb, bs, Hkv, D, device=dev, dtype=dtype)
    return kc, vc, tables


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Hq,Hkv", [(8, 8), (32, 8), (16, 2)])
@pytest.mark.parametrize("bs", [16, 64])
def test_paged_decode_attention(dtype, D, Hq, Hkv, bs):
    dev = torch.device("cuda")
    torch.manual_seed(0)
    n, max_len = 7, 700
    kc, vc, tables = _mk_cache(n, max_len, bs, Hkv, D, dtype, dev)
    lens = torch.tensor([1, 15, 16, 17, 300, 699, 700], device=dev, dtype=torch.int32)
    q = torch.randn(n, Hq, D, device=dev, dtype=dtype)
    out = iops.paged_decode_attention(q, kc, vc, tables, lens)
    ref = iops.paged_decode_attention_ref(q.float(), kc.float(), vc.float(), tables, lens)
    torch.testing.assert_close(out.float(), ref, atol=2e-2, rtol=2e-2)


def test_paged_decode_long_context_split_kv():
    dev = torch.device("cuda")
    torch.manual_seed(1)
    kc, vc, tables = _mk_cache(2, 8192, 16, 8, 128, torch.bfloat16, dev)
    lens = torch.tensor([8192, 4097], device=dev, dtype=torch.int32)
    q = torch.randn(2, 32, 128, device=dev, dtype=torch.bfloat16)
    out = iops.paged_decode_attention(q, kc, vc, tables, lens)
    ref = iops.paged_decode_attention_ref(q.float(), kc.float(), vc.float(), tables, lens)
    torch.testing.assert_close(out.float(), ref, atol=2e-2, rtol=2e-2)


def test_paged_decode_alibi():
    dev = torch.device("cuda")
    torch.manual_seed(2)
    kc, vc, tables = _mk_cache(3, 256, 16, 8, 128, torch.float16, dev)
    lens = torch.tensor([5, 100, 256], device=dev, dtype=torch.int32)
    q = torch.randn(3, 8, 128, device=dev, dtype=torch.float16)
    slopes = torch.tensor([2 ** (-(i + 1)) for i in range(8)], device=dev, dtype=torch.float32)
    out = iops.paged_decode_attention(q, kc, vc, tables, lens, alibi_slopes=slopes)
    ref = iops.paged_decode_attention_ref(q.float(), kc.float(), vc.float(), tables, lens, alibi_slopes=slopes)
    torch.testing.assert_close(out.float(), ref, atol=2e-2, rtol=2e-2)


# wider grid in the spirit of the reference's flash-decoding test
# (tests/test_infer/test_kernels/cuda/test_flash_decoding_attention.py:59-66: batch x block size x context x group size x
#  head dim x same / mixed context lengths, with and without ALiBi)
@pytest.mark.parametrize("bsz", [1, 7, 32])
@pytest.mark.parametrize("bs", [8, 16, 32])
@pytest.mark.parametrize("max_blocks", [1, 8, 67])
@pytest.mark.parametrize("group", [1, 4, 8])
@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("same_len", [True, False])
def test_paged_decode_grid(bsz, bs, max_blocks, group, D, same_len):
    dev = torch.device("cuda")
    torch.manual_seed(bsz * 131 + bs * 17 + max_blocks + group + D)
    Hkv = 2
    Hq = Hkv * group
    max_len = bs * max_blocks
    kc, vc, tables = _mk_cache(bsz, max_len, bs, Hkv, D, torch.bfloat16, dev)
    lens = torch.full((bsz,), max_len, dtype=torch.int32) if same_len else torch.randint(1, max_len + 1, (bsz,)).int()
    lens = lens.to(dev)
    q = torch.randn(bsz, Hq, D, device=dev, dtype=torch.bfloat16)
    out = iops.paged_decode_attention(q, kc, vc, tables, lens)
    ref = iops.paged_decode_attention_ref(q.float(), kc.float(), vc.float(), tables, lens)
    torch.testing.assert_close(out.float(), ref, atol=2e-2, rtol=2e-2)


@pytest.mark.parametrize("window", [1, 16, 100, 4096])
@pytest.mark.parametrize("alibi", [False, True])
def test_paged_decode_sliding_window(window, alibi):
    """`window_start` inside the split-KV kernel: only the last `window` cached tokens are visible."""
    dev = torch.device("cuda")
    torch.manual_seed(3)
    kc, vc, tables = _mk_cache(5, 3000, 16, 4, 128, torch.bfloat16, dev)
    lens = torch.tensor([1, 15, 100, 1025, 3000], device=dev, dtype=torch.int32)
    q = torch.randn(5, 16, 128, device=dev, dtype=torch.bfloat16)
    slopes = torch.tensor([2 ** (-(i + 1) / 2) for i in range(16)], device=dev, dtype=torch.float32) if alibi else None
    out = iops.paged_decode_attention(q, kc, vc, tables, lens, alibi_slopes=slopes, window=window)
    ref = iops.paged_decode_attention_ref(q.float(), kc.float(), vc.float(), tables, lens, alibi_slopes=slopes,
                                          window=window)
    torch.testing.assert_close(out.float(), ref, atol=2e-2, rtol=2e-2)


@pytest.mark.parametrize("tokens,Hkv,D", [(1, 8, 128), (33, 2, 64), (4096, 8, 128), (515, 4, 256)])
def test_kv_cache_write_vectorised_shapes(tokens, Hkv, D):
    """The 16-byte path of `cb_kv_cache_write` over prefill-sized token counts and strided (fused-QKV view) inputs."""
    dev = torch.device("cuda")
    torch.manual_seed(tokens)
    bs = 16
    n_seqs = max(1, tokens // 100)
    per = (tokens + n_seqs - 1) // n_seqs
    seq = (torch.arange(tokens, device=dev) // per).int()
    pos = (torch.arange(tokens, device=dev) % per).int()
    kc, vc, tables = _mk_cache(n_seqs, per, bs, Hkv, D, torch.bfloat16, dev)
    fused = torch.randn(tokens, 3 * Hkv * D, device=dev, dtype=torch.bfloat16)
    k = fused[:, Hkv * D: 2 * Hkv * D].view(tokens, Hkv, D)          # row stride 3 * Hkv * D
    v = fused[:, 2 * Hkv * D:].view(tokens, Hkv, D)
    kc.zero_(); vc.zero_()
    iops.kv_cache_write(k, v, kc, vc, tables, seq, pos)
    blk = tables[seq.long(), (pos // bs).long()].long()
    torch.testing.assert_close(kc[blk, (pos % bs).long()], k, atol=0, rtol=0)
    torch.testing.assert_close(vc[blk, (pos % bs).long()], v, atol=0, rtol=0)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_kv_cache_write(dtype):
    dev = torch.device("cuda")
    torch.manual_seed(3)
    bs, Hkv, D = 16, 4, 128
    kc, vc, tables = _mk_cache(3, 64, bs, Hkv, D, dtype, dev)
    kc0, vc0 = kc.clone(), vc.clone()
    lens = [5, 33, 64]
    seq = torch.repeat_interleave(torch.arange(3), torch.tensor(lens)).to(dev, torch.int32)
    pos = torch.cat([torch.arange(l) for l in lens]).to(dev, torch.int32)
    T = sum(lens)
    kv = torch.randn(T, 2 * Hkv * D + 7, device=dev, dtype=dtype)   # strided views like a fused qkv output
    k = kv[:, : Hkv * D].view(T, Hkv, D)
    v = kv[:, Hkv * D: 2 * Hkv * D].view(T, Hkv, D)
    iops.kv_cache_write(k, v, kc, vc, tables, seq, pos)
    blk = tables[seq.long(), (pos // bs).long()].long()
    slot = (pos % bs).long()
    kc0[blk, slot] = k
    vc0[blk, slot] = v
    assert torch.equal(kc, kc0) and torch.equal(vc, vc0)


def test_convert_fp8_roundtrip():
    dev = torch.device("cuda")
    x = torch.randn(1000, 130, device=dev, dtype=torch.bfloat16)
    q = iops.convert_fp8(x, True)
    ref = x.to(torch.float8_e5m2)
    assert torch.equal(q, ref.view(torch.uint8))
    back = iops.convert_fp8(q, False, torch.bfloat16)
    assert torch.equal(back, ref.to(torch.bfloat16))


def test_engine_gpu_cuda_graph_matches_eager():
    from colossalai_b200.inference import InferenceConfig, InferenceEngine
    from colossalai_b200.inference.config import GenerationConfig
    from colossalai_b200.kernel import loader
    from colossalai_b200.models import build_model, get_config

    torch.manual_seed(0)
    # head_dim 64 so the decode step runs the native paged kernel (the torch reference path syncs and cannot be captured)
    model = build_model(get_config("llama-tiny", hidden_size=256, intermediate_size=512)).to(torch.bfloat16).cuda().eval()
    loader.launch_counter.reset()
    prompts = [[5, 9, 13, 200, 7], [11, 3], [400, 401, 402, 403, 404, 405, 406, 407, 408, 409]]
    outs = []
    for graph in (False, True):
        cfg = InferenceConfig(max_batch_size=4, max_input_len=32, max_output_len=12, block_size=16, dtype="bf16",
                              use_cuda_graph=graph)
        eng = InferenceEngine(model, None, cfg)
        _, ids = eng.generate(prompts_token_ids=prompts, return_token_ids=True,
                              generation_config=GenerationConfig(max_new_tokens=12))
        outs.append(ids)
    assert outs[0] == outs[1]
    assert loader.launch_counter.by_name.get("paged_decode_attention", 0) > 0


@pytest.mark.parametrize("lens", [[0, 0, 0], [1], [0, 1, 0, 33, 0], [16] * 33, [4097] + [1] * 40, [5000, 3, 0, 2048], list(range(1, 130))])
@pytest.mark.parametrize("Hq,Hkv,D,window", [(4, 4, 64, 0), (10, 2, 128, 0), (48, 6, 64, 40), (3, 1, 128, 1)])
def test_paged_decode_pieces(lens, Hq, Hkv, D, window):
    """The balanced split of all visible tokens over the CTAs: empty sequences (zeros), sequences in one piece and in many,
    shares that span many sequences, more than one round of 32 sequences, head counts that leave a CTA partly filled."""
    dev = torch.device("cuda")
    torch.manual_seed(len(lens))
    kc, vc, tables = _mk_cache(len(lens), max(max(lens), 1) + 5, 16, Hkv, D, torch.bfloat16, dev)
    q = torch.randn(len(lens), Hq, D, device=dev, dtype=torch.bfloat16)
    seq = torch.tensor(lens, device=dev, dtype=torch.int32)
    out = iops.paged_decode_attention(q, kc, vc, tables, seq, window=window or None)
    live = [i for i, n in enumerate(lens) if n]
    assert not out[[i for i, n in enumerate(lens) if not n]].any()
    if live:
        ref = iops.paged_decode_attention_ref(q.float()[live], kc.float(), vc.float(), tables[live], seq[live], window=window or None)
        torch.testing.assert_close(out[live].float(), ref, atol=2e-2, rtol=2e-2)      # weights rounded to bf16


@pytest.mark.parametrize("window", [0, 20, 300])
@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("width", [4, 5])
def test_paged_decode_stops_at_the_page_table(D, window, width):
    """A length beyond what a row of the page table has room for: what the row holds is attended, and neither the next row's pages
    nor what lies behind the table is looked at (the row behind holds pages of NaN)."""
    dev = torch.device("cuda")
    torch.manual_seed(D + window)
    n, bs, Hkv = 3, 16, 2
    kc, vc = (torch.randn(n * width + 1, bs, Hkv, D, device=dev, dtype=torch.bfloat16) for _ in range(2))
    kc[-1] = vc[-1] = float("nan")
    tables = torch.full((n + 1, width), n * width, device=dev, dtype=torch.int32)
    tables[:n] = torch.randperm(n * width, device=dev).view(n, width).int()
    q = torch.randn(n, 8, D, device=dev, dtype=torch.bfloat16)
    lens = torch.tensor([width * bs, 5, width * bs + 11], device=dev, dtype=torch.int32)
    out = iops.paged_decode_attention(q, kc, vc, tables[:n], lens, window=window or None)
    for i, m in enumerate(lens.tolist()):
        first, end = max(0, m - window) if window else 0, min(m, width * bs)
        k, v = (c[tables[i].long()].flatten(0, 1)[first:end].double().repeat_interleave(4, 1) for c in (kc, vc))
        ref = torch.einsum("hk,khd->hd", (torch.einsum("hd,khd->hk", q[i].double(), k) / D ** 0.5).softmax(-1), v)
        torch.testing.assert_close(out[i].double(), ref, atol=2e-2, rtol=2e-2)      # weights rounded to bf16


@pytest.mark.parametrize("length", [16, 2000])
@pytest.mark.parametrize("keys", ["one", "page", "all"])
def test_paged_decode_shows_nan(length, keys):
    """NaN keys give NaN, whether the sequence is finished in one piece or merged from many."""
    dev = torch.device("cuda")
    torch.manual_seed(length)
    kc, vc, tables = _mk_cache(2, length, 16, 2, 128, torch.bfloat16, dev)
    q = torch.randn(2, 8, 128, device=dev, dtype=torch.bfloat16)
    lens = torch.tensor([length, length], device=dev, dtype=torch.int32)
    good = iops.paged_decode_attention(q, kc, vc, tables, lens)
    for p in tables[1].tolist() if keys == "all" else [int(tables[1, -1])]:
        kc[p, 3 if keys == "one" else slice(None)] = float("nan")
    out = iops.paged_decode_attention(q, kc, vc, tables, lens)
    assert out[1].isnan().all() and torch.equal(out[0], good[0])


@pytest.mark.parametrize("n,longest", [(1, 47 * 64), (1, 48 * 64), (1, 129 * 64), (3, 47 * 64 + 1), (6, 5000), (7, 5000)])
@pytest.mark.parametrize("D", [64, 128, 256])
def test_paged_decode_by_number_of_partitions(n, longest, D):
    """Both ways of summing the partitions, on both sides of the line and past one round of the wide one; a sequence that leaves
    most of its partitions empty."""
    dev = torch.device("cuda")
    torch.manual_seed(longest)
    kc, vc, tables = _mk_cache(n, longest, 16, 2, D, torch.bfloat16, dev)
    q = torch.randn(n, 6, D, device=dev, dtype=torch.bfloat16)
    lens = torch.tensor([longest, 70, 0, 1, 999, longest - 1, 64][:n], device=dev, dtype=torch.int32)
    out = iops.paged_decode_attention(q, kc, vc, tables, lens)
    live = [i for i, m in enumerate(lens.tolist()) if m]
    ref = iops.paged_decode_attention_ref(q.float()[live], kc.float(), vc.float(), tables[live], lens[live])
    torch.testing.assert_close(out[live].float(), ref, atol=2e-2, rtol=2e-2)      # weights rounded to bf16
    assert not out[[i for i in range(n) if i not in live]].any()


def test_a_refused_launch_is_reported_once():
    """More partitions than a grid has room for: the runtime refuses the launch before anything runs, the launcher says so, and the
    next launcher of the library does not say it once more."""
    import ctypes

    from colossalai_b200.kernel import loader

    lib = loader.load("cb200_infer")
    t = torch.zeros(8, 128, device="cuda", dtype=torch.bfloat16)
    p, i = loader.ptr(t), torch.zeros(1, device="cuda", dtype=torch.int32)
    rc = lib.cb_paged_decode_attention(p, p, p, loader.ptr(i), loader.ptr(i), p, p, p, 1, 8, 8, 128, 16, 1, 70000, 32,
                                       ctypes.c_float(1.0), loader.ptr(None), ctypes.c_int64(1024), ctypes.c_int64(1024), 2, 0,
                                       loader.stream_ptr())
    assert rc != 0
    c = torch.arange(24.0, device="cuda").view(3, 8)
    o = torch.zeros(2, 1, 8, device="cuda")
    pos = torch.tensor([2], device="cuda", dtype=torch.int32)
    assert lib.cb_gather_cos_sin(loader.ptr(c), loader.ptr(c), loader.ptr(pos), loader.ptr(o[0]), loader.ptr(o[1]), 1, 8,
                                 loader.stream_ptr()) == 0
    assert torch.equal(o[0, 0], c[2]) and torch.equal(o[1, 0], c[2])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Hkv", [9, 12, 16, 31, 32])
@pytest.mark.parametrize("group", [1, 4])
@pytest.mark.parametrize("window", [None, 100])
def test_paged_decode_more_than_eight_kv_heads(dtype, D, Hkv, group, window):
    """CTAs of four warps, the last of them with one to four heads."""
    torch.manual_seed(Hkv * 8 + group)
    n, max_len = 5, 700
    kc, vc, tables = _mk_cache(n, max_len, 16, Hkv, D, dtype, torch.device("cuda"))
    lens = torch.tensor([1, 17, 64, 333, 700], device="cuda", dtype=torch.int32)
    q = torch.randn(n, Hkv * group, D, device="cuda", dtype=dtype)
    out = iops.paged_decode_attention(q, kc, vc, tables, lens, window=window).double()
    ref = iops.paged_decode_attention_ref(q.double(), kc, vc, tables, lens, window=window).double()
    # every head of every sequence: weights rounded to 16 bits (bf16: 2^-9 each), the result once more
    assert ((out - ref).norm(dim=-1) <= 6e-3 * ref.norm(dim=-1)).all()


@pytest.mark.gpu
@pytest.mark.parametrize("heads,kv,D,rot,interleaved", [(32, 8, 128, 128, False), (4, 2, 64, 32, False), (3, 1, 128, 64, True), (2, 2, 16, 16, False),
                                                        (1, 1, 64, 64, True)])
@pytest.mark.parametrize("tokens,page", [(1, 16), (5, 16), (300, 7)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_rotation_with_page_write(heads, kv, D, rot, interleaved, tokens, page, dtype):
    """Rotation and page write in one launch: the bits of both, one after the other, and nothing else in the pages, from rows that are a
    part of wider ones and with several tokens a sequence."""
    from colossalai_b200 import ops
    from colossalai_b200.ops import inference

    g = torch.Generator(device="cuda").manual_seed(tokens)
    width = (heads + 2 * kv) * D
    qkv = torch.randn(tokens, width + 16, device="cuda", generator=g).to(dtype)[:, 8:8 + width]
    seqs, most = (tokens + 1) // 2, 3 * page
    tables = torch.randperm(seqs * 3, device="cuda", generator=g).to(torch.int32).view(seqs, 3)
    seq = (torch.arange(tokens, device="cuda") // 2).to(torch.int32)
    pos = (torch.randint(0, most // 2, (tokens,), device="cuda", generator=g) * 2 + torch.arange(tokens, device="cuda") % 2).clamp(max=most - 1)
    cos, sin = ops.build_rope_cache(most, rot, 1e4, device="cuda")
    pages = [torch.randn(seqs * 3, page, kv, D, device="cuda", generator=g).to(dtype) for _ in "kv"]
    want = ops.rope_qkv(qkv, pos, cos, sin, heads, kv, D, rot_dim=rot, interleaved=interleaved)
    kw, vw = pages[0].clone(), pages[1].clone()
    _, k, v = (t.view(tokens, -1, D) for t in want.split([heads * D, kv * D, kv * D], -1))
    inference.kv_cache_write(k, v, kw, vw, tables, seq, pos.to(torch.int32))
    args = (qkv, pos, cos, sin, heads, kv, D, rot, interleaved, *pages, tables, seq, pos.to(torch.int32))
    with torch.no_grad():
        got = inference.rope_pages(*args)
    assert torch.equal(got, want) and torch.equal(pages[0], kw) and torch.equal(pages[1], vw)
    refused = [(0, qkv.float()), (0, qkv[:, 8:]), (1, None), (1, pos.int()), (9, pages[0].float()), (10, pages[1][:, :, :, : D // 2]), (11, tables.long()),
               (2, cos.half())]
    assert all(inference.rope_pages(*(value if i == at else a for i, a in enumerate(args))) is None for at, value in refused)
    assert torch.equal(pages[0], kw) and torch.equal(pages[1], vw)


def _attention_in_64_bits(q, kc, vc, tables, lens, window=0):
    out = []
    for i, m in enumerate(lens.tolist()):
        first = max(0, m - window) if window else 0
        k, v = (c[tables[i].long()].flatten(0, 1)[first:m].double().repeat_interleave(q.shape[1] // c.shape[2], 1) for c in (kc, vc))
        w = (torch.einsum("hd,khd->hk", q[i].double(), k) * q.shape[2] ** -0.5).softmax(-1)
        out.append(torch.einsum("hk,khd->hd", w, v))
    return torch.stack(out)


@pytest.mark.gpu
@pytest.mark.parametrize("n,Hq,Hkv,D", [(1, 16, 8, 128), (2, 4, 2, 64), (29, 8, 8, 128), (30, 8, 8, 128), (49, 8, 8, 128), (50, 8, 8, 128), (9, 32, 32, 128), (3, 12, 12, 128),
                                        (118, 4, 2, 128), (119, 4, 2, 128), (150, 4, 4, 64), (7, 8, 8, 64), (1, 4, 1, 128), (3, 4, 4, 128)])
@pytest.mark.parametrize("room", [80, 1100, 5000, 20000])
def test_paged_decode_partitions_of_a_length(n, Hq, Hkv, D, room):
    """Sequences cut by their own length and by what a table has room for, on both sides of the rules between them, in tables as wide as the
    longest of uneven lengths: against 64 bits, and a sequence's bits do not depend on how long the others are."""
    dev, page = "cuda", 16
    g = torch.Generator(device=dev).manual_seed(n + room)
    width = (room + page - 1) // page
    lens = torch.randint(1, min(room, 700) + 1, (n,), device=dev, generator=g)
    edges = torch.tensor([room, room // 2, 65, 64, 63, 16, 1, room - 1], device=dev)[:n]
    lens[: len(edges)] = edges.clamp(max=room)
    tables = torch.randint(0, 200, (n, width), device=dev, generator=g).to(torch.int32)
    q = torch.randn(n, Hq, D, device=dev, generator=g).bfloat16()
    kc, vc = (torch.randn(200, page, Hkv, D, device=dev, generator=g).bfloat16() for _ in "kv")
    lens = lens.to(torch.int32)
    out = iops.paged_decode_attention(q, kc, vc, tables, lens)
    ref = _attention_in_64_bits(q, kc, vc, tables, lens)
    # every head of every sequence: weights rounded to 16 bits (2^-9 each), the result once more
    assert ((out.double() - ref).norm(dim=-1) <= 6e-3 * ref.norm(dim=-1)).all()
    other = lens.clone()
    other[1::4] = (lens[1::4] // 2).clamp(min=1)
    other[3::4] = (lens[3::4] * 2 + 5).clamp(max=room)
    assert torch.equal(iops.paged_decode_attention(q, kc, vc, tables, other)[0::2], out[0::2])


@pytest.mark.gpu
@pytest.mark.parametrize("n,Hq,Hkv,D", [(1, 8, 8, 128), (3, 4, 2, 64), (9, 32, 32, 128), (16, 16, 8, 128), (40, 8, 8, 128), (60, 8, 8, 128)])
@pytest.mark.parametrize("window", [1, 40, 64, 1000, 4096])
@pytest.mark.parametrize("capacity", [500, 6000])
def test_paged_decode_partitions_of_a_window(n, Hq, Hkv, D, window, capacity):
    """What partitions of a sequence's own length share out are the tokens that a window shows, however many are cached, in as many as a table of
    that size has: the result against 64 bits, with lengths on and beside the window's edges."""
    import ctypes

    lib, cut = iops._get_lib(), []
    for room, w in ((capacity, window), (min(capacity, window + 15), 0), (capacity, 0)):
        part = ctypes.c_int(0)
        cut.append((lib.cb_decode_num_splits(n, Hkv, D, room, w, ctypes.byref(part)), part.value))
    assert cut[0][0] == (cut[1] if cut[0][1] < 0 else cut[2])[0]
    dev, page = "cuda", 16
    g = torch.Generator(device=dev).manual_seed(n + window)
    width = (capacity + page - 1) // page
    kc, vc = (torch.randn(300, page, Hkv, D, device=dev, generator=g).bfloat16() for _ in "kv")
    tables = torch.randint(0, 300, (n, width), device=dev, generator=g).to(torch.int32)
    edges = [capacity, capacity - 1, window, window + 1, window + 15, window + 16, window + 17, window // 2 + 1, 1, 17]
    lens = torch.tensor([min(max(1, edges[i % len(edges)]), capacity) for i in range(n)], device=dev, dtype=torch.int32)
    q = torch.randn(n, Hq, D, device=dev, generator=g).bfloat16()
    out = iops.paged_decode_attention(q, kc, vc, tables, lens, window=window)
    ref = _attention_in_64_bits(q, kc, vc, tables, lens, window)
    # weights rounded to 16 bits (2^-9 each), the result once more
    assert ((out.double() - ref).norm(dim=-1) <= 6e-3 * ref.norm(dim=-1)).all()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n,Hq,Hkv,D,length", [(1, 8, 8, 128, 8000), (4, 16, 4, 64, 7200), (12, 8, 1, 128, 6400), (16, 16, 8, 128, 800),
                                                   (4, 8, 8, 128, 3520), (8, 12, 12, 128, 1120), (1, 8, 8, 128, 7680)])
def test_paged_decode_weights_with_their_remainders(n, Hq, Hkv, D, length, dtype):
    """Sequences in partitions of more than 64 tokens (80 and 96 among them): the weights are not rounded to 16 bits, so what differs from 64 bits is the result's own rounding, and an
    infinite value is infinite in the result."""
    dev, page = "cuda", 16
    g = torch.Generator(device=dev).manual_seed(length)
    width = length // page
    lens = torch.tensor([length - 37 * i for i in range(n)], dtype=torch.int32, device=dev)
    tables = torch.randperm(n * width, device=dev, generator=g).view(n, width).to(torch.int32)
    q = torch.randn(n, Hq, D, device=dev, generator=g).to(dtype)
    kc, vc = (torch.randn(n * width, page, Hkv, D, device=dev, generator=g).to(dtype) for _ in "kv")
    out = iops.paged_decode_attention(q, kc, vc, tables, lens)
    ref = _attention_in_64_bits(q, kc, vc, tables, lens)
    # half a unit of the last place; weights, one in all, of values of about one: with twice eight bits and two signs 2^-18 (4e-6), and from scores whose
    # fp32 sums are off by some 2^-17 (8e-6)
    bits = 8 if dtype == torch.bfloat16 else 11
    assert ((out.double() - ref).abs() <= 2.0 ** -bits * ref.abs() + 2e-5).all()
    vc[tables[0, 3].long(), 5, 0, 7] = float("inf")
    got = iops.paged_decode_attention(q, kc, vc, tables, lens)
    same = torch.ones(n, Hq, D, dtype=torch.bool, device=dev)
    same[0, : Hq // Hkv, 7] = False
    assert (got[~same] == float("inf")).all() and torch.equal(got[same], out[same])
