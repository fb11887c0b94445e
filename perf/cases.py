"""What a user of the framework has it do, at the sizes of its own configurations: the cases that its speed is measured on.

A case is one call (forward, or forward and backward) of a public entry point:

  norm       ops.rms_norm with the residual sum fused, as between the sublayers of every decoder
  rope       ops.rope_qkv on the packed q | k | v rows of a projection
  glu        ops.glu on packed gate | up rows
  loss       the causal language-model loss and its gradient over the whole vocabulary
  attention  ops.attention over a packed batch of sequences (fine-tuning, and with no gradient the prefill of serving)
  decode     paged attention of one new token per sequence
  experts    dispatch, expert feed-forwards and combine of a sparse mixture-of-experts layer
  scan       decayed outer-product memory (lightning attention) over the prompts of a hybrid decoder
  step       one whole decode step of a decoder as the serving engine replays it, to the logits

`listed()` gives the cases, `draw()` more of the same ranges, `prepare()` what the caller holds before the call, `run()` one
pass, `work()` the bytes and operations the pass cannot do without, `tolerance()` what another correct implementation may
differ by, `exact()` the same results in 64 bits from plain torch operations.
"""
import math

import torch

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
SIZE = {"bf16": 2, "fp16": 2, "fp32": 4}
PAGE = 16                      # tokens per page of the key / value cache


def listed():
    return [
        # training, 2 x 4096 tokens of the 8B decoder: the second norm of a layer, forward and backward
        {"name": "norm_train", "kind": "norm", "rows": 8192, "hidden": 4096, "dtype": "bf16", "grad": True},
        # the same norm for the 16 tokens of a decode step: the smallest call there is
        {"name": "norm_serve", "kind": "norm", "rows": 16, "hidden": 4096, "dtype": "bf16", "grad": False},
        # rotary positions of the same layer (32 query and 8 key heads of 128), forward and backward
        {"name": "rope_train", "kind": "rope", "tokens": 8192, "heads": 32, "kv_heads": 8, "dim": 128, "rot": 128,
         "interleaved": False, "dtype": "bf16", "grad": True},
        # the gated unit of the same layer, forward and backward
        {"name": "glu_train", "kind": "glu", "rows": 8192, "inter": 14336, "act": "silu", "dtype": "bf16", "grad": True},
        # the loss over 4096 tokens and 128256 words, a third of the labels masked (prompts of instruction tuning)
        {"name": "loss_train", "kind": "loss", "rows": 4096, "vocab": 128256, "masked": 0.33, "dtype": "bf16"},
        # attention of the same decoder over 8192 packed tokens of uneven documents, forward and backward
        {"name": "attention_train", "kind": "attention", "tokens": 8192, "seqs": 5, "heads": 32, "kv_heads": 8, "dim": 128,
         "dtype": "bf16", "grad": True},
        # prefill of 16 prompts of about a thousand tokens, heads of 64
        {"name": "attention_prefill", "kind": "attention", "tokens": 16384, "seqs": 16, "heads": 32, "kv_heads": 8, "dim": 64,
         "dtype": "bf16", "grad": False},
        # decode attention of a full batch
        {"name": "decode_batch", "kind": "decode", "seqs": 64, "context": 2048, "heads": 32, "kv_heads": 8, "dim": 128,
         "dtype": "bf16"},
        # decode attention of a single conversation (four heads of a kind, an odd context)
        {"name": "decode_single", "kind": "decode", "seqs": 1, "context": 4097, "heads": 32, "kv_heads": 8, "dim": 128,
         "dtype": "fp16"},
        # a mixture-of-experts layer of the 16B model: 64 experts of which a token takes 6, forward and backward
        {"name": "experts_train", "kind": "experts", "tokens": 4096, "hidden": 2048, "inter": 1408, "experts": 64, "top": 6,
         "dtype": "bf16"},
        # lightning attention over eight prompts of uneven length (2048 wide hybrid decoder)
        {"name": "scan_prefill", "kind": "scan", "tokens": 12000, "seqs": 8, "heads": 16, "dim": 128, "vdim": 128,
         "carried": False, "dtype": "bf16"},
        # a whole decode step of four layers of the 8B decoder, 16 sequences, replayed from its graph
        {"name": "decode_step", "kind": "step", "seqs": 16, "context": 1024, "layers": 4, "hidden": 4096, "inter": 14336,
         "heads": 32, "kv_heads": 8, "dim": 128, "vocab": 32000, "dtype": "bf16"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["norm", "norm", "rope", "glu", "loss", "attention", "attention", "decode", "decode", "experts",
                       "scan", "step"])
    half = rng.choice(["bf16", "bf16", "fp16"])
    wide = rng.choice(["bf16", "bf16", "fp16", "fp32"])
    heads, kv = rng.choice([(32, 8), (32, 32), (16, 2), (40, 8), (12, 12), (64, 8), (24, 8)])
    if kind == "norm":
        hidden = rng.choice([768, 1024, 2048, 2560, 4096, 5120, 6144, 8192])
        grad = rng.random() < 0.6
        return {"kind": kind, "rows": _log(rng, 1, min(8192, 8192 * 4096 // hidden)), "hidden": hidden, "dtype": wide, "grad": grad}
    if kind == "rope":
        dim, rot, inter = rng.choice([(128, 128, False), (64, 64, False), (128, 64, True), (64, 32, False), (96, 96, False),
                                      (256, 64, True)])
        most = 8192 * 6144 // ((heads + 2 * kv) * dim)
        return {"kind": kind, "tokens": _log(rng, 1, most), "heads": heads, "kv_heads": kv, "dim": dim, "rot": rot,
                "interleaved": inter, "dtype": wide, "grad": rng.random() < 0.6}
    if kind == "glu":
        inter = rng.choice([1408, 2816, 5632, 8192, 11008, 13824, 14336])
        return {"kind": kind, "rows": _log(rng, 1, 8192 * 14336 // inter // 2), "inter": inter,
                "act": rng.choice(["silu", "silu", "gelu_tanh", "gelu"]), "dtype": wide, "grad": rng.random() < 0.6}
    if kind == "loss":
        vocab = rng.choice([32000, 50304, 102400, 128256, 151936])
        return {"kind": kind, "rows": _log(rng, 64, 4096 * 128256 // vocab // 2), "vocab": vocab,
                "masked": rng.choice([0.0, 0.33, 0.9]), "dtype": wide}
    if kind == "attention":
        grad = rng.random() < 0.5
        dim = 128 if grad else rng.choice([64, 128])
        seqs = _log(rng, 1, 24)
        return {"kind": kind, "tokens": max(_log(rng, 64, 8192 if grad else 16384), 2 * seqs), "seqs": seqs, "heads": heads,
                "kv_heads": kv, "dim": dim, "dtype": half, "grad": grad}
    if kind == "decode":
        seqs = _log(rng, 1, 128)
        return {"kind": kind, "seqs": seqs, "context": _log(rng, 17, min(16384, 131072 // seqs)), "heads": heads, "kv_heads": kv,
                "dim": rng.choice([64, 128, 128]), "dtype": half}
    if kind == "experts":
        experts, top = rng.choice([(8, 2), (16, 4), (64, 6), (64, 8)])
        hidden, inter = rng.choice([(1024, 512), (2048, 1408), (2048, 1024), (1536, 768)])
        return {"kind": kind, "tokens": _log(rng, 64, 4096), "hidden": hidden, "inter": inter, "experts": experts, "top": top,
                "dtype": half}
    if kind == "scan":
        dim = rng.choice([64, 128, 128])
        seqs = _log(rng, 1, 16)
        return {"kind": kind, "tokens": max(_log(rng, 32, 12000), 2 * seqs), "seqs": seqs, "heads": rng.choice([4, 8, 16]), "dim": dim,
                "vdim": rng.choice([dim, 96, 128]), "carried": rng.random() < 0.5, "dtype": wide}
    return {"kind": kind, "seqs": rng.choice([1, 2, 5, 8, 16, 24]), "context": _log(rng, 32, 1024), "layers": rng.choice([1, 2, 4]),
            "hidden": rng.choice([1024, 2048, 4096]), "inter": rng.choice([2816, 8192]), "heads": 16, "kv_heads": rng.choice([2, 4, 16]),
            "dim": rng.choice([64, 128]), "vocab": 32000, "dtype": half}


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, *shape, dtype=torch.float32, scale=1.0):
    return (torch.randn(*shape, device="cuda", generator=g) * scale).to(dtype)


def _lengths(total, parts, g):
    """`parts` uneven positive lengths that sum to `total`."""
    w = torch.rand(parts, device="cuda", generator=g).add_(0.35).cpu()
    out = [max(1, int(x)) for x in (w / w.sum() * total).tolist()]
    out[max(range(parts), key=lambda i: out[i])] += total - sum(out)
    return out


def _decays(heads):
    return [math.exp(-2.0 ** (-8.0 * (h + 1) / heads)) for h in range(heads)]


class _Unsharded:
    """What the loss reads of a shard configuration when nothing is sharded."""
    enable_tensor_parallelism = False
    enable_sequence_parallelism = False
    parallel_output = False
    tensor_parallel_process_group = None
    sequence_parallel_process_group = None
    sequence_parallelism_mode = None


def _pages(case, g, lens):
    """Key / value pages of `lens` cached tokens per sequence, in an order of their own, and the page tables."""
    width = -(-(case["context"] + 1) // PAGE)
    total = case["seqs"] * width
    table = torch.randperm(total, device="cuda", generator=g).to(torch.int32).view(case["seqs"], width)
    shape = (total, PAGE, case["kv_heads"], case["dim"])
    return table, shape


def prepare(case, seed):
    g = _gen(seed)
    dt = DTYPES[case["dtype"]]
    kind = case["kind"]
    s = {"case": case}
    if kind == "norm":
        R, H = case["rows"], case["hidden"]
        s.update(x=_randn(g, R, H, dtype=dt), r=_randn(g, R, H, dtype=dt, scale=2.0),
                 w=(1 + _randn(g, H, scale=0.1)).to(dt))
        if case["grad"]:
            s.update(gy=_randn(g, R, H, dtype=dt, scale=1e-2), gh=_randn(g, R, H, dtype=dt, scale=1e-2))
            for n in ("x", "r", "w"):
                s[n].requires_grad_(True)
    elif kind == "rope":
        from colossalai_b200 import ops

        T, width = case["tokens"], (case["heads"] + 2 * case["kv_heads"]) * case["dim"]
        s["qkv"] = _randn(g, T, width, dtype=dt)
        s["pos"] = torch.randint(0, 4096, (T,), device="cuda", generator=g)
        s["cos"], s["sin"] = ops.build_rope_cache(4096, case["rot"], 500000.0, device="cuda")
        if case["grad"]:
            s["qkv"].requires_grad_(True)
            s["g"] = _randn(g, T, width, dtype=dt, scale=1e-2)
    elif kind == "glu":
        s["gu"] = _randn(g, case["rows"], 2 * case["inter"], dtype=dt)
        if case["grad"]:
            s["gu"].requires_grad_(True)
            s["g"] = _randn(g, case["rows"], case["inter"], dtype=dt, scale=1e-2)
    elif kind == "loss":
        R, V = case["rows"], case["vocab"]
        s["logits"] = torch.empty(R, V, device="cuda", dtype=dt).normal_(0, 2.0, generator=g).requires_grad_(True)
        labels = torch.randint(0, V, (1, R), device="cuda", generator=g)
        labels[torch.rand(1, R, device="cuda", generator=g) < case["masked"]] = -100
        labels[0, -1] = 7                                        # one label counts whatever was masked
        s["labels"] = labels
    elif kind == "attention":
        T, D = case["tokens"], case["dim"]
        s["lens"] = _lengths(T, case["seqs"], g)
        cu = [0]
        for n in s["lens"]:
            cu.append(cu[-1] + n)
        s["cu"] = torch.tensor(cu, dtype=torch.int32, device="cuda")
        for n, h in (("q", case["heads"]), ("k", case["kv_heads"]), ("v", case["kv_heads"])):
            s[n] = _randn(g, T, h, D, dtype=dt).requires_grad_(case["grad"])
        if case["grad"]:
            s["g"] = _randn(g, T, case["heads"], D, dtype=dt, scale=1e-2)
    elif kind == "decode":
        n, C = case["seqs"], case["context"]
        lens = torch.randint(max(1, C // 2), C + 1, (n,), device="cuda", generator=g)
        lens[0] = C
        s["lens"] = lens.to(torch.int32)
        s["table"], shape = _pages(case, g, lens)
        s["kc"] = torch.empty(shape, device="cuda", dtype=dt).normal_(generator=g)
        s["vc"] = torch.empty(shape, device="cuda", dtype=dt).normal_(generator=g)
        s["q"] = _randn(g, n, case["heads"], case["dim"], dtype=dt)
    elif kind == "experts":
        from colossalai_b200.models import get_config
        from colossalai_b200.models.moe import GroupedExperts

        T, H, E = case["tokens"], case["hidden"], case["experts"]
        cfg = get_config("deepseek-moe-16b", hidden_size=H)
        torch.manual_seed(seed)
        with torch.device("cuda"):
            s["experts"] = GroupedExperts(cfg, E, case["inter"]).to(dt)
        s["x"] = _randn(g, T, H, dtype=dt).requires_grad_(True)
        # router scores with popular and unpopular experts
        score = (_randn(g, T, E) + _randn(g, 1, E, scale=0.5)).softmax(-1)
        w, s["idx"] = score.topk(case["top"], dim=-1)
        s["w"] = w.requires_grad_(True)
        s["g"] = _randn(g, T, H, dtype=dt, scale=1e-2)
    elif kind == "scan":
        from colossalai_b200.ops import mixers

        T, n, H, D, V = case["tokens"], case["seqs"], case["heads"], case["dim"], case["vdim"]
        s["lens"] = _lengths(T, n, g)
        s["ctx"] = [64 if case["carried"] and i % 2 == 0 else 0 for i in range(n)]
        s["meta"] = mixers.RaggedMeta.build(s["lens"], s["ctx"], list(range(n)), "cuda")
        s["q"], s["k"], s["v"] = (_randn(g, T, H * d, dtype=dt) for d in (D, D, V))
        s["decay"] = torch.tensor(_decays(H), device="cuda")
        s["state"] = _randn(g, n, H, D, V)
    else:
        s.update(_prepare_step(case, seed, g, dt))
    return s


def _prepare_step(case, seed, g, dt):
    from colossalai_b200.inference.graph_runner import CUDAGraphRunner
    from colossalai_b200.inference.modeling import PagedKVRuntime
    from colossalai_b200.models import build_model, get_config
    from colossalai_b200.models.transformer import SeqMeta

    n, C = case["seqs"], case["context"]
    cfg = get_config("llama3-8b", hidden_size=case["hidden"], intermediate_size=case["inter"], vocab_size=case["vocab"],
                     num_hidden_layers=case["layers"], num_attention_heads=case["heads"],
                     num_key_value_heads=case["kv_heads"], head_dim=case["dim"])
    torch.manual_seed(seed)
    with torch.device("cuda"):
        model = build_model(cfg).to(dt).eval()
    lens = torch.randint(max(1, C // 2), C + 1, (n,), device="cuda", generator=g)
    lens[0] = C
    table, shape = _pages(case, g, lens)
    caches = [[torch.empty(shape, device="cuda", dtype=dt).normal_(generator=g) for _ in range(case["layers"])] for _ in "kv"]
    rt = PagedKVRuntime(caches[0], caches[1], PAGE)
    ids = torch.randint(0, case["vocab"], (n,), device="cuda", generator=g)

    def forward(input_ids, block_tables, seq_lens, positions, token_seq, token_pos):
        rt.block_tables, rt.seq_lens, rt.is_prompt, rt.q_per_seq = block_tables, seq_lens, False, 1
        rt.token_seq, rt.token_pos, rt.cu_seqlens = token_seq, token_pos, None
        meta = SeqMeta(batch=1, seqlen=n, positions=positions)
        return model(input_ids=input_ids.view(1, -1), kv_cache=rt, meta=meta)["logits"]

    step = dict(input_ids=ids, block_tables=table, seq_lens=lens.to(torch.int32), positions=(lens - 1).long(),
                token_seq=torch.arange(n, dtype=torch.int32, device="cuda"), token_pos=(lens - 1).to(torch.int32))
    runner = CUDAGraphRunner(forward)
    with torch.inference_mode():
        runner.capture(**step)
    return {"model": model, "caches": caches, "runner": runner, "step": step}


# ------------------------------------------------------------------------------------------------ the pass
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "norm":
        from colossalai_b200 import ops

        if not case["grad"]:
            with torch.no_grad():
                return ops.rms_norm(s["x"], s["w"], 1e-5, s["r"])
        y, h = ops.rms_norm(s["x"], s["w"], 1e-5, s["r"])
        dx, dr, dw = torch.autograd.grad((y, h), (s["x"], s["r"], s["w"]), (s["gy"], s["gh"]))
        return y, h, dx, dr, dw
    if kind == "rope":
        from colossalai_b200 import ops

        def call():
            return ops.rope_qkv(s["qkv"], s["pos"], s["cos"], s["sin"], case["heads"], case["kv_heads"], case["dim"],
                                rot_dim=case["rot"], interleaved=case["interleaved"])

        if not case["grad"]:
            with torch.no_grad():
                return call()
        y = call()
        return y, torch.autograd.grad(y, s["qkv"], s["g"])[0]
    if kind == "glu":
        from colossalai_b200 import ops

        if not case["grad"]:
            with torch.no_grad():
                return ops.glu(s["gu"], case["act"])
        y = ops.glu(s["gu"], case["act"])
        return y, torch.autograd.grad(y, s["gu"], s["g"])[0]
    if kind == "loss":
        from colossalai_b200.shardformer.layer import dist_cross_entropy

        loss = dist_cross_entropy(s["labels"], s["logits"], _Unsharded, case["vocab"])
        return loss, torch.autograd.grad(loss, s["logits"])[0]
    if kind == "attention":
        from colossalai_b200 import ops

        if not case["grad"]:
            with torch.no_grad():
                return ops.attention(s["q"], s["k"], s["v"], causal=True, cu_seqlens_q=s["cu"], cu_seqlens_k=s["cu"],
                                     max_seqlen=max(s["lens"]))
        o = ops.attention(s["q"], s["k"], s["v"], causal=True, cu_seqlens_q=s["cu"], cu_seqlens_k=s["cu"],
                          max_seqlen=max(s["lens"]))
        return (o,) + torch.autograd.grad(o, (s["q"], s["k"], s["v"]), s["g"])
    if kind == "decode":
        from colossalai_b200.ops import inference

        with torch.no_grad():
            return inference.paged_decode_attention(s["q"], s["kc"], s["vc"], s["table"], s["lens"])
    if kind == "experts":
        from colossalai_b200.moe import dispatch_combine

        ex = s["experts"]
        y = dispatch_combine.moe_forward(s["x"], s["w"], s["idx"], ex, case["experts"], None)
        return (y,) + torch.autograd.grad(y, (s["x"], s["w"], ex.w_up, ex.w_down), s["g"])
    if kind == "scan":
        from colossalai_b200.ops import mixers

        with torch.no_grad():
            o = mixers.state_scan_decay(s["q"], s["k"], s["v"], s["decay"], s["state"], s["meta"], case["heads"], case["dim"],
                                        case["vdim"], act_silu=True)
        return o, s["state"]
    with torch.inference_mode():
        return s["runner"](**s["step"])


# ------------------------------------------------------------------------------------------------ work and tolerance
def work(case):
    kind, e = case["kind"], SIZE[case["dtype"]]
    if kind == "norm":
        n = case["rows"] * case["hidden"]
        # forward: x, residual in; y, sum out.  backward: dy, dsum, sum in; dx out
        return {"bytes": e * n * (8 if case["grad"] else 4), "flops": n * (14 if case["grad"] else 5)}
    if kind == "rope":
        n = case["tokens"] * (case["heads"] + 2 * case["kv_heads"]) * case["dim"]
        return {"bytes": e * n * (4 if case["grad"] else 2), "flops": 3 * n * (2 if case["grad"] else 1)}
    if kind == "glu":
        n = case["rows"] * case["inter"]
        return {"bytes": e * n * (8 if case["grad"] else 3), "flops": n * (20 if case["grad"] else 6)}
    if kind == "loss":
        n = case["rows"] * case["vocab"]
        # the gradient depends on the whole row: the logits are read twice and the gradient is written
        return {"bytes": 3 * e * n, "flops": 7 * n}
    if kind == "attention":
        T, H, G, D = case["tokens"], case["heads"], case["kv_heads"], case["dim"]
        n = T / case["seqs"]
        f = 4 * T * (n + 1) / 2 * H * D
        io = T * D * (2 * H + 2 * G)                             # q, k, v in, o out
        if not case["grad"]:
            return {"bytes": e * io, "flops": f}
        return {"bytes": e * (io + T * D * (4 * H + 4 * G)), "flops": 3.5 * f}
    if kind == "decode":
        n = case["seqs"] * case["context"] * 0.75 if case["seqs"] > 1 else case["context"]
        return {"bytes": e * (2 * n * case["kv_heads"] * case["dim"] + 2 * case["seqs"] * case["heads"] * case["dim"]),
                "flops": 4 * n * case["heads"] * case["dim"]}
    if kind == "experts":
        R, H, I, E = case["tokens"] * case["top"], case["hidden"], case["inter"], case["experts"]
        # weights in and their gradients out, tokens in and out in both directions
        return {"bytes": e * (3 * 3 * E * H * I + 4 * case["tokens"] * H), "flops": 3 * 2 * R * H * I * 3}
    if kind == "scan":
        T, H, D, V = case["tokens"], case["heads"], case["dim"], case["vdim"]
        return {"bytes": T * H * (e * (2 * D + V) + 4 * V) + 4 * case["seqs"] * H * D * V * (1.5 if case["carried"] else 1),
                "flops": 4 * T * H * D * V}
    n, L, W = case["seqs"], case["layers"], case["hidden"]
    q, kv = case["heads"] * case["dim"], case["kv_heads"] * case["dim"]
    params = L * (W * (2 * q + 2 * kv) + 3 * W * case["inter"]) + W * case["vocab"]
    tokens = n * case["context"] * 0.75 if n > 1 else case["context"]
    return {"bytes": e * (params + 2 * L * tokens * kv + n * case["vocab"]), "flops": 2 * n * params + 4 * L * tokens * q}


#: relative errors that a correct implementation shows by rounding its inputs, probabilities and results to 16 bits
_HALF = {"bf16": 6e-3, "fp16": 1e-3}


def tolerance(case):
    kind, dt = case["kind"], case["dtype"]
    if dt == "fp32":
        return {"rel": 1e-5, "max": 1e-3}
    rel = _HALF[dt]
    if kind in ("attention", "decode"):
        return {"rel": 2 * rel, "max": 40 * rel}
    if kind == "experts":
        return {"rel": 2.5 * rel, "max": 60 * rel}
    if kind == "scan":
        return {"rel": 1e-5, "max": 1e-3}                        # results and sums are 32-bit whatever the inputs are
    if kind == "step":
        return {"rel": 4 * rel, "max": 40 * rel}
    return {"rel": rel, "max": 8 * rel}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _rms(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _rotate(x, c, s, rot, interleaved):
    """x [T, heads, dim]; c, s [T, 1, rot / 2]."""
    a, b = (x[..., 0:rot:2], x[..., 1:rot:2]) if interleaved else (x[..., : rot // 2], x[..., rot // 2: rot])
    u, v = a * c - b * s, b * c + a * s
    y = torch.stack([u, v], -1).flatten(-2) if interleaved else torch.cat([u, v], -1)
    return torch.cat([y, x[..., rot:]], -1)


def _act(x, act):
    if act == "silu":
        return torch.nn.functional.silu(x)
    return torch.nn.functional.gelu(x, approximate="tanh" if act == "gelu_tanh" else "none")


def _causal(q, k, v):
    """One sequence: q [n, H, D], k / v [n, G, D]."""
    n, H, D = q.shape
    rep = H // k.shape[1]
    k, v = k.repeat_interleave(rep, 1), v.repeat_interleave(rep, 1)
    p = torch.einsum("qhd,khd->hqk", q, k) / math.sqrt(D)
    p = p.masked_fill(~torch.ones(n, n, dtype=torch.bool, device=q.device).tril(), float("-inf")).softmax(-1)
    return torch.einsum("hqk,khd->qhd", p, v)


def _cached(q, kc, vc, table, length):
    """One new token: q [H, D] over `length` cached tokens."""
    H, D = q.shape
    pages = table[: -(-length // PAGE)].long()
    k = kc[pages].flatten(0, 1)[:length].double()
    v = vc[pages].flatten(0, 1)[:length].double()
    rep = H // k.shape[1]
    p = (torch.einsum("hd,khd->hk", q, k.repeat_interleave(rep, 1)) / math.sqrt(D)).softmax(-1)
    return torch.einsum("hk,khd->hd", p, v.repeat_interleave(rep, 1))


def exact(case, seed):
    s = prepare(case, seed)
    kind = case["kind"]
    if kind == "norm":
        x, r, w = (s[n].detach().double().requires_grad_(case["grad"]) for n in ("x", "r", "w"))
        h = x + r
        y = _rms(h, w, 1e-5)
        if not case["grad"]:
            return y, h
        return (y.detach(), h.detach()) + torch.autograd.grad((y, h), (x, r, w), (s["gy"].double(), s["gh"].double()))
    if kind == "rope":
        def call(z):
            T, D, n = z.shape[0], case["dim"], case["heads"] + case["kv_heads"]
            c, sn = s["cos"][s["pos"]].double()[:, None], s["sin"][s["pos"]].double()[:, None]
            z = z.view(T, -1, D)
            return torch.cat([_rotate(z[:, :n], c, sn, case["rot"], case["interleaved"]), z[:, n:]], 1).flatten(1)

        z = s["qkv"].detach().double().requires_grad_(case["grad"])
        y = call(z)
        return (y.detach(), torch.autograd.grad(y, z, s["g"].double())[0]) if case["grad"] else y
    if kind == "glu":
        z = s["gu"].detach().double().requires_grad_(case["grad"])
        a, b = z.chunk(2, -1)
        y = _act(a, case["act"]) * b
        return (y.detach(), torch.autograd.grad(y, z, s["g"].double())[0]) if case["grad"] else y
    if kind == "loss":
        labels = torch.cat([s["labels"][0, 1:], s["labels"].new_full((1,), -100)])
        valid = labels != -100
        z = s["logits"].detach()
        total, n = 0.0, int(valid.sum())
        grad = torch.zeros(z.shape, dtype=torch.float64, device="cuda")
        for a in range(0, z.shape[0], 512):                      # a few hundred rows of 64-bit logits at a time
            rows = torch.arange(a, min(a + 512, z.shape[0]), device="cuda")
            zz, ok, t = z[rows].double(), valid[rows], labels[rows].clamp(min=0)
            lp = torch.log_softmax(zz, -1)
            total = total - (lp.gather(1, t[:, None])[:, 0] * ok).sum()
            p = lp.exp_()
            p[torch.arange(len(rows), device="cuda"), t] -= 1
            grad[rows] = p * (ok.double() / max(n, 1))[:, None]
        return total / max(n, 1), grad
    if kind == "attention":
        o, gs, a = [], [], 0
        for n in s["lens"]:
            q, k, v = (s[x][a:a + n].detach().double().requires_grad_(case["grad"]) for x in "qkv")
            parts, H, G = [], case["heads"], case["kv_heads"]
            rep = H // G
            if not case["grad"]:
                o.append(torch.cat([_causal(q[:, g * rep:(g + 1) * rep], k[:, g:g + 1], v[:, g:g + 1]) for g in range(G)], 1))
            else:
                for g in range(G):                               # one group of heads at a time: the weights are n x n
                    y = _causal(q[:, g * rep:(g + 1) * rep], k[:, g:g + 1], v[:, g:g + 1])
                    y.backward(s["g"][a:a + n, g * rep:(g + 1) * rep].double())
                    parts.append(y.detach())
                o.append(torch.cat(parts, 1))
                gs.append((q.grad, k.grad, v.grad))
            a += n
        return (torch.cat(o),) + tuple(torch.cat(t) for t in zip(*gs)) if case["grad"] else torch.cat(o)
    if kind == "decode":
        return torch.stack([_cached(s["q"][i].double(), s["kc"], s["vc"], s["table"][i], n)
                            for i, n in enumerate(s["lens"].tolist())])
    if kind == "experts":
        x, w = (s[n].detach().double().requires_grad_(True) for n in ("x", "w"))
        up, down = (getattr(s["experts"], n).detach().double().requires_grad_(True) for n in ("w_up", "w_down"))
        y = torch.zeros_like(x)
        for e in range(case["experts"]):
            tok, j = (s["idx"] == e).nonzero(as_tuple=True)
            a, b = (x[tok] @ up[e].t()).chunk(2, -1)
            y = y.index_add(0, tok, (torch.nn.functional.silu(a) * b) @ down[e].t() * w[tok, j][:, None])
        return (y.detach(),) + torch.autograd.grad(y, (x, w, up, down), s["g"].double())
    if kind == "scan":
        return _exact_scan(case, s)
    return _exact_step(case, s)


def _exact_scan(case, s):
    H, D, V, C = case["heads"], case["dim"], case["vdim"], 256
    lam = torch.tensor(_decays(H), dtype=torch.float32).double().cuda()          # the caller's decays are 32-bit numbers
    state, out, a = s["state"].double(), [], 0
    act = torch.nn.functional.silu
    q, k, v = (act(s[n].double()).view(-1, H, d) for n, d in (("q", D), ("k", D), ("v", V)))
    for i, n in enumerate(s["lens"]):
        S = state[i] if s["ctx"][i] > 0 else torch.zeros_like(state[i])
        for b in range(a, a + n, C):                             # chunks: inside one the weights are lam^(t - u)
            m = min(C, a + n - b)
            t = torch.arange(m, device="cuda", dtype=torch.float64)
            diff = t[:, None] - t[None]
            wt = torch.where(diff >= 0, lam[:, None, None] ** diff.clamp(min=0), torch.zeros_like(diff))
            sc = torch.einsum("thd,uhd->htu", q[b:b + m], k[b:b + m]) * wt
            o = torch.einsum("htu,uhv->thv", sc, v[b:b + m])
            o = o + torch.einsum("thd,hdv->thv", q[b:b + m], S) * (lam[None] ** (t[:, None] + 1))[..., None]
            S = S * (lam ** m)[:, None, None] + torch.einsum("uhd,uhv->hdv", k[b:b + m] * (lam[None] ** (m - 1 - t[:, None]))[..., None],
                                                             v[b:b + m])
            out.append(o.flatten(1))
        state[i] = S
        a += n
    return torch.cat(out), state


def _exact_step(case, s):
    sd = {k: v.detach() for k, v in s["model"].state_dict().items()}
    n, H, G, D = case["seqs"], case["heads"], case["kv_heads"], case["dim"]
    pos, lens = s["step"]["positions"], s["step"]["seq_lens"].tolist()
    base = 500000.0
    freq = base ** -(torch.arange(0, D, 2, dtype=torch.float64, device="cuda") / D)
    ang = pos.double()[:, None] * freq
    c, sn = ang.cos()[:, None], ang.sin()[:, None]
    eps = s["model"].cfg.norm_eps
    lin = lambda x, name: x @ sd[name].double().t()              # noqa: E731
    x = sd["model.embed_tokens.weight"][s["step"]["input_ids"]].double()
    for i in range(case["layers"]):
        p = "model.layers.%d." % i
        h = _rms(x, sd[p + "input_layernorm.weight"].double(), eps)
        q, k, v = lin(h, p + "self_attn.qkv_proj.weight").split([H * D, G * D, G * D], -1)
        q = _rotate(q.view(n, H, D), c, sn, D, False)
        k = _rotate(k.view(n, G, D), c, sn, D, False)
        v = v.view(n, G, D)
        o = []
        for j, m in enumerate(lens):                             # the new token's row stands in for the page's
            kc, vc = s["caches"][0][i], s["caches"][1][i]
            pages = s["step"]["block_tables"][j][: -(-m // PAGE)].long()
            kk = torch.cat([kc[pages].flatten(0, 1)[: m - 1].double(), k[j:j + 1]])
            vv = torch.cat([vc[pages].flatten(0, 1)[: m - 1].double(), v[j:j + 1]])
            rep = H // G
            w = (torch.einsum("hd,khd->hk", q[j], kk.repeat_interleave(rep, 1)) / math.sqrt(D)).softmax(-1)
            o.append(torch.einsum("hk,khd->hd", w, vv.repeat_interleave(rep, 1)).flatten())
        x = x + lin(torch.stack(o), p + "self_attn.o_proj.weight")
        h = _rms(x, sd[p + "post_attention_layernorm.weight"].double(), eps)
        a, b = lin(h, p + "mlp.gate_up_proj.weight").chunk(2, -1)
        x = x + lin(torch.nn.functional.silu(a) * b, p + "mlp.down_proj.weight")
    return lin(_rms(x, sd["model.norm.weight"].double(), eps), "lm_head.weight")
