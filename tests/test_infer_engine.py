"""Inference engine: continuous batching + paged KV vs naive full-recompute greedy decoding (CPU tier), scheduler /
KV manager / batch bucket unit checks (reference: tests/test_infer/test_{batch_bucket,kvcache_manager,
request_handler,inference_engine,continuous_batching,drafter}.py)."""
import pytest
import torch

from colossalai_b200.inference import InferenceConfig, InferenceEngine
from colossalai_b200.inference.batch_bucket import BatchBucket
from colossalai_b200.inference.config import GenerationConfig
from colossalai_b200.inference.kv_cache import KVCacheManager
from colossalai_b200.inference.struct import Sequence
from colossalai_b200.models import build_model, get_config


def _naive_greedy(model, prompt, n_new):
    ids = list(prompt)
    for _ in range(n_new):
        with torch.no_grad():
            logits = model(input_ids=torch.tensor([ids]))["logits"]
        ids.append(int(logits[-1, : model.cfg.vocab_size].argmax()))
    return ids


def test_kvcache_manager_alloc_free():
    cfg = InferenceConfig(max_batch_size=4, max_input_len=32, max_output_len=32, block_size=8, dtype="fp32")
    mc = get_config("llama-tiny")
    mgr = KVCacheManager(cfg, mc)
    total = mgr.total_num_blocks
    table = torch.full((mgr.get_max_blocks_per_sequence(),), -1, dtype=torch.int32)
    mgr.allocate_context_from_block_table(table, 19)
    assert (table >= 0).sum() == 3 and mgr.num_available_blocks == total - 3
    mgr.allocate_token_from_block_table(table, 25)          # position 24 -> needs block 3
    assert (table >= 0).sum() == 4
    mgr.free_block_table(table)
    assert mgr.num_available_blocks == total and (table < 0).all()


def test_batch_bucket_ops():
    bb = BatchBucket(4, 16, max_batch_size=4, max_length=64, block_size=8, kv_max_split_num=1)
    seqs = [Sequence(i, None, list(range(3 + i)), 8, None, 2, 0, 8) for i in range(3)]
    for s in seqs:
        bb.add_seq(s, alloc_block_table=torch.full((8,), i, dtype=torch.int32) if (i := s.request_id) >= 0 else None)
    assert bb.current_batch_size == 3 and bb.seq_lengths[:3].tolist() == [3, 4, 5]
    bb.append_batch_tokens(torch.tensor([7, 8, 9]))
    assert seqs[1].output_token_id == [8] and bb.seq_lengths[:3].tolist() == [4, 5, 6]
    bb.pop_seq_update_batch(0)
    assert bb.current_batch_size == 2 and bb.is_compact and bb.seq_lengths[:2].tolist() == [5, 6]


def test_engine_matches_naive_greedy_with_continuous_batching():
    torch.manual_seed(0)
    model = build_model("llama-tiny").float().eval()
    cfg = InferenceConfig(max_batch_size=3, max_input_len=24, max_output_len=6, block_size=8, dtype="fp32",
                          use_cuda_graph=False)
    engine = InferenceEngine(model, None, cfg)
    prompts = [[5, 9, 13, 200, 7], [11, 3], [400, 401, 402, 403, 404, 405, 406, 407, 408, 409], [17] * 6, [99, 98, 97]]
    outs, token_ids = engine.generate(prompts_token_ids=prompts, return_token_ids=True,
                                      generation_config=GenerationConfig(max_new_tokens=6))
    assert len(token_ids) == len(prompts)
    for p, got in zip(prompts, token_ids):
        ref = _naive_greedy(model, p, 6)
        # generation may stop early on EOS (id 2)
        assert got == ref[: len(got)], (p, got, ref)
        assert len(got) == len(ref) or got[-1] == 2


@pytest.mark.parametrize("replaced", ["nothing", "instance", "class", "subclass", "wrapper"])
def test_a_replaced_attend_of_the_cache_is_called_as_it_always_was(monkeypatch, replaced):
    """A step may leave the page write to the rotation's kernel only where the cache's own `attend` is what runs: a replacement gets the
    arguments that it always got, with keys and values not written yet.  (A stand-in for the kernel takes every call.)"""
    from colossalai_b200 import ops
    from colossalai_b200.inference.modeling import PagedKVRuntime
    from colossalai_b200.ops import inference as iops

    fused, calls = [], []

    def rope_pages(qkv, positions, cos, sin, heads, kv_heads, dim, rot, interleaved, kc, vc, tables, seq, pos):
        y = ops.rope_qkv(qkv, positions, cos, sin, heads, kv_heads, dim, rot_dim=rot, interleaved=interleaved)
        _, k, v = (t.reshape(len(y), -1, dim) for t in y.split([heads * dim, kv_heads * dim, kv_heads * dim], -1))
        iops.kv_cache_write(k, v, kc, vc, tables, seq, pos)
        fused.append(1)
        return y

    def attend(self, layer_idx, q, k, v, meta, scale):                    # a user's own, of before
        calls.append(1)
        return original(self, layer_idx, q, k, v, meta, scale)

    class Sub(PagedKVRuntime):
        def attend(self, layer_idx, q, k, v, meta, scale):
            calls.append(1)
            return super().attend(layer_idx, q, k, v, meta, scale)

    class Wrapper:
        def __init__(self, inner):
            self.inner = inner

        def attend(self, layer_idx, q, k, v, meta, scale):
            calls.append(1)
            return self.inner.attend(layer_idx, q, k, v, meta, scale)

        def __getattr__(self, name):
            return getattr(self.inner, name)

    original = PagedKVRuntime.attend
    monkeypatch.setattr(iops, "rope_pages", rope_pages)
    torch.manual_seed(0)
    model = build_model("llama-tiny").float().eval()
    cfg = InferenceConfig(max_batch_size=2, max_input_len=24, max_output_len=6, block_size=8, dtype="fp32", use_cuda_graph=False)
    engine = InferenceEngine(model, None, cfg)
    owner = engine.engine
    rt = owner.kv_runtime
    if replaced == "instance":
        rt.attend = attend.__get__(rt)
    elif replaced == "class":
        monkeypatch.setattr(PagedKVRuntime, "attend", attend)
    elif replaced == "subclass":
        rt.__class__ = Sub
    elif replaced == "wrapper":
        owner.kv_runtime = Wrapper(rt)
    prompt = [5, 9, 13, 200, 7]
    _, ids = engine.generate(prompts_token_ids=[prompt], return_token_ids=True, generation_config=GenerationConfig(max_new_tokens=6))
    want = _naive_greedy(model, prompt, 6)
    assert len(ids[0]) > 1 and ids[0] == want[: len(ids[0])]
    assert bool(fused) == (replaced == "nothing") and bool(calls) == (replaced != "nothing")


def test_speculative_decoding_matches_plain_greedy():
    torch.manual_seed(0)
    model = build_model("llama-tiny").float().eval()
    torch.manual_seed(1)
    drafter = build_model(get_config("llama-tiny", num_hidden_layers=1)).float().eval()
    cfg = InferenceConfig(max_batch_size=2, max_input_len=16, max_output_len=8, block_size=8, dtype="fp32",
                          max_n_spec_tokens=4)
    plain = InferenceEngine(model, None, cfg)
    prompts = [[5, 9, 13, 200, 7], [11, 3, 4]]
    _, ref_ids = plain.generate(prompts_token_ids=prompts, return_token_ids=True,
                                generation_config=GenerationConfig(max_new_tokens=8))
    spec = InferenceEngine(model, None, cfg)
    spec.enable_spec_dec(drafter, n_spec_tokens=3)
    _, got_ids = spec.generate(prompts_token_ids=prompts, return_token_ids=True,
                               generation_config=GenerationConfig(max_new_tokens=8))
    for r, g in zip(ref_ids, got_ids):
        n = min(len(r), len(g))
        assert r[:n] == g[:n], (r, g)


def test_async_engine_and_http_server():
    import asyncio

    from fastapi.testclient import TestClient

    from colossalai_b200.inference.core.async_engine import AsyncInferenceEngine
    from colossalai_b200.inference.server.api_server import build_app

    torch.manual_seed(0)
    model = build_model("llama-tiny").float().eval()
    cfg = InferenceConfig(max_batch_size=4, max_input_len=64, max_output_len=8, block_size=8, dtype="fp32")

    async def run():
        eng = AsyncInferenceEngine(start_engine_loop=True, model_or_path=model, tokenizer=None, inference_config=cfg)
        outs = await asyncio.gather(*[_collect(eng, i, p) for i, p in enumerate(["hello", "abc", "xyzw"])])
        assert eng.background_loop_status
        return outs

    async def _collect(eng, rid, prompt):
        res = None
        async for o in eng.generate(rid, prompt):
            res = o
        return res

    outs = asyncio.run(run())
    assert len(outs) == 3 and all(isinstance(o, str) for o in outs)

    eng = AsyncInferenceEngine(start_engine_loop=True, model_or_path=model, tokenizer=None, inference_config=cfg)
    with TestClient(build_app(eng, "llama-tiny")) as client:
        assert client.get("/ping").json() == {"status": "Healthy"}
        assert "cb200_kv_blocks_free" in client.get("/metrics").text
        r = client.post("/generate", json={"prompt": "hello", "max_new_tokens": 4})
        assert r.status_code == 200 and "text" in r.json()
        r = client.post("/completion", json={"prompt": "hi there", "max_new_tokens": 4})
        assert r.status_code == 200 and r.json()["model"] == "llama-tiny"
        r = client.post("/chat", json={"messages": [{"role": "user", "content": "hi"}], "max_new_tokens": 4})
        assert r.status_code == 200 and r.json()["choices"][0]["message"]["role"] == "assistant"


def test_rpc_engine_matches_local_engine():
    from colossalai_b200.inference.core.rpc_engine import RPCInferenceEngine

    cfg = InferenceConfig(max_batch_size=2, max_input_len=16, max_output_len=6, block_size=8, dtype="fp32", tp_size=1)
    prompts = [[5, 9, 13, 200, 7], [11, 3, 4]]
    torch.manual_seed(1234)
    local = InferenceEngine(build_model("llama-tiny").float().eval(), None, cfg)
    _, ref = local.generate(prompts_token_ids=prompts, return_token_ids=True,
                            generation_config=GenerationConfig(max_new_tokens=6))
    rpc = RPCInferenceEngine("llama-tiny", None, cfg)
    try:
        _, got = rpc.generate(prompts_token_ids=prompts, return_token_ids=True,
                              generation_config=GenerationConfig(max_new_tokens=6))
    finally:
        rpc.kill_workers()
    assert got == ref


def _tp_worker(rank, world_size, port):
    import copy

    import torch.distributed as dist

    import colossalai_b200

    colossalai_b200.launch(rank, world_size, "127.0.0.1", port, backend="gloo", verbose=False)
    torch.manual_seed(0)
    model = build_model("llama-tiny").float().eval()
    prompts = [[5, 9, 13, 200, 7], [11, 3], [17] * 6]
    gen = GenerationConfig(max_new_tokens=6)
    kw = dict(max_batch_size=4, max_input_len=16, max_output_len=6, block_size=8, dtype="fp32")
    _, ref_ids = InferenceEngine(copy.deepcopy(model), None, InferenceConfig(**kw)).generate(
        prompts_token_ids=prompts, return_token_ids=True, generation_config=gen)
    eng = InferenceEngine(model, None, InferenceConfig(tp_size=2, **kw))        # TP-sharded through the policy
    _, ids = eng.generate(prompts_token_ids=prompts, return_token_ids=True, generation_config=gen)
    assert ids == ref_ids, (ids, ref_ids)
    dist.barrier()
    dist.destroy_process_group()


def test_tensor_parallel_engine_matches_single_rank():
    from colossalai_b200.testing import spawn

    spawn(_tp_worker, 2)


def _tp_ckpt_worker(rank, world_size, port, tmp):
    import torch.distributed as dist
    import transformers

    import colossalai_b200

    colossalai_b200.launch(rank, world_size, "127.0.0.1", port, backend="gloo", verbose=False)
    if rank == 0:
        torch.manual_seed(0)
        hf = transformers.LlamaForCausalLM(transformers.LlamaConfig(
            vocab_size=128, hidden_size=64, intermediate_size=96, num_hidden_layers=2, num_attention_heads=4,
            num_key_value_heads=2, max_position_embeddings=64))
        hf.save_pretrained(tmp, safe_serialization=True)
    dist.barrier()
    prompts = [[5, 9, 13, 20, 7], [11, 3]]
    gen = GenerationConfig(max_new_tokens=5)
    kw = dict(max_batch_size=2, max_input_len=16, max_output_len=5, block_size=8, dtype="fp32")
    _, ref_ids = InferenceEngine(tmp, None, InferenceConfig(**kw)).generate(
        prompts_token_ids=prompts, return_token_ids=True, generation_config=gen)
    _, ids = InferenceEngine(tmp, None, InferenceConfig(tp_size=2, **kw)).generate(
        prompts_token_ids=prompts, return_token_ids=True, generation_config=gen)
    assert ids == ref_ids, (ids, ref_ids)
    dist.barrier()
    dist.destroy_process_group()


def test_tp_engine_loads_hf_checkpoint(tmp_path):
    pytest.importorskip("transformers")
    from colossalai_b200.testing import spawn

    spawn(_tp_ckpt_worker, 2, tmp=str(tmp_path))


def test_engine_alibi_family_matches_naive_greedy():
    """Baichuan-13B-style ALiBi model through the paged runtime (reference: test_infer/test_models/test_baichuan.py)."""
    torch.manual_seed(0)
    model = build_model("baichuan-tiny").float().eval()
    model.fold_norm_head()
    cfg = InferenceConfig(max_batch_size=2, max_input_len=16, max_output_len=5, block_size=8, dtype="fp32",
                          use_cuda_graph=False)
    engine = InferenceEngine(model, None, cfg)
    prompts = [[5, 9, 13, 200, 7, 8, 9, 10, 11], [11, 3, 77]]
    _, token_ids = engine.generate(prompts_token_ids=prompts, return_token_ids=True,
                                   generation_config=GenerationConfig(max_new_tokens=5))
    for p, got in zip(prompts, token_ids):
        ref = _naive_greedy(model, p, 5)
        assert got == ref[: len(got)], (p, got, ref)


def test_glide_drafter_spec_dec_matches_plain_greedy():
    """GLIDE drafter (cross-attends to the target model's paged KV) must not change the verified output."""
    from colossalai_b200.inference.modeling.models import GlideLlamaConfig, GlideLlamaForCausalLM

    torch.manual_seed(0)
    model = build_model("llama-tiny").float().eval()
    mc = model.cfg
    torch.manual_seed(1)
    gcfg = GlideLlamaConfig(vocab_size=mc.vocab_size, hidden_size=32, intermediate_size=64, num_hidden_layers=1,
                            num_attention_heads=2, num_key_value_heads=2, max_position_embeddings=256,
                            large_hidden_size=mc.hidden_size, large_num_attention_heads=mc.num_attention_heads,
                            large_num_key_value_heads=mc.num_key_value_heads, large_head_dim=mc.head_dim)
    drafter = GlideLlamaForCausalLM(gcfg).float().eval()
    cfg = InferenceConfig(max_batch_size=2, max_input_len=16, max_output_len=8, block_size=8, dtype="fp32",
                          max_n_spec_tokens=4)
    plain = InferenceEngine(model, None, cfg)
    prompts = [[5, 9, 13, 200, 7], [11, 3, 4]]
    _, ref_ids = plain.generate(prompts_token_ids=prompts, return_token_ids=True,
                                generation_config=GenerationConfig(max_new_tokens=8))
    spec = InferenceEngine(model, None, cfg)
    spec.enable_spec_dec(drafter, n_spec_tokens=3, use_glide_drafter=True)
    _, got_ids = spec.generate(prompts_token_ids=prompts, return_token_ids=True,
                               generation_config=GenerationConfig(max_new_tokens=8))
    for r, g in zip(ref_ids, got_ids):
        n = min(len(r), len(g))
        assert r[:n] == g[:n]
    # the glimpse path really ran: a glide forward differs from the plain drafter forward
    from colossalai_b200.inference.spec import GlideInput

    kc = torch.randn(4, 8, mc.num_key_value_heads, mc.head_dim)
    g = GlideInput(block_tables=torch.tensor([[0, 1]], dtype=torch.int32), large_k_cache=kc, large_v_cache=kc.clone(),
                   sequence_lengths=torch.tensor([11]), n_spec_tokens=3)
    ids = torch.tensor([[5, 6, 7]])
    a = drafter(input_ids=ids)["logits"]
    b = drafter(input_ids=ids, glide_input=g)["logits"]
    assert not torch.allclose(a, b)


def test_attention_backends_agree_with_runtime_reference():
    from colossalai_b200.inference.modeling.backends import (AttentionMetaData, ReferenceAttentionBackend,
                                                             get_attention_backend, get_pre_attention_backend)

    torch.manual_seed(0)
    Hq, Hkv, D, bs = 4, 2, 16, 4
    lens = [5, 3]
    T = sum(lens)
    q, k, v = torch.randn(T, Hq, D), torch.randn(T, Hkv, D), torch.randn(T, Hkv, D)
    kc, vc = torch.zeros(6, bs, Hkv, D), torch.zeros(6, bs, Hkv, D)
    bt = torch.tensor([[0, 1, -1], [2, 3, -1]], dtype=torch.int32)
    cu = torch.tensor([0, 5, 8], dtype=torch.int32)
    seq = torch.tensor([0] * 5 + [1] * 3, dtype=torch.int32)
    pos = torch.tensor([0, 1, 2, 3, 4, 0, 1, 2], dtype=torch.int32)
    md = AttentionMetaData(q, k, v, kc, vc, bt, bs, kv_seq_len=5, sequence_lengths=torch.tensor(lens, dtype=torch.int32),
                           cu_seqlens=cu)
    get_pre_attention_backend(use_alibi_attn=True).prefill(md, token_seq=seq, token_pos=pos)
    assert torch.equal(kc[1, 0], k[4]) and torch.equal(vc[2, 2], v[7])
    be = get_attention_backend(use_cuda_kernel=False)
    assert isinstance(be, ReferenceAttentionBackend)
    out = be.prefill(md)
    # last token of every sequence: decode over the cache must reproduce the prefill row
    md2 = AttentionMetaData(q[[4, 7]], None, None, kc, vc, bt, bs, sequence_lengths=torch.tensor(lens, dtype=torch.int32))
    dec = be.decode(md2)
    torch.testing.assert_close(dec, out[[4, 7]], atol=1e-5, rtol=1e-5)


def test_streamingllm_window_eviction_bounds_kv_blocks():
    """StreamingLLM (reference inference/config.py:enable_streamingllm, batch_bucket.py:streamingllm_update_batch):
    once sink + generated window is full the oldest non-sink block is recycled, so a long generation holds a bounded
    number of KV blocks; until the first eviction the tokens equal plain greedy decoding."""
    torch.manual_seed(0)
    model = build_model("llama-tiny").float().eval()
    kw = dict(max_batch_size=2, max_input_len=16, max_output_len=64, block_size=8, dtype="fp32", use_cuda_graph=False,
              ignore_eos=True)
    prompts = [[5, 9, 13, 200, 7], [11, 3, 8]]
    gen = GenerationConfig(max_new_tokens=60)
    _, plain = InferenceEngine(model, None, InferenceConfig(**kw)).generate(
        prompts_token_ids=prompts, return_token_ids=True, generation_config=gen)
    cfg = InferenceConfig(enable_streamingllm=True, start_token_size=4, generated_token_size=16, **kw)
    assert cfg.start_token_size == 8                         # sinks are rounded up to one block
    eng = InferenceEngine(model, None, cfg)
    mgr = eng.request_handler.cache_manager
    total = mgr.num_available_blocks
    peak = []
    orig = eng.request_handler.update

    def spy():
        out = orig()
        peak.append(total - mgr.num_available_blocks)
        return out

    eng.request_handler.update = spy
    _, ids = eng.generate(prompts_token_ids=prompts, return_token_ids=True, generation_config=gen)
    window = cfg.start_token_size + cfg.generated_token_size + cfg.block_size        # eviction threshold (tokens)
    for p, a, b in zip(prompts, plain, ids):
        assert len(b) == len(p) + 60
        n_same = window - 1
        assert a[:n_same] == b[:n_same]
    # two sequences, each at most window/block_size (+1 being filled) blocks
    assert max(peak) <= 2 * (window // cfg.block_size + 1)
    assert max(peak) < 2 * ((16 + 64) // cfg.block_size)
    assert mgr.num_available_blocks == total


def test_engine_sliding_window_matches_naive_greedy():
    """Mistral-style sliding window in the paged engine: prompts and generations that outgrow the window follow the
    banded full-recompute oracle (prefill band mask, decode over the last `window` cached tokens)."""
    torch.manual_seed(0)
    model = build_model(get_config("mistral-tiny", sliding_window=6)).float().eval()
    cfg = InferenceConfig(max_batch_size=2, max_input_len=16, max_output_len=10, block_size=8, dtype="fp32",
                          use_cuda_graph=False, ignore_eos=True)
    eng = InferenceEngine(model, None, cfg)
    prompts = [[5, 9, 13, 200, 7, 21, 22, 23, 24, 25, 26], [11, 3, 8]]          # one prompt already beyond the window
    _, ids = eng.generate(prompts_token_ids=prompts, return_token_ids=True,
                          generation_config=GenerationConfig(max_new_tokens=10))
    for p, got in zip(prompts, ids):
        assert got == _naive_greedy(model, p, 10), (p, got)


def test_async_engine_drains_waiting_requests():
    """More concurrent requests than batch slots: the background loop must keep stepping while requests are WAITING
    even when a step retired every running sequence (it used to park on the new-request event and hang)."""
    import asyncio

    from colossalai_b200.inference.core.async_engine import AsyncInferenceEngine

    torch.manual_seed(0)
    model = build_model("llama-tiny").float().eval()
    cfg = InferenceConfig(max_batch_size=2, max_input_len=32, max_output_len=4, block_size=8, dtype="fp32")

    async def one(eng, rid):
        out = None
        async for o in eng.generate(rid, f"prompt number {rid}", generation_config=GenerationConfig(max_new_tokens=2 + rid % 3)):
            out = o
        return out

    async def run():
        eng = AsyncInferenceEngine(start_engine_loop=True, model_or_path=model, tokenizer=None, inference_config=cfg)
        for wave in range(3):                           # waves: clients only send the next request after an answer
            outs = await asyncio.wait_for(asyncio.gather(*[one(eng, 10 * wave + i) for i in range(7)]), timeout=120)
            assert len(outs) == 7 and all(isinstance(o, str) for o in outs)
        rh = eng.engine.engine.request_handler
        assert not rh.check_unfinished_reqs() and rh.total_requests_in_batch_bucket() == 0

    asyncio.run(run())
