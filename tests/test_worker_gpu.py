"""The drop-in itself on a B200: the reference's BaseWorker / BrokerManager (unmodified, from
baseline/_ref or the mounted reference) + B200Worker loading a model DIRECTORY (config.json, safetensors,
tokenizer files — what `llmq worker run <model> <queue>` gets), jobs in through the broker,
results out of `<queue>.results`, texts compared with the CPU oracle's greedy decode."""
import asyncio
import os
import sys

import pytest

from tests.conftest import needs_reference

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "tests", "shims"))
for p in (os.path.join(ROOT, "baseline", "_ref"), "/root/reference"):
    if os.path.isdir(os.path.join(p, "llmq")):
        sys.path.insert(0, p)
        break
os.environ.setdefault("LLMQ_LOG_LEVEL", "WARNING")


@needs_reference
def test_b200_worker_end_to_end_from_model_dir(cuda, tmp_path, monkeypatch):
    import aio_pika
    from llmq.core.broker import BrokerManager
    from llmq.core.models import Job, Result

    from llmq_b200.fixtures import seeded_state_dict, write_model_dir
    from llmq_b200.model import ModelSpec
    from llmq_b200.worker import B200Worker
    from oracle.model import LlamaDims, LlamaOracle

    spec = ModelSpec(hidden=512, n_layers=2, n_q_heads=8, n_kv_heads=2, head_dim=128, intermediate=1024,
                     vocab=2048, max_position_embeddings=256, name="tiny")
    mdir = write_model_dir(str(tmp_path / "tiny-llama"), spec, seed=77, with_weights=True)
    monkeypatch.setenv("VLLM_MAX_TOKENS", "10")
    monkeypatch.setenv("VLLM_MAX_NUM_SEQS", "8")
    monkeypatch.setenv("VLLM_MAX_MODEL_LEN", "256")
    monkeypatch.setenv("VLLM_GPU_MEMORY_UTILIZATION", "0.3")
    monkeypatch.setenv("B200Q_MAX_NUM_BATCHED_TOKENS", "256")
    aio_pika.reset_brokers()

    async def main():
        w = B200Worker(mdir, "gq", tensor_parallel_size=1)
        task = asyncio.create_task(w.run())
        b = BrokerManager()
        await b.connect()
        await b.setup_queue_infrastructure("gq")
        # greedy for the oracle comparison: B200Q_TEMPERATURE=0 for j0..j5, a per-job `temperature`
        # extra for j6..j11 (the worker's default is the reference's 0.7, exercised by "sampled")
        jobs = [Job(id=f"j{i}", prompt="w5 {x} w9", x=f"w{20 + i}", tag=i, temperature=0) for i in range(12)]
        jobs.append(Job(id="sampled", prompt="w5 w6", seed=5))
        jobs.append(Job(id="sampled-again", prompt="w5 w6", seed=5))
        jobs.append(Job(id="sampled-other", prompt="w5 w6", seed=6))
        jobs.append(Job(id="chat", messages=[{"role": "user", "content": "w5 w6 w7"}]))
        jobs.append(Job(id="long", prompt=" ".join(["w11"] * 300)))  # > VLLM_MAX_MODEL_LEN: dropped
        for j in jobs:
            await b.publish_job("gq", j)
        got = {}

        async def on_res(m):
            r = Result.parse_raw(m.body)
            got[r.id] = r
            await m.ack()

        await b.consume_results("gq", on_res)
        for _ in range(600):
            if len(got) >= len(jobs) - 1:
                break
            await asyncio.sleep(0.05)
        tok = w.service.tokenizer
        w.running = False
        await asyncio.wait_for(task, 30)
        return got, tok

    got, tok = asyncio.run(main())
    assert "long" not in got and len(got) == 16
    assert got["sampled"].result == got["sampled-again"].result  # same prompt + seed => same draw
    assert len(got["sampled"].result.split()) >= 1
    sd = seeded_state_dict(spec, 77)
    oracle = LlamaOracle(LlamaDims.from_hf_config(spec.to_hf_config()), sd, "bf16", max_pos=256)
    n_exact = 0
    for i in range(12):
        ids = tok(f"w5 w{20 + i} w9", add_special_tokens=True).input_ids
        ref, lg = oracle.greedy(ids, 10, eos_id=tok.eos_token_id, return_logits=True)
        # the worker returns the continuation of the prompt's text (vLLM's prompt-primed DecodeStream)
        ref_text = tok.decode(list(ids) + list(ref), skip_special_tokens=True)[len(tok.decode(ids, skip_special_tokens=True)):]
        r = got[f"j{i}"]
        assert r.prompt == f"w5 w{20 + i} w9" and r.model_dump()["tag"] == i and r.worker_id.startswith("b200-")
        if r.result == ref_text:
            n_exact += 1
        else:  # allowed only from a bf16 near-tie onwards
            out = tok(r.result, add_special_tokens=False).input_ids
            k = next((j for j in range(min(len(out), len(ref))) if out[j] != ref[j]), min(len(out), len(ref)))
            top2 = lg[min(k, len(lg) - 1)].topk(2).values
            assert (top2[0] - top2[1]).item() < 0.12, (i, k, r.result, ref_text)
    assert n_exact >= 9, f"only {n_exact}/12 texts identical to the oracle's"
    assert got["chat"].prompt == "Chat with 1 messages" and isinstance(got["chat"].result, str)


@needs_reference
def test_b200_worker_end_to_end_from_gemma2_model_dir(cuda, tmp_path, monkeypatch):
    """the same drop-in path with a Gemma-2 checkpoint directory (config.json says
    Gemma2ForCausalLM; tests/test_gemma2_host.py shows transformers loads the very same directory):
    greedy texts against the Gemma-2 oracle, prompts and generations crossing the 16-token window"""
    import aio_pika
    from llmq.core.broker import BrokerManager
    from llmq.core.models import Job, Result

    from llmq_b200.fixtures import seeded_state_dict, write_model_dir
    from llmq_b200.model import ModelSpec
    from llmq_b200.worker import B200Worker
    from oracle.gemma2 import Gemma2Dims, Gemma2Oracle

    spec = ModelSpec(hidden=256, n_layers=3, n_q_heads=4, n_kv_heads=2, head_dim=128, intermediate=512, vocab=2048,
                     rms_eps=1e-6, rope_theta=10000.0, tie_embeddings=True, max_position_embeddings=256,
                     name="tiny-gemma2", arch="gemma2", query_pre_attn_scalar=128.0, attn_softcap=50.0,
                     final_softcap=30.0, sliding_window=16)
    mdir = write_model_dir(str(tmp_path / "tiny-gemma2"), spec, seed=78, with_weights=True)
    monkeypatch.setenv("VLLM_MAX_TOKENS", "10")
    monkeypatch.setenv("VLLM_MAX_NUM_SEQS", "8")
    monkeypatch.setenv("VLLM_MAX_MODEL_LEN", "256")
    monkeypatch.setenv("VLLM_GPU_MEMORY_UTILIZATION", "0.3")
    monkeypatch.setenv("B200Q_MAX_NUM_BATCHED_TOKENS", "64")
    monkeypatch.setenv("B200Q_TEMPERATURE", "0")
    aio_pika.reset_brokers()
    prompts = [" ".join(f"w{30 + 7 * i + j}" for j in range(3 + 5 * i)) for i in range(8)]  # 3 .. 38 words

    async def main():
        w = B200Worker(mdir, "gq2", tensor_parallel_size=1)
        task = asyncio.create_task(w.run())
        b = BrokerManager()
        await b.connect()
        await b.setup_queue_infrastructure("gq2")
        for i, p in enumerate(prompts):
            await b.publish_job("gq2", Job(id=f"g{i}", prompt=p))
        got = {}

        async def on_res(m):
            r = Result.parse_raw(m.body)
            got[r.id] = r
            await m.ack()

        await b.consume_results("gq2", on_res)
        for _ in range(600):
            if len(got) >= len(prompts):
                break
            await asyncio.sleep(0.05)
        tok = w.service.tokenizer
        w.running = False
        await asyncio.wait_for(task, 30)
        return got, tok

    got, tok = asyncio.run(main())
    assert len(got) == len(prompts)
    d = Gemma2Dims(hidden=256, n_layers=3, n_q_heads=4, n_kv_heads=2, head_dim=128, intermediate=512, vocab=2048,
                   query_pre_attn_scalar=128.0, sliding_window=16, max_pos=256)
    oracle = Gemma2Oracle(d, seeded_state_dict(spec, 78), "bf16")
    n_exact = 0
    for i, p in enumerate(prompts):
        ids = tok(p, add_special_tokens=True).input_ids
        ref, lg = oracle.greedy(ids, 10, return_logits=True)
        if tok.eos_token_id in ref:  # the worker stops at EOS; the oracle's greedy() does not
            ref = ref[: ref.index(tok.eos_token_id)]
        # the worker returns the continuation of the prompt's text (vLLM's prompt-primed DecodeStream)
        ref_text = tok.decode(list(ids) + list(ref), skip_special_tokens=True)[len(tok.decode(ids, skip_special_tokens=True)):]
        r = got[f"g{i}"]
        assert r.prompt == p and r.worker_id.startswith("b200-")
        if r.result == ref_text:
            n_exact += 1
        else:  # allowed only from a bf16 near-tie onwards
            out = tok(r.result, add_special_tokens=False).input_ids
            k = next((j for j in range(min(len(out), len(ref))) if out[j] != ref[j]), min(len(out), len(ref)))
            top2 = lg[min(k, len(lg) - 1)].topk(2).values
            assert (top2[0] - top2[1]).item() < 0.16, (i, k, r.result, ref_text)
    # random-init Gemma-2 logits are soft-capped and close together (top-2 margins of 0.00-0.06 on
    # this model), so the margin rule above carries the check; exact agreement is the common case
    assert n_exact >= 3, f"only {n_exact}/8 texts identical to the oracle's"


def test_two_engines_back_to_back_in_one_process_get_the_same_kv_pool(cuda):
    """`gpu_memory_utilization` sizes the KV pool from what the device
    has left; memory this process had freed to torch's caching allocator (the previous engine's
    pool) used to be counted as in use, so a second engine in the same process got 0 blocks.
    Building, closing and rebuilding at the same utilisation must give the same pool (± a few MB of
    allocator granularity), and the close must return the memory to the driver."""
    import torch

    from llmq_b200.service import build_service

    sizes, free_after = [], []
    torch.cuda.empty_cache()
    free0 = torch.cuda.mem_get_info()[0]
    for _ in range(3):
        svc = build_service("random:gemma-2-2b", max_num_seqs=16, max_model_len=256, gpu_memory_utilization=0.3,
                            max_num_batched_tokens=256, seed=1)
        sizes.append(svc.engine.model.num_blocks)
        eng, model = svc.engine, svc.engine.model
        eng.add_request(0, [5, 6, 7], 4, ignore_eos=True)
        n = 0
        while eng.has_work():
            n += len(eng.step()[0])
        assert n == 4
        eng.close()
        model.close()
        del svc, eng, model
        free_after.append(torch.cuda.mem_get_info()[0])
    assert min(sizes) > 1000, sizes
    assert max(sizes) - min(sizes) <= max(sizes) // 100, f"KV pool shrank across rebuilds: {sizes}"
    assert min(free_after) > free0 - (1 << 30), f"memory not returned to the driver: {free_after} vs {free0} before"


@needs_reference
def test_two_stage_pipeline_on_the_gpu_with_braces_in_stage1_output(cuda, tmp_path, monkeypatch):
    """config #4 with real model output: two B200Worker stages on the GPU, stage 1's
    text routed into stage 2's queue by the reference's unmodified `publish_pipeline_result`
    (ref:llmq/core/broker.py:145-193).  The reference formats every prompt with str.format
    (ref:llmq/core/models.py:46), so a stage-1 OUTPUT that contains a stray brace makes the stage-2
    job un-formattable: ValueError => logged + acked/dropped (ref:llmq/workers/base.py:228-235).  The quirk is replicated, not fixed: such jobs produce no final result, all
    others produce exactly the greedy continuation of their stage-1 text."""
    import json

    import aio_pika
    from llmq.core.broker import BrokerManager
    from llmq.core.models import Job, Result

    from llmq_b200.fixtures import seeded_state_dict, write_model_dir
    from llmq_b200.model import ModelSpec
    from llmq_b200.worker import B200Worker
    from oracle.model import LlamaDims, LlamaOracle

    spec = ModelSpec(hidden=512, n_layers=2, n_q_heads=8, n_kv_heads=2, head_dim=128, intermediate=1024,
                     vocab=2048, max_position_embeddings=256, name="tiny")
    mdir = write_model_dir(str(tmp_path / "tiny-llama"), spec, seed=91, with_weights=True)
    # give every 8th ordinary word of the vocabulary a stray closing brace: "w13" -> "w13}"
    tj = os.path.join(mdir, "tokenizer.json")
    t = json.load(open(tj))
    t["model"]["vocab"] = {(k + "}" if k.startswith("w") and v % 8 == 5 else k): v for k, v in t["model"]["vocab"].items()}
    json.dump(t, open(tj, "w"))
    monkeypatch.setenv("VLLM_MAX_TOKENS", "6")
    monkeypatch.setenv("VLLM_MAX_NUM_SEQS", "16")
    monkeypatch.setenv("VLLM_MAX_MODEL_LEN", "256")
    monkeypatch.setenv("B200Q_MAX_NUM_BATCHED_TOKENS", "256")
    monkeypatch.setenv("B200Q_TEMPERATURE", "0")
    aio_pika.reset_brokers()
    stages = ["translate", "format"]
    n_jobs = 40
    # remember every text either stage hands back (the stage-1 texts are otherwise only visible as
    # stage-2 prompts, and not at all when the stage-2 job is dropped)
    from llmq_b200.service import GenerationService
    produced, owner = [], {}
    detokenize_batch = GenerationService.detokenize_batch

    def recording_detokenize(self, pairs):
        texts = detokenize_batch(self, pairs)
        produced.extend((owner.get(id(self)), text) for text in texts)
        return texts

    monkeypatch.setattr(GenerationService, "detokenize_batch", recording_detokenize)

    async def main():
        # two engines share the GPU: vLLM's meaning of the knob is "this fraction of the device in total"
        monkeypatch.setenv("VLLM_GPU_MEMORY_UTILIZATION", "0.2")
        w1 = B200Worker(mdir, "pipeline.p.translate", pipeline_name="p", stage_name="translate", pipeline_stages=stages)
        monkeypatch.setenv("VLLM_GPU_MEMORY_UTILIZATION", "0.45")
        w2 = B200Worker(mdir, "pipeline.p.format", pipeline_name="p", stage_name="format", pipeline_stages=stages)
        t1 = asyncio.create_task(w1.run())
        while w1.service is None and not t1.done():
            await asyncio.sleep(0.05)
        owner[id(w1.service)] = "translate"
        t2 = asyncio.create_task(w2.run())
        while w2.service is None and not t2.done():
            await asyncio.sleep(0.05)
        owner[id(w2.service)] = "format"
        b = BrokerManager()
        await b.connect()
        await b.setup_pipeline_infrastructure("p", stages)
        for i in range(n_jobs):
            await b.publish_job("pipeline.p.translate", Job(id=f"p{i}", prompt=f"w{20 + 3 * i} w6 w7", src=f"s{i}"))
        got = {}

        async def on_res(m):
            r = Result.parse_raw(m.body)
            got[r.id] = r
            await m.ack()

        await b.consume_results("pipeline.p.results", on_res)
        # stage 1 finishes every job; stage 2 finishes or drops (un-formattable prompt) each of them:
        # wait until stage 1 is through and the number of final results has been stable for a second
        stable, last = 0, -1
        for _ in range(1200):
            if w1.jobs_processed >= n_jobs:
                stable = stable + 1 if len(got) == last else 0
                last = len(got)
                if stable >= 20:
                    break
            await asyncio.sleep(0.05)
        assert w1.jobs_processed >= n_jobs
        tok = w1.service.tokenizer
        w1.running = w2.running = False
        await asyncio.wait_for(asyncio.gather(t1, t2), 60)
        return got, tok

    got, tok = asyncio.run(main())
    stage1_texts = [t for svc, t in produced if svc == "translate"]
    assert len(stage1_texts) == n_jobs
    with_brace = [t for t in stage1_texts if "}" in t or "{" in t]
    formattable = [t for t in stage1_texts if t not in with_brace]
    assert len(with_brace) >= 5 and len(formattable) >= 5, (len(with_brace), len(formattable))
    # every formattable stage-1 text became a stage-2 prompt and produced a final result; none of the others did
    assert sorted(r.prompt for r in got.values()) == sorted(formattable)
    assert all("}" not in r.prompt for r in got.values())
    assert all(r.model_dump()["src"] == f"s{r.id[1:]}" for r in got.values())   # extras ride along both hops
    # and the final text is the model's greedy continuation of the stage-2 prompt (oracle, near-tie rule)
    oracle = LlamaOracle(LlamaDims.from_hf_config(spec.to_hf_config()), seeded_state_dict(spec, 91), "bf16", max_pos=256)
    n_exact = 0
    sample = sorted(got.values(), key=lambda r: r.id)[:10]
    for r in sample:
        ids = tok(r.prompt, add_special_tokens=True).input_ids
        ref, lg = oracle.greedy(ids, 6, eos_id=tok.eos_token_id, return_logits=True)
        if tok.eos_token_id in ref:
            ref = ref[: ref.index(tok.eos_token_id)]
        want = tok.decode(ids + ref, skip_special_tokens=True)[len(tok.decode(ids, skip_special_tokens=True)):]
        if r.result == want:
            n_exact += 1
        else:
            assert any((l.topk(2).values[0] - l.topk(2).values[1]).item() < 0.12 for l in lg), (r.id, r.result, want)
    # (stage-2 prompts are 6 model-generated tokens, often repetitive: this tiny model's top-2 margins
    # there are mostly below the tolerance, so identical texts are the exception — numerics are pinned
    # by the other worker tests; this one is about routing and the brace quirk)
    assert n_exact >= 1, (n_exact, len(sample))
