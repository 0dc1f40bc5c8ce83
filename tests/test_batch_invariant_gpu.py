"""B200Q_BATCH_INVARIANT=1: bit for bit, what a request gives does not depend on its batch-mates: prompt attention beside a long
sequence (which makes the block table wide) and cut into blocks elsewhere, single tokens among enough others for the streaming kernel,
products at every range of rows, an engine's tokens beside a long sequence.  The variable is read once, so the checks run in a process of their own."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.gpu
@pytest.mark.parametrize("what", ["prompts", "tokens", "products", "engine"])
def test_same_bits_whatever_the_batch(cuda, what):
    env = dict(os.environ, B200Q_BATCH_INVARIANT="1", PYTHONPATH=ROOT + os.pathsep + os.environ.get("PYTHONPATH", ""))
    r = subprocess.run([sys.executable, os.path.abspath(__file__), what], env=env, cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "equal" in r.stdout, r.stdout + r.stderr


def prompts():
    import torch
    from llmq_b200 import lib
    from tests.test_prefill_attn_gpu import BF, BS, make_cache
    for D, n_q, n_kv, cap, window in [(64, 8, 2, 0.0, 0), (128, 8, 2, 0.0, 0), (128, 8, 8, 0.0, 100), (256, 4, 2, 20.0, 0), (256, 8, 8, 20.0, 70)]:
        portions = [(0, 300), (0, 100), (40, 77), (0, 1900), (500, 130), (0, 20), (0, 9)] + [(0, 33)] * 40
        kv, bt, _ = make_cache([a + n for a, n in portions], n_kv, D, 5, False)
        kv, bt = kv.cuda(), bt.cuda()
        qkv = [torch.randn(n, (n_q + 2 * n_kv) * D, generator=torch.Generator().manual_seed(i)).to(BF).cuda()
               for i, (_, n) in enumerate(portions)]

        def run(which, columns):
            tiles, row = [], 0
            for k, i in enumerate(which):
                a, n = portions[i]
                tiles += [[k, row + j, min(16, n - j), a + j] for j in range(0, n, 16)]
                row += n
            out = torch.empty(row, n_q * D, dtype=BF, device="cuda")
            lib.prefill_attn(torch.cat([qkv[i] for i in which]), out, kv, bt[list(which), :columns].contiguous(),
                             torch.tensor(tiles, dtype=torch.int32, device="cuda"), n_q, n_kv, D, BS, 0.3, softcap=cap, window=window)
            parts, row = {}, 0
            for i in which:
                parts[i] = out[row: row + portions[i][1]].view(torch.int16)
                row += portions[i][1]
            return parts
        together, turned = run(range(len(portions)), bt.shape[1]), run([6, 5, 4, 3, 2, 1, 0], bt.shape[1])
        for i in range(7):
            alone = run([i], (sum(portions[i]) + 15) // 16)[i]
            assert torch.equal(alone, together[i]) and torch.equal(alone, turned[i]), (D, n_kv, window, portions[i])


def tokens():
    import torch
    from llmq_b200 import lib
    from tests.test_prefill_attn_gpu import BF, BS, make_cache
    for D, n_q, n_kv, cap, window in [(64, 32, 8, 0.0, 0), (128, 8, 8, 0.0, 300), (256, 16, 8, 20.0, 0)]:
        ctxs = [700, 1, 64, 130, 1500] + [40] * 395   # 400 sequences of 8 heads: the streaming kernel's range
        kv, bt, _ = make_cache(ctxs, n_kv, D, 6, False)
        kv, bt = kv.cuda(), bt.cuda()
        qkv = torch.randn(len(ctxs), (n_q + 2 * n_kv) * D, generator=torch.Generator().manual_seed(3)).to(BF).cuda()

        def run(lo, hi, columns):
            out = torch.empty(hi - lo, n_q * D, dtype=BF, device="cuda")
            lib.decode_attn(qkv[lo:hi], out, kv, bt[lo:hi, :columns].contiguous(), torch.tensor(ctxs[lo:hi], dtype=torch.int32, device="cuda"),
                            n_q, n_kv, D, BS, D ** -0.5, softcap=cap, window=window)
            return out.view(torch.int16)
        full = run(0, 400, bt.shape[1])
        for i in range(5):
            assert torch.equal(run(i, i + 1, (ctxs[i] + 15) // 16)[0], full[i]), (D, ctxs[i])
        assert torch.equal(run(0, 20, bt.shape[1]), full[:20])


def engine():
    """short prompts admitted beside a running sequence of 900 tokens and alone: the same tokens"""
    import dataclasses

    from llmq_b200.model import Engine
    from tests.test_model_gpu import TINY, build
    from tests.test_model_gpu import prompts as make
    dims = dataclasses.replace(TINY["d128"], max_pos=1024)
    model, _, _ = build(dims, max_tokens=1024)
    reqs = make(dims.vocab, [900, 30, 7, 130, 64, 16, 250], seed=3)

    def run(which):
        eng = Engine(model, max_num_seqs=8, max_num_batched_tokens=1024, eos_token_id=None)
        outs = {i: [] for i in which}
        eng.add_request(which[0], reqs[which[0]], 20 + 10 * (which[0] == 0), ignore_eos=True)
        for i in which[1:]:
            ids, toks, _ = eng.step()
            for r, t in zip(ids.tolist(), toks.tolist()):
                outs[r].append(t)
            eng.add_request(i, reqs[i], 20, ignore_eos=True)
        while eng.has_work():
            ids, toks, _ = eng.step()
            for r, t in zip(ids.tolist(), toks.tolist()):
                outs[r].append(t)
        eng.close()
        return outs
    together = run(list(range(7)))
    for i in range(7):
        assert run([i])[i] == together[i], i


def products():
    import torch
    from llmq_b200 import lib
    BF = torch.bfloat16
    g = torch.Generator(device="cuda").manual_seed(1)
    for N, K in [(2048, 4096), (4096, 2048), (512, 512), (38144, 2048)]:
        a = torch.randn(1200, K, generator=g, device="cuda").to(BF)
        w = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).to(BF)
        for f, n in ((lib.gemm_bf16, N), (lib.gemm_swiglu_bf16, N // 2)):
            rows = {}
            for M in (1, 17, 64, 65, 112, 113, 128, 129, 200, 256, 300, 700, 1200):
                c = torch.empty(M, n, dtype=BF, device="cuda")
                f(a[:M], w, c)
                rows[M] = c.view(torch.int16)
            for M, c in rows.items():
                assert torch.equal(c, rows[1200][:M]), (N, K, M)


if __name__ == "__main__":
    {"prompts": prompts, "tokens": tokens, "products": products, "engine": engine}[sys.argv[1]]()
    print("equal")
