"""Single-token attention whose pages are shared by a cluster of CTAs (csrc/attn.cu: few sequences, block tables wide enough for long
contexts) against a plain fp64 form: contexts shorter than the number of warps' pages, at page edges, windows that leave warps without
pages, soft caps, every number of CTAs per sequence."""
import pytest
import torch

from tests.test_prefill_attn_gpu import BF, BS, make_cache, reference
from tests.util import bf16_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,n_q,n_kv", [(64, 8, 2), (128, 8, 1), (256, 4, 2)])
@pytest.mark.parametrize("ctxs", [[5000], [1, 16, 17, 640], [333, 2049, 65], [700] * 9, list(range(100, 2000, 70)), list(range(1, 74))])
@pytest.mark.parametrize("cap,window", [(0.0, 0), (20.0, 100), (0.0, 1000)])
def test_shared_pages(cuda, D, n_q, n_kv, ctxs, cap, window):
    from llmq_b200 import lib
    kv, bt, rows = make_cache(ctxs, n_kv, D, seed=len(ctxs), wide=True)
    wide = torch.zeros(len(ctxs), max(bt.shape[1], 160), dtype=torch.int32)   # 160 columns: up to 8 CTAs of 4 warps and 4 pages each
    wide[:, : bt.shape[1]] = bt
    B = len(ctxs)
    qkv = torch.randn(B, (n_q + 2 * n_kv) * D, generator=torch.Generator().manual_seed(7)).to(BF)
    out = torch.full((B + 1, n_q * D), float("nan"), dtype=BF, device=cuda)
    lib.decode_attn(qkv.to(cuda), out, kv.to(cuda), wide.to(cuda), torch.tensor(ctxs, dtype=torch.int32, device=cuda), n_q, n_kv, D, BS,
                    D ** -0.5, softcap=cap, window=window)
    got = out.cpu()
    assert torch.isnan(got[B].float()).all()
    for i, c in enumerate(ctxs):
        q = qkv[i: i + 1, : n_q * D].view(1, n_q, D)
        ref = reference(q, *rows[i], torch.tensor([c - 1]), D ** -0.5, cap, window).to(BF)
        # probabilities are rounded to bf16 before the value product: 2^-9 each, outputs agree to ~5e-3 or 2 ulps
        bf16_close(got[i].view(1, n_q, D), ref, ulps=2.0, atol=5e-3, max_mismatch_frac=0.6, what=f"ctx {c}")


@pytest.mark.parametrize("D,n_q,n_kv", [(64, 16, 8), (128, 8, 8), (256, 16, 8)])
# dealt out over the resident warps; a warp to an item; an item to a CTA from 24 (D = 64), 40 (128) and 96 (256) columns on
@pytest.mark.parametrize("columns", [8, 9, 23, 24, 39, 40, 95, 96])
def test_many_sequences(cuda, D, n_q, n_kv, columns):
    """296 sequences and a few more: items enough for the streaming kernel, contexts of one token up to the whole table"""
    from llmq_b200 import lib
    for B, window in ((296, 0), (301, 70)):
        ctxs = [1 + (i * i * 37) % min(16 * columns, 300) for i in range(B)]
        ctxs[5] = 16 * columns
        kv, bt, rows = make_cache(ctxs, n_kv, D, seed=B, wide=False)
        assert bt.shape[1] == columns + 1
        bt = bt[:, :columns].contiguous()
        qkv = torch.randn(B, (n_q + 2 * n_kv) * D, generator=torch.Generator().manual_seed(7)).to(BF)
        out = torch.full((B + 1, n_q * D), float("nan"), dtype=BF, device=cuda)
        lib.decode_attn(qkv.to(cuda), out, kv.to(cuda), bt.to(cuda), torch.tensor(ctxs, dtype=torch.int32, device=cuda), n_q, n_kv, D, BS, D ** -0.5,
                        softcap=20.0 if window else 0.0, window=window)
        got = out.cpu()
        assert torch.isnan(got[B].float()).all()
        for i, c in enumerate(ctxs):
            ref = reference(qkv[i: i + 1, : n_q * D].view(1, n_q, D), *rows[i], torch.tensor([c - 1]), D ** -0.5, 20.0 if window else 0.0, window).to(BF)
            bf16_close(got[i].view(1, n_q, D), ref, ulps=2.0, atol=5e-3, max_mismatch_frac=0.6, what=f"ctx {c}")   # (as above)
