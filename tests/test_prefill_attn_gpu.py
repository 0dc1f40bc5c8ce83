"""Attention of prompt portions (csrc/prefill_attn.cu) against a plain fp64 form: portions at the edges of pages, of key steps and of
query tiles, behind cached tokens, several of them to a block of tiles, every group size, windows, soft caps, unaligned rows, a negative
and a zero scale; unused cache rows hold NaN."""
import math

import pytest
import torch

from oracle import ops as O
from tests.util import bf16_close

pytestmark = pytest.mark.gpu
BF = torch.bfloat16
BS = 16


def make_cache(ctxs, n_kv, D, seed, wide):
    g = torch.Generator().manual_seed(seed)
    blocks = sum((c + BS - 1) // BS for c in ctxs) + 3
    perm = torch.randperm(blocks, generator=g).tolist()
    kv = torch.zeros(blocks, 2, n_kv, BS, D, dtype=BF)
    kv.view(torch.int16)[:] = 0x7FC0
    # (a table of 40 columns and more could hold contexts that the tensor-memory kernel takes at every head size)
    bt = torch.zeros(len(ctxs), max((max(ctxs) + BS - 1) // BS + 1, 40 if wide else 0), dtype=torch.int32)
    sw = O.kv_swizzle_index(BS, D)
    rows = []
    for i, c in enumerate(ctxs):
        k, v = torch.randn(c, n_kv, D, generator=g).to(BF), torch.randn(c, n_kv, D, generator=g).to(BF)
        rows.append((k, v))
        for b in range((c + BS - 1) // BS):
            blk = perm.pop()
            bt[i, b] = blk
            n = min(BS, c - b * BS)
            for which, src in ((0, k), (1, v)):
                page = src[b * BS: b * BS + n].transpose(0, 1)                      # [n_kv, n, D]
                kv[blk, which, :, :n] = torch.zeros_like(page).scatter(2, sw[:n].expand(n_kv, n, D), page)
    return kv, bt, rows


def reference(q, k, v, pos, scale, cap, window):
    G = q.shape[1] // k.shape[1]
    kk, vv = k.double().repeat_interleave(G, 1), v.double().repeat_interleave(G, 1)
    s = torch.einsum("qhd,khd->hqk", q.double(), kk) * scale
    s = cap * torch.tanh(s / cap) if cap else s
    j = torch.arange(k.shape[0])[None]
    hide = j > pos[:, None]
    hide = hide | (j <= pos[:, None] - window) if window else hide
    return torch.einsum("hqk,khd->qhd", torch.softmax(s.masked_fill(hide[None], -math.inf), -1), vv)


def check(cuda, D, n_q, n_kv, portions, scale=None, cap=0.0, window=0, pad=0, order=None, seed=1, wide=True, more_rows=0, routes=None):
    """portions: (cached tokens, tokens of this step) per sequence; more_rows: of other sequences in the block table"""
    from llmq_b200 import lib
    scale = D ** -0.5 if scale is None else scale
    kv, bt, rows = make_cache([a + n for a, n in portions], n_kv, D, seed, wide)
    bt = torch.cat([bt, torch.zeros(more_rows, bt.shape[1], dtype=torch.int32)])
    T = sum(n for _, n in portions)
    g = torch.Generator().manual_seed(seed + 50)
    qkv = torch.randn(T, (n_q + 2 * n_kv) * D + pad, generator=g).to(BF)
    tiles, row = [], 0
    for i, (a, n) in enumerate(portions):
        tiles += [[i, row + j, min(16, n - j), a + j] for j in range(0, n, 16)]
        row += n
    if order is not None:
        tiles = order(tiles)
    t = torch.tensor(tiles, dtype=torch.int32, device=cuda)
    refs, row = [], 0
    for i, (a, n) in enumerate(portions):
        q = qkv[row: row + n, : n_q * D].view(n, n_q, D)
        refs.append(reference(q, *rows[i], torch.arange(a, a + n), scale, cap, window).to(BF))
        row += n
    for route in routes or ((-1, 1) if wide else (-1,)):   # the one that is chosen, and the tensor-memory kernel
        out = torch.full((T + 1, n_q * D), float("nan"), dtype=BF, device=cuda)
        lib.check(lib.load().b200q_prefill_attn_set_route(route))
        try:
            lib.prefill_attn(qkv.to(cuda), out, kv.to(cuda), bt.to(cuda), t, n_q, n_kv, D, BS, scale, softcap=cap, window=window)
        finally:
            lib.check(lib.load().b200q_prefill_attn_set_route(-1))
        got = out.cpu()
        assert torch.isnan(got[T].float()).all(), "rows behind the last one stay as they were"
        assert lib.load().b200q_wait_failures() == 0
        row = 0
        for i, (a, n) in enumerate(portions):
            # probabilities are rounded to bf16 before the value product: 2^-9 each, outputs agree to ~5e-3 or 2 ulps
            bf16_close(got[row: row + n].view(n, n_q, D), refs[i], ulps=2.0, atol=5e-3, max_mismatch_frac=0.6,
                       what=f"portion {i} ({a} + {n}) route {route}")
            row += n


MIX = [(0, 128), (0, 5), (16, 16), (100, 37), (3, 49), (0, 1), (0, 64), (250, 70), (0, 257), (127, 2), (0, 300)]


@pytest.mark.parametrize("D,n_q,n_kv", [(64, 32, 8), (128, 32, 8), (256, 16, 8), (64, 2, 2), (128, 6, 2), (128, 10, 2), (64, 6, 1), (128, 7, 1),
                                        (128, 8, 1), (256, 3, 3), (256, 3, 1), (256, 8, 2)])
def test_head_layouts(cuda, D, n_q, n_kv):
    check(cuda, D, n_q, n_kv, MIX)
    check(cuda, D, n_q, n_kv, MIX, wide=False, window=30)
    check(cuda, D, n_q, n_kv, MIX[:2] + [(60, 40)] * 40)          # many short runs to a block


@pytest.mark.parametrize("D,n_q,n_kv", [(64, 4, 1), (128, 8, 2), (256, 4, 2)])
@pytest.mark.parametrize("cap,window", [(0.0, 40), (20.0, 0), (20.0, 1), (5.0, 130), (50.0, 64)])
def test_caps_and_windows(cuda, D, n_q, n_kv, cap, window):
    check(cuda, D, n_q, n_kv, MIX + [(900, 150), (0, 700)], cap=cap, window=window, seed=3)


@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("kind", ["unaligned", "negative", "zero", "large", "shuffled", "reversed"])
def test_forms(cuda, D, kind):
    g = torch.Generator().manual_seed(9)
    kw = {"unaligned": dict(pad=2), "negative": dict(scale=-0.3), "zero": dict(scale=0.0), "large": dict(scale=4.0),
          "shuffled": dict(order=lambda t: [t[i] for i in torch.randperm(len(t), generator=g).tolist()]),
          "reversed": dict(order=lambda t: t[::-1])}[kind]
    check(cuda, D, 4, 1, MIX, **kw)
    if kind in ("negative", "zero"):
        check(cuda, D, 4, 1, MIX, cap=10.0, window=50, **kw)


@pytest.mark.parametrize("n", [1, 15, 16, 17, 63, 64, 65, 127, 129, 255, 256, 511, 1500])
def test_lengths(cuda, n):
    for D in (64, 128, 256):
        check(cuda, D, 8, 2, [(0, n)], seed=n)
        check(cuda, D, 4, 2, [(n, 33)], seed=n + 1)


@pytest.mark.parametrize("D,n_q,n_kv", [(64, 8, 8), (128, 16, 8), (256, 16, 8)])
@pytest.mark.parametrize("cap", [0.0, 50.0, 12.0, 2.0])     # none; arguments of tanh up to 0.1, to 0.3 and beyond: 3 terms, 5 terms, all of it
def test_many_runs_to_a_cta(cuda, D, n_q, n_kv, cap):
    """more runs than the ring between the roles holds, of 1 to 6 steps, whole query tiles and parts of them"""
    check(cuda, D, n_q, n_kv, [(17 * i % 90 if i % 3 else 0, 9 + 31 * i % 290) for i in range(220)], cap=cap, seed=5, routes=(1,))


def step(cuda, D, n_q, n_kv, portions, seed, scale, cap=0.0, window=0, wide=True, rows_of=None, k_scale=1.0):
    """one call's inputs on the GPU and the call"""
    from llmq_b200 import lib
    kv, bt, _ = make_cache([a + n for a, n in portions], n_kv, D, seed, wide)
    kv = (kv.float() * k_scale).to(BF)
    T = sum(n for _, n in portions)
    qkv = torch.randn(T, (n_q + 2 * n_kv) * D, generator=torch.Generator().manual_seed(seed)).to(BF)
    tiles, row = [], 0
    for i, (a, n) in enumerate(portions):
        tiles += [[i, row + j, min(16, n - j), a + j] for j in range(0, n, 16)]
        row += n
    dev = [x.to(cuda) for x in (qkv, kv, bt, torch.tensor(tiles, dtype=torch.int32))]

    def call():
        out = torch.empty(T, n_q * D, dtype=BF, device=cuda)
        lib.check(lib.load().b200q_prefill_attn_set_route(1))
        lib.prefill_attn(dev[0], out, dev[1], dev[2], dev[3], n_q, n_kv, D, BS, scale, softcap=cap, window=window)
        lib.check(lib.load().b200q_prefill_attn_set_route(-1))
        return out.cpu()
    return call


@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("cap,window", [(0.0, 0), (30.0, 0), (30.0, 77)])
def test_same_bits_whatever_ran_before(cuda, D, cap, window):
    """products of a soft-capped call stay below the bound up to which tanh is a short series; another call leaves large keys in shared
    memory, behind the last key of portions that do not fill a step"""
    small = step(cuda, D, 4, 2, [(0, n) for n in (700, 5, 33, 140, 257, 1, 90, 600, 301)] * 8, 21, 0.02, cap, window)
    large = step(cuda, D, 4, 2, [(0, 1024)] * 24, 22, 0.02, cap, window, k_scale=1000.0)
    small()
    first = small()
    large()
    second = small()
    assert torch.equal(first.view(torch.int16), second.view(torch.int16))
    assert torch.equal(first.view(torch.int16), small().view(torch.int16))


@pytest.mark.parametrize("D,n_q,n_kv", [(64, 4, 2), (64, 2, 2), (128, 8, 2), (128, 2, 2), (256, 4, 2), (256, 2, 2)])
@pytest.mark.parametrize("cap,window", [(0.0, 0), (20.0, 0), (0.0, 90)])
@pytest.mark.parametrize("value", [float("inf"), float("nan"), -float("inf")])
def test_values_that_are_not_finite_stay_with_those_who_see_them(cuda, D, n_q, n_kv, cap, window, value):
    """one element of a cached value row is not finite: tokens before it, and tokens whose window has passed it, get what they would"""
    from llmq_b200 import lib
    portions, bad = [(0, 1500), (300, 700), (0, 40)], {0: 1333, 1: 700}      # (sequence: token)
    kv, bt, rows = make_cache([a + n for a, n in portions], n_kv, D, 31, True)
    sw = O.kv_swizzle_index(BS, D)
    for i, t in bad.items():
        kv[bt[i, t // BS], 1, 0, t % BS, sw[t % BS, D // 3]] = value       # head 0, column D // 3
    T = sum(n for _, n in portions)
    qkv = torch.randn(T, (n_q + 2 * n_kv) * D, generator=torch.Generator().manual_seed(8)).to(BF)
    tiles, row = [], 0
    for i, (a, n) in enumerate(portions):
        tiles += [[i, row + j, min(16, n - j), a + j] for j in range(0, n, 16)]
        row += n
    out = torch.full((T + 1, n_q * D), float("nan"), dtype=BF, device=cuda)
    lib.check(lib.load().b200q_prefill_attn_set_route(1))   # (the kernel of 16-token tiles passes on what its own 16 tokens see)
    lib.prefill_attn(qkv.to(cuda), out, kv.to(cuda), bt.to(cuda), torch.tensor(tiles, dtype=torch.int32, device=cuda), n_q, n_kv, D, BS,
                     D ** -0.5, softcap=cap, window=window)
    lib.check(lib.load().b200q_prefill_attn_set_route(-1))
    got, row = out.cpu(), 0
    assert torch.isnan(got[T].float()).all() and lib.load().b200q_wait_failures() == 0
    for i, (a, n) in enumerate(portions):
        q = qkv[row: row + n, : n_q * D].view(n, n_q, D)
        ref = reference(q, *rows[i], torch.arange(a, a + n), D ** -0.5, cap, window)
        mine, pos = got[row: row + n].view(n, n_q, D), torch.arange(a, a + n)
        sees = (pos >= bad.get(i, 1 << 30)) & ((pos < bad.get(i, 0) + window) if window else True)
        touched = torch.zeros(n, n_q, D, dtype=torch.bool)
        touched[sees, : n_q // n_kv, D // 3] = True
        # (head 0's column of the tokens that see it is value itself, or NaN; everything else is as it was without it)
        assert not torch.isfinite(mine[touched].float()).any()
        bf16_close(torch.where(touched, ref.to(BF), mine), ref.to(BF), ulps=2.0, atol=5e-3, max_mismatch_frac=0.6, what=f"portion {i}")
        row += n


@pytest.mark.parametrize("D,n_q,n_kv", [(64, 8, 2), (128, 8, 2), (128, 2, 2), (128, 8, 1), (256, 4, 2), (256, 3, 3)])
@pytest.mark.parametrize("cap,window", [(0.0, 0), (20.0, 150)])
@pytest.mark.parametrize("order", ["listed", "turned", "shuffled"])
def test_portions_shared_by_both_kernels(cuda, D, n_q, n_kv, cap, window, order):
    """where the table says nothing about the portions, each is looked at on the GPU.  Portions at the edge of what counts as
    long (160, 320, 512 keys), longer than the 32 tiles that are looked at, and short ones between them"""
    g = torch.Generator().manual_seed(4)
    turn = {"listed": None, "turned": lambda t: t[::-1], "shuffled": lambda t: [t[i] for i in torch.randperm(len(t), generator=g).tolist()]}
    portions = [(0, 159), (0, 160), (0, 161), (300, 19), (300, 20), (0, 511), (480, 32), (480, 33), (0, 7), (0, 700), (900, 2), (0, 30),
                (0, 31), (3, 1100), (0, 16), (511, 1)]
    check(cuda, D, n_q, n_kv, portions, cap=cap, window=window, order=turn[order], seed=17, more_rows=300, routes=(2,))


def test_only_short_and_only_long_portions_of_a_wide_table(cuda):
    for D in (64, 128, 256):
        check(cuda, D, 8, 4, [(0, n) for n in (5, 16, 31, 40)] * 6, more_rows=300, seed=2, routes=(-1, 2))
        check(cuda, D, 8, 4, [(0, 600), (1000, 40), (0, 900)], more_rows=300, seed=3, routes=(-1, 2))


@pytest.mark.parametrize("D,n_q,n_kv", [(64, 8, 1), (128, 8, 2), (256, 8, 2)])
@pytest.mark.parametrize("stride", ["8 more", "24 more", "0", "back"])
def test_query_strides(cuda, D, n_q, n_kv, stride):
    """rows of queries that are 16-byte aligned, at any distance: no multiple of a head, the same row for every token, from the last one back"""
    from llmq_b200 import lib
    row, n = n_q * D, 200
    kv, bt, rows = make_cache([n], n_kv, D, 1, True)
    q = torch.randn(n, row + {"8 more": 8, "24 more": 24}.get(stride, 0), generator=torch.Generator().manual_seed(3)).to(BF)
    dev, used = q.to(cuda), q[:, :row]
    at, step = dev.data_ptr(), q.shape[1]
    if stride == "0":
        step, used = 0, q[:1, :row].expand(n, row)
    elif stride == "back":
        at, step, used = at + 2 * (n - 1) * step, -step, q.flip(0)
    tiles = torch.tensor([[0, j, min(16, n - j), j] for j in range(0, n, 16)], dtype=torch.int32, device=cuda)
    ref = reference(used.view(n, n_q, D), *rows[0], torch.arange(n), D ** -0.5, 0.0, 0).to(BF)
    kv, bt = kv.to(cuda), bt.to(cuda)
    for route in (0, 1):
        out = torch.empty(n, row, dtype=BF, device=cuda)
        lib.check(lib.load().b200q_prefill_attn_set_route(route))
        try:
            lib.check(lib.load().b200q_prefill_attn_seqs(at, step, out.data_ptr(), kv.data_ptr(), bt.data_ptr(), bt.shape[1], 1, tiles.data_ptr(),
                                                         tiles.shape[0], n_q, n_kv, D, BS, D ** -0.5, 0.0, 0, lib._stream()))
        finally:
            lib.check(lib.load().b200q_prefill_attn_set_route(-1))
        # (as in check)
        bf16_close(out.cpu().view(n, n_q, D), ref, ulps=2.0, atol=5e-3, max_mismatch_frac=0.6, what=f"stride {stride} route {route}")
