"""Kernels begin while the one before them on the stream still runs (csrc/common.cuh: launch_early, follow_previous): what the one before
writes, weights included, has to be what the next one reads, back to back, on a stream of its own and in a graph."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def chain(lib, st, gap):
    """every kernel reads, as activations, weights or rows, what the one before it wrote; `gap()` is called between all of them"""
    lib.gather_rows(st["w_src"], st["rows_w"], st["w"])      # the weights of the product behind it
    gap()
    lib.gemm_bf16(st["a"], st["w"], st["c"])
    gap()
    lib.rmsnorm(st["c"], st["norm"], st["y"], 1e-5)
    gap()
    lib.gemm_swiglu_bf16(st["y"], st["gate_up"], st["act"])
    gap()
    lib.gather_rows(st["act"], st["rows"], st["a"])          # activations of the next round: the buffer the first product read
    gap()
    lib.gemm_bf16(st["a"], st["w"], st["c"])
    gap()
    lib.add_rmsnorm(st["c"], st["residual"], st["norm"], 1e-5)
    gap()
    lib.gemm_bf16(st["c"], st["vocab"], st["logits"])
    gap()
    lib.argmax_bf16(st["logits"], st["ids"])
    gap()
    lib.sample_bf16(st["logits"], st["params"], st["ids2"])
    gap()
    lib.embed(st["ids"], st["vocab"], st["a"])
    gap()


def state(cuda, M, K):
    g = torch.Generator(device=cuda).manual_seed(M * K)
    rnd = lambda *s, scale=1.0: (torch.randn(*s, generator=g, device=cuda) * scale).to(BF)
    N = K
    st = {"w_src": rnd(N, K, scale=K ** -0.5), "rows_w": torch.randperm(N, generator=g, device=cuda).to(torch.int32), "w": rnd(N, K),
          "a": rnd(M, K), "c": rnd(M, N), "norm": rnd(N), "y": rnd(M, N), "gate_up": rnd(2 * N, N, scale=N ** -0.5), "act": rnd(M, N),
          "rows": torch.arange(M - 1, -1, -1, device=cuda, dtype=torch.int32), "residual": rnd(M, N), "vocab": rnd(4096, N, scale=N ** -0.5),
          "logits": rnd(M, 4096), "ids": torch.zeros(M, dtype=torch.int32, device=cuda), "ids2": torch.zeros(M, dtype=torch.int32, device=cuda)}
    p = torch.zeros(M, 4, dtype=torch.int32)
    p[:, 0] = torch.tensor([0.7]).view(torch.int32)
    p[:, 1] = torch.arange(M)
    st["params"] = p.to(cuda)
    return st


def back_to_back_is_one_by_one(cuda, lib, chain, state, how, rounds=6, any_order=()):
    """chain(lib, state, round, gap); round changes what the chain reads first, two ways in turn"""
    ref, st = state(), state()
    for r in range(rounds):
        chain(lib, ref, r, torch.cuda.synchronize)
    torch.cuda.synchronize()
    if how == "default stream":
        for r in range(rounds):
            chain(lib, st, r, lambda: None)
    else:
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        if how == "own stream":
            with torch.cuda.stream(s):
                for r in range(rounds):
                    chain(lib, st, r, lambda: None)
        else:
            keep = {k: v.clone() for k, v in st.items()}
            with torch.cuda.stream(s):
                chain(lib, st, 0, lambda: None)     # (kernel attributes and scratch, once)
            torch.cuda.synchronize()
            for k, v in keep.items():
                st[k].copy_(v)
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=s):
                for r in range(2):
                    chain(lib, st, r, lambda: None)
            for _ in range(rounds // 2):
                graph.replay()
    torch.cuda.synchronize()
    for k in ref:
        assert k in any_order or torch.equal(ref[k].view(torch.uint8), st[k].view(torch.uint8)), k


HOW = ["default stream", "own stream", "graph"]


@pytest.mark.parametrize("how", HOW)
@pytest.mark.parametrize("M,K", [(1, 1024), (48, 2048), (128, 1024), (300, 2048)])
def test_back_to_back_is_one_by_one(cuda, M, K, how):
    from llmq_b200 import lib
    back_to_back_is_one_by_one(cuda, lib, lambda lib, st, r, gap: chain(lib, st, gap), lambda: state(cuda, M, K), how)


def copy(lib, src, dst):
    """any 4-byte values, by a kernel that begins early"""
    lib.check(lib.load().b200q_copy_f32(src.data_ptr(), dst.data_ptr(), dst.numel(), lib._stream()))


def layer_state(cuda, T, gemma):
    g = torch.Generator(device=cuda).manual_seed(T)
    rnd = lambda *s, scale=1.0: (torch.randn(*s, generator=g, device=cuda) * scale).to(BF)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=cuda)
    H, n_q, n_kv, D = (2048, 8, 4, 256) if gemma else (2048, 32, 8, 64)
    I, Q, R = 4096, n_q * D, (n_q + 2 * n_kv) * D
    order = [torch.randperm(4 * T, generator=torch.Generator().manual_seed(i)).tolist() for i in range(2)]
    st = {"a": rnd(T, H), "qkv_w": rnd(R, H, scale=H ** -0.5), "qkv": torch.zeros(T, R, dtype=BF, device=cuda), "rot": rnd(64, D),
          "kv": rnd(4 * T, 2, n_kv, 16, D), "dec": torch.zeros(T, Q, dtype=BF, device=cuda), "pre": torch.zeros(T, Q, dtype=BF, device=cuda),
          "o_w": rnd(H, Q, scale=Q ** -0.5), "y": torch.zeros(T, H, dtype=BF, device=cuda), "residual": rnd(T, H), "norm": rnd(H, scale=0.1),
          "gu_w": rnd(2 * I, H, scale=H ** -0.5), "gu": torch.zeros(T, 2 * I, dtype=BF, device=cuda),
          "act": torch.zeros(T, I, dtype=BF, device=cuda), "down_w": rnd(H, I, scale=I ** -0.5)}
    for name in ("pos", "slot", "bt", "ctx", "tiles"):
        rows = []
        for r in range(2):   # two sets of tables, both whole: pages of every sequence lie elsewhere, contexts differ
            pages = [order[r][4 * t:4 * t + 4] for t in range(T)]
            pos = [(7 * t + 11 * r) % 48 for t in range(T)]
            rows.append({"pos": pos, "slot": [pages[t][p // 16] * 16 + p % 16 for t, p in enumerate(pos)], "bt": pages,
                         "ctx": [p + 1 for p in pos],
                         "tiles": [[i, 16 * i, min(16, T - 16 * i), (5 * i + 3 * r) % 32] for i in range((T + 15) // 16)]}[name])
        st[name + "_src"] = ints(rows)
        st[name] = ints(rows[0])
    return st


def layer_chain(gemma):
    n_q, n_kv, D = (8, 4, 256) if gemma else (32, 8, 64)

    def chain(lib, st, r, gap):
        for name in ("pos", "slot", "bt", "ctx", "tiles"):
            copy(lib, st[name + "_src"][r % 2], st[name])
            gap()
        part, splits = lib.gemm_bf16_splitk(st["a"], st["qkv_w"])
        gap()
        if splits > 1:
            lib.rope_kvwrite_splitk(st["qkv"], part, splits, st["rot"], st["pos"], st["slot"], st["kv"], n_q, n_kv, D, 16)
        else:
            lib.gemm_bf16(st["a"], st["qkv_w"], st["qkv"])
            gap()
            lib.rope_kvwrite(st["qkv"], st["rot"], st["pos"], st["slot"], st["kv"], n_q, n_kv, D, 16)
        gap()
        options = {"softcap": 50.0, "window": 32} if gemma else {}
        lib.decode_attn(st["qkv"], st["dec"], st["kv"], st["bt"], st["ctx"], n_q, n_kv, D, 16, D ** -0.5, **options)
        gap()
        lib.prefill_attn(st["qkv"], st["pre"], st["kv"], st["bt"], st["tiles"], n_q, n_kv, D, 16, D ** -0.5, **options)
        gap()
        lib.gemm_bf16(st["dec"], st["o_w"], st["y"])
        gap()
        if gemma:
            lib.gemma_norm_add_norm(st["y"], st["residual"], st["norm"], st["norm"], 1e-6)
            gap()
            lib.gemm_geglu_bf16(st["y"], st["gu_w"], st["act"])
        else:
            lib.add_rmsnorm(st["y"], st["residual"], st["norm"], 1e-5)
            gap()
            lib.gemm_bf16(st["y"], st["gu_w"], st["gu"])
            gap()
            lib.swiglu(st["gu"], st["act"])
        gap()
        lib.gemm_bf16(st["act"], st["down_w"], st["a"])      # 200 rows: parts and their sum
        gap()
        if gemma:
            lib.softcap_bf16(st["a"], 30.0)
            gap()
            lib.gemma_rmsnorm(st["a"], st["norm"], st["a"], 1e-6)
            gap()
    return chain


@pytest.mark.parametrize("how", HOW)
@pytest.mark.parametrize("T", [1, 48, 200, 300])
@pytest.mark.parametrize("gemma", [False, True])
def test_layers_back_to_back(cuda, T, gemma, how):
    """tables, parts, cached rows and activations, each written by the kernel before the one that reads it"""
    from llmq_b200 import lib
    back_to_back_is_one_by_one(cuda, lib, layer_chain(gemma), lambda: layer_state(cuda, T, gemma), how)


def routed_state(cuda, T, W=512, F=256, E=16, top=4):
    g = torch.Generator(device=cuda).manual_seed(T)
    rnd = lambda *s, scale=1.0: torch.randn(*s, generator=g, device=cuda) * scale
    P = T * top
    zeros = lambda n, dtype=torch.int32: torch.zeros(n, dtype=dtype, device=cuda)
    bf = lambda *s: torch.zeros(*s, dtype=BF, device=cuda)
    return {"scores_src": rnd(2, T, E), "scores": rnd(T, E), "corr": rnd(E, scale=0.2), "h": rnd(T, W).to(BF), "x": rnd(T, W),
            "up": rnd(E * 2 * F, W, scale=W ** -0.5).to(BF), "down": rnd(E * W, F, scale=F ** -0.5).to(BF), "idx": zeros(P),
            "wts": zeros(P, torch.float32), "off": zeros(E + 1), "perm": zeros(P), "pair": zeros(P), "tab": zeros((P // 128 + E) * 4),
            "nt": zeros(1), "src": bf(P, W), "gu": bf(P, 2 * F), "act": bf(P, F), "eo": bf(P, W)}


def routed_chain(lib, st, r, gap):
    T, W = st["h"].shape
    E, P = st["corr"].numel(), st["idx"].numel()
    top, F, L = P // T, st["act"].shape[1], lib.load()
    p, s = {k: v.data_ptr() for k, v in st.items()}, lib._stream()
    copy(lib, st["scores_src"][r % 2], st["scores"])
    gap()
    lib.check(L.b200q_moe_route_gated(p["scores"], E, p["corr"], T, E, top, 4, 2, 0, p["idx"], p["wts"], p["off"], p["perm"], p["pair"],
                                      p["tab"], p["nt"], s))
    gap()
    lib.gather_rows(st["h"], st["perm"], st["src"])
    gap()
    lib.check(L.b200q_linear_grouped(p["src"], W, None, p["up"], 2 * F * W, p["gu"], 2 * F, p["off"], E, P, 2 * F, W, lib.DTYPE_BF16,
                                     p["tab"], p["nt"], s))
    gap()
    lib.check(L.b200q_silu_glu(p["gu"], p["act"], P, F, lib.DTYPE_BF16, s))
    gap()
    lib.check(L.b200q_linear_grouped(p["act"], F, None, p["down"], W * F, p["eo"], W, p["off"], E, P, W, F, lib.DTYPE_BF16, p["tab"],
                                     p["nt"], s))
    gap()
    lib.check(L.b200q_residual_add_routed(p["x"], p["eo"], p["pair"], p["idx"], p["wts"], top, E, p["h"], T, W, lib.DTYPE_BF16, s))
    gap()


@pytest.mark.parametrize("how", HOW)
@pytest.mark.parametrize("T", [1, 40, 128, 700])
def test_routed_layers_back_to_back(cuda, T, how):
    """routes, tables, gathered rows and sums, on the same buffers with other scores in every round"""
    from llmq_b200 import lib
    # (an expert's rows stand in the order in which threads took their places; sums go by choices)
    back_to_back_is_one_by_one(cuda, lib, routed_chain, lambda: routed_state(cuda, T), how,
                               any_order=("perm", "pair", "src", "gu", "act", "eo"))


@pytest.mark.parametrize("how", ["eager", "graph"])
@pytest.mark.parametrize("B", [16, 200, 300])
def test_forward_reads_weights_and_tables_that_were_just_written(cuda, B, how):
    """A pass fetches weights into shared memory and reads tables ahead of the kernels before it, but not ahead of what came before the
    pass, although that is the library's own kernels, which let the next one begin while they run.  16 rows: gemm_skinny.cu; 200: tiles of
    one CTA; 300: of pairs."""
    import ctypes as C

    from llmq_b200 import lib as L
    from tests.test_model_gpu import TINY, build
    model, _, _ = build(TINY["d128"], max_seqs=304, num_blocks=640)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=cuda)
    # (what is there before the last write is as whole as what is written: another page of the sequence, another context)
    tables = {n: (ints([[2 * i, 2 * i + 1] + [0] * 6 for i in range(B)]), ints([[2 * i + 1, 2 * i] + [0] * 6 for i in range(B)]))[n] for n in (0, 1)}
    ctx = {n: ints([1 + (i + 5 * n) % 16 for i in range(B)]) for n in (0, 1)}
    pos = [int(c) - 1 for c in ctx[0].tolist()]
    meta = {"tok": ints([3 + i for i in range(B)]), "pos": ints(pos), "slot": ints([2 * i * 16 + p for i, p in enumerate(pos)]),
            "bt": tables[0].clone(), "ctx": ctx[0].clone(), "tiles": ints([[0, 0, 0, 0]]), "rows": ints(list(range(B)))}
    model.kv.copy_(torch.randn(model.kv.shape, generator=torch.Generator(device=cuda).manual_seed(1), device=cuda).to(BF))
    kv = model.kv.clone()
    ids = torch.empty(B, dtype=torch.int32, device=cuda)
    p = {n: t.data_ptr() for n, t in meta.items()}
    batch = L.Batch(T=B, n_dec=B, n_tiles=0, n_sample=B, bt_stride=8, token_ids=p["tok"], positions=p["pos"], slot_mapping=p["slot"],
                    block_table=p["bt"], ctx_lens=p["ctx"], tiles=p["tiles"], sample_rows=p["rows"], out_ids=ids.data_ptr())
    w = next(t for t in model._keep if t.shape == (12 * 128, 512))   # the first layer's query / key / value weights
    weights = {0: w.clone(), 1: (w.float() * 0.5 + 0.01).to(BF)}
    rows = torch.arange(w.shape[0], dtype=torch.int32, device=cuda)
    logits = model.logits_view(B)

    def write_and_run(n, gap):
        for turn in (n, 1 - n, n, 1 - n, n):     # (several writers, so that the queue is full when the pass comes)
            L.gather_rows(weights[turn], rows, w)
            gap()
            copy(L, tables[turn], meta["bt"])
            gap()
            copy(L, ctx[turn], meta["ctx"])
            gap()
        L.check(model.lib.b200q_model_forward(model.handle, C.byref(batch), torch.cuda.current_stream().cuda_stream))

    want = {}
    for n in (0, 1):
        model.kv.copy_(kv)
        write_and_run(n, torch.cuda.synchronize)
        torch.cuda.synchronize()
        want[n] = logits.clone()
    assert not torch.equal(want[0], want[1])
    graphs = {}
    if how == "graph":
        for n in (0, 1):
            graphs[n] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graphs[n]):
                write_and_run(n, lambda: None)
    for i in range(20):
        n = i % 2
        model.kv.copy_(kv)
        torch.cuda.synchronize()
        busy = torch.randn(2048, 2048, device=cuda)
        for _ in range(5):
            busy = busy @ busy * 1e-3            # (launches queue up behind this)
        graphs[n].replay() if graphs else write_and_run(n, lambda: None)
        torch.cuda.synchronize()
        assert torch.equal(logits, want[n]), i
    del graphs
    model.close()


def test_rows_of_a_pass_see_each_other(cuda):
    """two tokens of one sequence in one pass: the second reads from an earlier page what the first writes in the same pass, although
    the pages are asked into L2 before that is written"""
    import ctypes as C

    from llmq_b200 import lib as L
    from tests.test_model_gpu import TINY, build
    model, _, _ = build(TINY["d64"])
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=cuda)
    ids = torch.empty(2, dtype=torch.int32, device=cuda)

    def forward(rows):   # (token, position) each, one sequence on pages 5 and 9
        n = len(rows)
        meta = {"tok": ints([t for t, _ in rows]), "pos": ints([p for _, p in rows]), "slot": ints([(5, 9)[p // 16] * 16 + p % 16 for _, p in rows]),
                "bt": ints([[5, 9] + [0] * 6] * n), "ctx": ints([p + 1 for _, p in rows]), "tiles": ints([[0, 0, 0, 0]]), "rows": ints(list(range(n)))}
        p = {k: t.data_ptr() for k, t in meta.items()}
        batch = L.Batch(T=n, n_dec=n, n_tiles=0, n_sample=n, bt_stride=8, token_ids=p["tok"], positions=p["pos"], slot_mapping=p["slot"],
                        block_table=p["bt"], ctx_lens=p["ctx"], tiles=p["tiles"], sample_rows=p["rows"], out_ids=ids.data_ptr())
        L.check(model.lib.b200q_model_forward(model.handle, C.byref(batch), torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        return model.logits_view(n).float().clone()

    g = torch.Generator(device=cuda).manual_seed(3)
    model.kv.copy_(torch.randn(model.kv.shape, generator=g, device=cuda).to(BF))
    keep = model.kv.clone()
    forward([(17, 15)])
    want = forward([(40, 16)])[0]
    for _ in range(5):
        model.kv.copy_(keep)
        model.kv[:, 5, :, :, 15] = 30.0     # (what is read if the first token's row is not waited for)
        got = forward([(17, 15), (40, 16)])[1]
        # one row or two: the same kernels and orders of sums
        assert torch.equal(got, want)
    model.close()


def test_calls_go_to_the_current_stream(cuda):
    """of the thread that calls, inside and outside of a stream context"""
    import threading

    from llmq_b200 import lib
    assert lib._stream() == torch.cuda.current_stream().cuda_stream
    s, other, seen = torch.cuda.Stream(), torch.cuda.Stream(), {}

    def look():
        with torch.cuda.stream(other):
            seen["there"] = lib._stream()
        seen["outside"] = lib._stream()

    with torch.cuda.stream(s):
        assert lib._stream() == s.cuda_stream != 0
        t = threading.Thread(target=look)
        t.start()
        t.join()
    assert seen == {"there": other.cuda_stream, "outside": torch.cuda.default_stream().cuda_stream}
    assert lib._stream() == torch.cuda.current_stream().cuda_stream and lib._stream(s) == s.cuda_stream
