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


@pytest.mark.parametrize("how", ["default stream", "own stream", "graph"])
@pytest.mark.parametrize("M,K", [(1, 1024), (48, 2048), (128, 1024), (300, 2048)])
def test_back_to_back_is_one_by_one(cuda, M, K, how):
    from llmq_b200 import lib
    ref, st = state(cuda, M, K), state(cuda, M, K)
    rounds = 6
    for _ in range(rounds):
        chain(lib, ref, torch.cuda.synchronize)
    torch.cuda.synchronize()
    if how == "default stream":
        for _ in range(rounds):
            chain(lib, st, lambda: None)
    else:
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        if how == "own stream":
            with torch.cuda.stream(s):
                for _ in range(rounds):
                    chain(lib, st, lambda: None)
        else:
            keep = {k: v.clone() for k, v in st.items()}
            with torch.cuda.stream(s):
                chain(lib, st, lambda: None)     # (kernel attributes and scratch, once)
            torch.cuda.synchronize()
            for k, v in keep.items():
                st[k].copy_(v)
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=s):
                for _ in range(2):
                    chain(lib, st, lambda: None)
            for _ in range(rounds // 2):
                graph.replay()
    torch.cuda.synchronize()
    for k in ref:
        assert torch.equal(ref[k], st[k]), k


def test_forward_reads_weights_that_were_just_written(cuda):
    """a pass fetches weights ahead of the kernels before it, but not ahead of what came before the pass"""
    import ctypes as C

    from llmq_b200 import lib as L
    from tests.test_model_gpu import TINY, build
    model, _, _ = build(TINY["d128"])
    B = 16
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=cuda)
    meta = {"tok": ints([3 + i for i in range(B)]), "pos": ints([0] * B), "slot": ints([16 * i for i in range(B)]),
            "bt": ints([[i] * 8 for i in range(B)]), "ctx": ints([1] * B), "tiles": ints([[0, 0, 0, 0]]), "rows": ints(list(range(B)))}
    ids = torch.empty(B, dtype=torch.int32, device=cuda)
    p = {n: t.data_ptr() for n, t in meta.items()}
    batch = L.Batch(T=B, n_dec=B, n_tiles=0, n_sample=B, bt_stride=8, token_ids=p["tok"], positions=p["pos"], slot_mapping=p["slot"],
                    block_table=p["bt"], ctx_lens=p["ctx"], tiles=p["tiles"], sample_rows=p["rows"], out_ids=ids.data_ptr())

    def forward():
        L.check(model.lib.b200q_model_forward(model.handle, C.byref(batch), torch.cuda.current_stream().cuda_stream))

    w = next(t for t in model._keep if t.shape == (12 * 128, 512))   # the first layer's query / key / value weights
    a, b = w.clone(), (w.float() * 0.5 + 0.01).to(BF)
    logits = model.logits_view(B)
    want = {}
    for name, v in (("a", a), ("b", b)):
        w.copy_(v)
        torch.cuda.synchronize()
        forward()
        torch.cuda.synchronize()
        want[name] = logits.clone()
    assert not torch.equal(want["a"], want["b"])
    for i in range(20):
        name, v = (("a", a), ("b", b))[i % 2]
        w.copy_(v)
        forward()
        assert torch.equal(logits, want[name]), i
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
