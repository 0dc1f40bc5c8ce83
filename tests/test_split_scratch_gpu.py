"""Parts of split reductions (csrc/gemm_tcgen05.cu: splitk_scratch) belong to whoever orders the products: a stream, a captured graph, a
model.  Nobody else's product may overwrite them before they are added."""
import ctypes as C
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16
M, N, K = 48, 2048, 2048   # parts of five splits or so (gemm_skinny.cu); 200 rows take the other kernel


def rnd(cuda, *shape, seed, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator(device=cuda).manual_seed(seed), device=cuda) * scale).to(BF)


def operands(cuda, seed, rows=M, K=K):
    return rnd(cuda, rows, K, seed=seed), rnd(cuda, N, K, seed=seed + 1, scale=K ** -0.5)


def parts_of(a, w):
    from llmq_b200 import lib
    ptr, splits = lib.gemm_bf16_splitk(a, w)
    assert splits > 1
    return ptr, splits


def added(cuda, ptr, splits, rows=M):
    """bf16 sums of the parts at ptr, by the kernel that a pass uses (norm weights of one over a residual of zero: residual = sum)"""
    from llmq_b200 import lib
    x, r = torch.empty(rows, N, dtype=BF, device=cuda), torch.zeros(rows, N, dtype=BF, device=cuda)
    lib.add_rmsnorm_splitk(x, r, torch.ones(N, dtype=BF, device=cuda), ptr, splits, 1e-5)
    return r


def test_a_stream_keeps_its_parts(cuda):
    from llmq_b200 import lib
    a, w = operands(cuda, 1)
    b, v = operands(cuda, 7)
    want = torch.empty(M, N, dtype=BF, device=cuda)
    lib.gemm_bf16(a, w, want)
    s, t = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        mine = parts_of(a, w)
    torch.cuda.synchronize()
    with torch.cuda.stream(t):
        other = parts_of(b, v)
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        got = added(cuda, *mine)
        assert parts_of(a, w) == mine   # and the place stays the same
    torch.cuda.synchronize()
    assert other[0] != mine[0]
    assert torch.equal(got, want)


@pytest.mark.parametrize("rows", [200, 256])
def test_streams_and_threads_side_by_side(cuda, rows):
    from llmq_b200 import lib
    sets = [operands(cuda, 10 * i, rows, 8192) for i in range(3)]
    want = []
    for a, w in sets:
        c = torch.empty(rows, N, dtype=BF, device=cuda)
        lib.gemm_bf16(a, w, c)
        want.append(c)
    torch.cuda.synchronize()
    bad = []

    def work(i, stream):
        a, w = sets[i]
        with torch.cuda.stream(stream):
            outs = [torch.empty(rows, N, dtype=BF, device=cuda) for _ in range(40)]
            for c in outs:
                lib.gemm_bf16(a, w, c)
            stream.synchronize()
            bad.extend((i, k) for k, c in enumerate(outs) if not torch.equal(c, want[i]))

    shared = torch.cuda.Stream()
    for streams in ([torch.cuda.Stream() for _ in range(3)], [shared] * 3):   # a stream each; all on one
        torch.cuda.synchronize()
        ts = [threading.Thread(target=work, args=(i, s)) for i, s in enumerate(streams)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
    assert not bad, bad


def test_a_graph_has_its_own_and_gives_it_back(cuda):
    from llmq_b200 import lib
    a, w = operands(cuda, 3)
    want = torch.empty(M, N, dtype=BF, device=cuda)
    lib.gemm_bf16(a, w, want)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        eager = parts_of(a, w)
    torch.cuda.synchronize()
    seen = []
    for _ in range(3):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            mine = parts_of(a, w)
            again = parts_of(a, w)
        assert mine[0] != eager[0] and again == mine
        seen.append(mine[0])
        g.replay()
        torch.cuda.synchronize()
        with torch.cuda.stream(s):
            parts_of(*operands(cuda, 5))
        torch.cuda.synchronize()
        assert torch.equal(added(cuda, *mine), want)
        del g
        torch.cuda.synchronize()
    assert len(set(seen)) < 3, "a graph that is gone gives its place to the next"


def test_two_graphs_of_one_capture_stream(cuda):
    """torch captures all graphs on one stream; their replays may run side by side"""
    from llmq_b200 import lib
    sets = [operands(cuda, 20 + 2 * i, 200, 8192) for i in range(2)]
    outs, want, graphs, cap = [], [], [], torch.cuda.Stream()
    for a, w in sets:
        c = torch.empty(200, N, dtype=BF, device=cuda)
        lib.gemm_bf16(a, w, c)
        want.append(c.clone())
        outs.append(c)
    torch.cuda.synchronize()
    for (a, w), c in zip(sets, outs):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=cap):
            for _ in range(10):
                lib.gemm_bf16(a, w, c)
        graphs.append(g)
    streams = [torch.cuda.Stream() for _ in graphs]
    for _ in range(10):
        for g, s in zip(graphs, streams):
            with torch.cuda.stream(s):
                g.replay()
        torch.cuda.synchronize()
        for c, x in zip(outs, want):
            assert torch.equal(c, x)


def test_a_pass_leaves_the_streams_parts_alone(cuda):
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
    a, w = operands(cuda, 31)
    want = torch.empty(M, N, dtype=BF, device=cuda)
    L.gemm_bf16(a, w, want)
    mine = parts_of(a, w)
    L.check(model.lib.b200q_model_forward(model.handle, C.byref(batch), torch.cuda.current_stream().cuda_stream))
    assert torch.equal(added(cuda, *mine), want)
    model.close()


def test_streams_come_and_go(cuda):
    """a stream per request: torch hands out the same few handles again and again, and each keeps its place"""
    from llmq_b200 import lib
    sets = [operands(cuda, 40), operands(cuda, 42)]
    refs = []
    for a, w in sets:
        refs.append(torch.empty(M, N, dtype=BF, device=cuda))
        lib.gemm_bf16(a, w, refs[-1])
    torch.cuda.synchronize()
    place = {}
    for i in range(100):
        s = torch.cuda.Stream(priority=-(i % 2))
        with torch.cuda.stream(s):
            ptr, splits = parts_of(*sets[i % 2])
            assert place.setdefault(s.cuda_stream, ptr) == ptr
            r = added(cuda, ptr, splits)
        s.synchronize()
        assert torch.equal(r, refs[i % 2])
    assert len(set(place.values())) == len(place)
