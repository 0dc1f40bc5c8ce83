"""Products of up to 128 rows (csrc/gemm_skinny.cu) where they can go wrong: one row, edges of the padding of 16, the largest sizes
of each plan, reductions of one k-block and odd numbers of them, tiles that are split over clusters and tiles that are not."""
import math

import pytest
import torch

from tests.util import bf16_close

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def rnd(cuda, *shape, seed, scale=1.0):
    g = torch.Generator(device=cuda).manual_seed(seed)
    return (torch.randn(*shape, generator=g, device=cuda) * scale).to(BF)


SHAPES = [(128, 64), (256, 192), (384, 576), (2048, 8192), (4096, 4160), (38144, 128)]


@pytest.mark.parametrize("M", [1, 8, 9, 16, 17, 64, 65, 112, 113, 128])
@pytest.mark.parametrize("N,K", SHAPES)
def test_plain(cuda, M, N, K):
    from llmq_b200 import lib
    a, w = rnd(cuda, M, K, seed=M), rnd(cuda, N, K, seed=N + K, scale=K ** -0.5)
    c = torch.full((M + 1, N), float("nan"), dtype=BF, device=cuda)
    lib.gemm_bf16(a, w, c[:M])
    ref = (a.double() @ w.double().t()).to(BF)
    # sums of K products of size K^-1/2 in fp32: order of summation moves them by about 1e-7 sqrt(K) K^-1/2, a rounding either way
    bf16_close(c[:M].cpu(), ref.cpu(), ulps=1.0, atol=2e-5, what=f"{M} x {N} x {K}")
    assert torch.isnan(c[M]).all(), "rows behind the last one stay as they were"
    assert lib.load().b200q_wait_failures() == 0


@pytest.mark.parametrize("act", ["swiglu", "geglu", "clamped", "clamped_bias"])
@pytest.mark.parametrize("M,N,K", [(1, 256, 64), (17, 512, 320), (64, 16384, 512), (100, 2304, 1024), (112, 28672, 128), (128, 16384, 256)])
def test_gated(cuda, M, N, K, act):
    from llmq_b200 import lib
    L = lib.load()
    a, w = rnd(cuda, M, K, seed=M), rnd(cuda, N, K, seed=N + K, scale=1.5 * K ** -0.5)
    ldc = N // 2 + (8 if "clamped" in act else 0)
    c = torch.full((M, ldc), 7.0, dtype=BF, device=cuda)
    gu = (a.double() @ w.double().t()).view(M, N // 256, 2, 128)
    s = torch.cuda.current_stream().cuda_stream
    if act in ("swiglu", "geglu"):
        (lib.gemm_swiglu_bf16 if act == "swiglu" else lib.gemm_geglu_bf16)(a, w, c)
        g, u = gu.to(BF).double().unbind(2)
        g.requires_grad_()
        h = torch.nn.functional.silu(g) if act == "swiglu" else torch.nn.functional.gelu(g, approximate="tanh")
        slope, = torch.autograd.grad(h.sum(), g)
        g, h = g.detach(), h.detach()
        ref = h.to(BF).double() * u
    else:
        bias = rnd(cuda, N, seed=5).float() if act == "clamped_bias" else None
        lib.check(L.b200q_gemm_clamped_glu_bf16(a.data_ptr(), w.data_ptr(), bias.data_ptr() if bias is not None else None, c.data_ptr(),
                                                ldc, M, N, K, 1.25, s))
        if bias is not None:
            gu = gu + bias.double().view(1, N // 256, 2, 128)
        g, u = gu.unbind(2)
        g, u = g.clamp(max=1.25), u.clamp(-1.25, 1.25)
        ref, slope = g * torch.sigmoid(1.702 * g) * (u + 1), torch.zeros_like(g)
        assert (c[:, N // 2:] == 7.0).all(), "the gap between rows stays as it was"
    # a gate that rounds the other way moves the product by an ulp (2^-7 at most) of the gate times the unit's slope, the other
    # roundings (unit, up, product) by an ulp of the product each
    got, ref = c[:, : N // 2].double(), ref.reshape(M, -1)
    tol = 3 * 2.0 ** -7 * ref.abs() + 2.0 ** -7 * (g * slope * u).abs().reshape(M, -1) + 2e-5
    off = (got - ref).abs()
    assert torch.isfinite(got).all() and (off <= tol).all(), f"{act} {M} x {N} x {K}: {float((off / tol).max())}"


@pytest.mark.parametrize("M", [1, 17, 33, 65, 113, 127, 128])
@pytest.mark.parametrize("N,K", [(128, 1024), (384, 1088), (256, 768), (512, 512), (8320, 4096), (19072, 768), (37760, 1024), (38144, 1024),
                                 (65536, 4096)])
def test_plain_at_the_edges_of_the_choice(cuda, M, N, K):
    test_plain(cuda, M, N, K)


@pytest.mark.parametrize("act", ["swiglu", "clamped_bias"])
@pytest.mark.parametrize("M,N,K", [(113, 28672, 256), (127, 19456, 128), (128, 16384, 1024), (128, 512, 512)])
def test_gated_at_the_edges_of_the_choice(cuda, M, N, K, act):
    test_gated(cuda, M, N, K, act)


@pytest.mark.parametrize("M", [129, 161, 257, 384, 640])
@pytest.mark.parametrize("N,K", [(2048, 512), (512, 64)])
def test_warps_without_rows(cuda, M, N, K):
    """more than 128 rows, the last tile's warps partly or all without any: rows behind the last one stay as they were"""
    test_plain(cuda, M, N, K)
    test_gated(cuda, M, N, K, "swiglu")
    from llmq_b200 import lib
    c = torch.full((M + 130, N // 2), 7.0, dtype=BF, device=cuda)
    lib.gemm_swiglu_bf16(rnd(cuda, M, K, seed=M), rnd(cuda, N, K, seed=N + K, scale=1.5 * K ** -0.5), c[:M])
    assert (c[M:] == 7.0).all()


def give_up():
    """in a process of its own (the flag stays set): every product gives up at its first wait with copies of the ring in flight, and the
    next ones are right"""
    from llmq_b200 import lib
    L, dev = lib.load(), torch.device("cuda")
    shapes = [(1, 128, 1024), (17, 512, 4096), (64, 2048, 8192), (100, 4096, 14336), (128, 2048, 8192), (100, 38144, 4096)]
    for M, N, K in shapes:
        a, w = rnd(dev, M, K, seed=M), rnd(dev, N, K, seed=N + K, scale=K ** -0.5)
        c, ref = torch.zeros(M, N, dtype=BF, device=dev), (a.double() @ w.double().t()).to(BF)
        L.b200q_gemm_set_give_up(1)
        for _ in range(20):
            lib.gemm_bf16(a, w, c)
            if N % 256 == 0:
                lib.gemm_swiglu_bf16(a, w, torch.empty(M, N // 2, dtype=BF, device=dev))
        torch.cuda.synchronize()
        assert L.b200q_wait_failures() != 0
        L.b200q_gemm_set_give_up(0)
        lib.gemm_bf16(a, w, c)
        bf16_close(c.cpu(), ref.cpu(), ulps=1.0, atol=2e-5, what=f"{M} x {N} x {K}")
    print("right again")


def test_waits_that_run_out(cuda):
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", "from tests.test_gemm_skinny_gpu import give_up; give_up()"], cwd=root, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and "right again" in r.stdout, r.stdout + r.stderr


@pytest.mark.parametrize("M", [31, 32, 33, 48, 96, 97])
@pytest.mark.parametrize("N,K", [(2048, 2048), (512, 4096), (33024, 128), (38144, 128)])
def test_rows_at_the_edges_of_accumulator_loads(cuda, M, N, K):
    """32 rows of A leave tensor memory at a time, 16 to a load: one load, a half, none of the second; tiles of 128 and 256 weight rows"""
    test_plain(cuda, M, N, K)
    test_gated(cuda, M, N, K, "swiglu")
    test_gated(cuda, M, N, K, "clamped_bias")


@pytest.mark.parametrize("M", [1, 16, 33, 64, 128])
def test_parts_are_the_sum(cuda, M):
    """the parts of a split reduction that the next kernel adds up are those that the product itself adds"""
    import ctypes as C
    from llmq_b200 import lib
    N, K = 2048, 2048
    a, w = rnd(cuda, M, K, seed=M), rnd(cuda, N, K, seed=N + K, scale=K ** -0.5)
    ptr, splits = lib.gemm_bf16_splitk(a, w)
    assert splits > 1
    torch.cuda.synchronize()
    parts = torch.empty(splits, M, N, device=cuda)
    lib.check(lib.load().b200q_copy_f32(C.c_void_p(ptr), C.c_void_p(parts.data_ptr()), parts.numel(), torch.cuda.current_stream().cuda_stream))
    c = torch.empty(M, N, dtype=BF, device=cuda)
    lib.gemm_bf16(a, w, c)
    total = parts[0].clone()
    for s in range(1, splits):
        total += parts[s]
    assert torch.equal(total.to(BF), c)
