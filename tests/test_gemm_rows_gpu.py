"""Products in tiles of any multiple of 32 rows (csrc/gemm_rows.cu): the rule that takes them, every width of tile, rows and columns at the
edges of tiles, of pairs of blocks and of the 32 x 64 boxes in which C leaves, against 64 bits and against the other tile kernels, which add in
the same order."""
import pytest
import torch

from oracle import ops as O
from tests.util import bf16_close

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def inputs(cuda, M, N, K):
    g = torch.Generator(device=cuda).manual_seed(M + N + K)
    return torch.randn(M, K, generator=g, device=cuda).to(BF), (torch.randn(N, K, generator=g, device=cuda) * K ** -0.5).to(BF)


# (M, N, K, tile): one round and several of 64 to 384 rows, a last part of one row and of all, an odd number of blocks of 128 columns
@pytest.mark.parametrize("M,N,K,tile", [(300, 2304, 9216, 64), (257, 4096, 14336, 96), (513, 3584, 8192, 128), (513, 4096, 14336, 160),
                                        (300, 8192, 3584, 160), (129, 38016, 2048, 160), (352, 8192, 3584, 192), (900, 3584, 8192, 192),
                                        (1024, 3584, 14336, 224), (450, 8832, 2048, 256), (300, 15104, 2048, 320), (1600, 3584, 14336, 320),
                                        (1700, 3712, 9216, 192), (65, 38400, 2048, 96), (128, 38016, 2048, 128), (1537, 4096, 14336, 192)])
def test_plain(cuda, M, N, K, tile):
    from llmq_b200 import lib
    assert lib.load().b200q_gemm_rows_tile(M, N, K) == tile
    a, w = inputs(cuda, M, N, K)
    whole = torch.full((M + 1, N), float("nan"), dtype=BF, device=cuda)
    lib.gemm_bf16(a, w, whole[:M])
    # sums of K products of size K^-1/2, 16 at a time into an fp32 accumulator of size 1 that the tensor core cuts off: K / 16 x 2^-24,
    # beside 1e-7 for every other rounding of a sum of 200 terms, and a rounding of the result either way
    bf16_close(whole[:M].cpu(), (a.double() @ w.double().t()).to(BF).cpu(), ulps=1.0, atol=2e-5 + K / 16 * 2.0 ** -24, what=f"{M} x {N} x {K}")
    assert torch.isnan(whole[M]).all() and lib.load().b200q_wait_failures() == 0
    other = torch.empty(M, N, dtype=BF, device=cuda)
    lib.gemm_set_mode(1)
    try:
        lib.gemm_bf16(a, w, other)
    finally:
        lib.gemm_set_mode(0)
    assert torch.equal(other, whole[:M])


def test_what_the_rule_leaves_alone(cuda):
    """few rows, split reductions, columns that are no multiple of 128, hooks"""
    from llmq_b200 import lib
    rows = lib.load().b200q_gemm_rows_tile
    assert [rows(*x) for x in ((64, 128256, 2048), (128, 4096, 4096), (200, 4096, 14336), (300, 8256, 3584), (256, 4096, 2048), (1024, 9600, 6400))] == [0] * 6
    lib.gemm_set_mode(1)
    try:
        assert rows(300, 8192, 3584) == 0
    finally:
        lib.gemm_set_mode(0)
