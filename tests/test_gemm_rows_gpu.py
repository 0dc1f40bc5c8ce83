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


@pytest.fixture
def whole_sums():
    from llmq_b200 import lib
    lib.check(lib.load().b200q_gemm_set_splitk(1))
    yield
    lib.check(lib.load().b200q_gemm_set_splitk(0))


# (M, N, K, tile): one round and several of 64 to 320 rows, a last part of one row and of all, an odd number of blocks of 128 columns, the first
# row count of large vocabularies
@pytest.mark.parametrize("M,N,K,tile", [(300, 2304, 9216, 64), (257, 4096, 14336, 96), (513, 3584, 8192, 128), (513, 4096, 14336, 160),
                                        (300, 8192, 3584, 160), (129, 38016, 2048, 160), (352, 8192, 3584, 192), (900, 3584, 8192, 192),
                                        (1024, 3584, 14336, 224), (450, 8832, 2048, 256), (300, 15104, 2048, 320), (1600, 3584, 14336, 320),
                                        (1700, 3712, 9216, 192), (65, 38400, 2048, 96), (128, 38016, 2048, 128), (65, 128256, 4096, 96),
                                        (1537, 4096, 14336, 192)])
def test_plain(cuda, M, N, K, tile, whole_sums):
    from llmq_b200 import lib
    assert lib.load().b200q_gemm_rows_tile(M, N, K) == tile and lib.load().b200q_gemm_rows_splits(M, N, K) == 1
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


# parts of K: all counts, uneven ones, one round and two, a last part of a few rows, an odd number of blocks of 128 columns, rows of one tile
@pytest.mark.parametrize("M,N,K,tile,splits", [(129, 128, 2048, 64, 4), (768, 384, 14336, 64, 2), (257, 128, 4160, 64, 5), (130, 1024, 4160, 64, 5),
                                               (257, 1024, 4160, 96, 5), (400, 1024, 4160, 96, 3), (300, 2048, 4160, 128, 3),
                                               (256, 4096, 4096, 128, 2), (256, 4096, 14336, 256, 4), (129, 7168, 14336, 160, 4), (513, 2304, 8192, 160, 2),
                                               (161, 3712, 9216, 192, 4), (161, 6144, 9216, 192, 3), (225, 3712, 14336, 256, 4),
                                               (256, 3584, 14336, 256, 5), (300, 5120, 14336, 320, 3), (193, 3584, 8192, 224, 5),
                                               (129, 2048, 28672, 160, 8)])
def test_parts(cuda, M, N, K, tile, splits):
    from llmq_b200 import lib
    L = lib.load()
    assert (L.b200q_gemm_rows_tile(M, N, K), L.b200q_gemm_rows_splits(M, N, K)) == (tile, splits)
    a, w = inputs(cuda, M, N, K)
    whole = torch.full((M + 1, N), float("nan"), dtype=BF, device=cuda)
    lib.gemm_bf16(a, w, whole[:M])
    # as above: a part's sum is shorter, and adding the parts is a rounding of fp32 each
    bf16_close(whole[:M].cpu(), (a.double() @ w.double().t()).to(BF).cpu(), ulps=1.0, atol=2e-5 + K / 16 * 2.0 ** -24, what=f"{M} x {N} x {K}")
    assert torch.isnan(whole[M]).all() and L.b200q_wait_failures() == 0
    # whoever sums the parts himself gets the same ones: with a residual of zeros the sum itself is what add + norm leaves there
    part, n = lib.gemm_bf16_splitk(a, w)
    assert n == splits
    y, res = torch.empty(M, N, dtype=BF, device=cuda), torch.zeros(M, N, dtype=BF, device=cuda)
    lib.add_rmsnorm_splitk(y, res, torch.ones(N, dtype=BF, device=cuda), part, n, 1e-5)
    assert torch.equal(res, whole[:M])


def test_what_the_rule_leaves_alone(cuda):
    """few rows, columns that are no multiple of 128, hooks"""
    from llmq_b200 import lib
    rows = lib.load().b200q_gemm_rows_tile
    assert [rows(*x) for x in ((64, 128256, 2048), (128, 4096, 4096), (300, 8256, 3584), (1024, 9600, 6400))] == [0] * 4
    lib.gemm_set_mode(1)
    try:
        assert rows(300, 8192, 3584) == 0
    finally:
        lib.gemm_set_mode(0)


@pytest.mark.parametrize("M,N,K,parts", [(193, 1024, 5120, 8), (256, 1024, 14336, 8), (256, 2048, 2560, 4), (200, 2048, 7168, 4)])
def test_parts_that_stay_with_tiles_of_128_rows(cuda, M, N, K, parts):
    """128 CTAs of tiles and parts: the first and last row count, the shortest and longest parts; their neighbours go to the tiles above"""
    from llmq_b200 import lib
    L = lib.load()
    assert L.b200q_gemm_rows_tile(M, N, K) == 0
    assert L.b200q_gemm_rows_tile(192, N, K) > 0 and L.b200q_gemm_rows_tile(200, 2048, 64 * 4 * 29) > 0
    a, w = inputs(cuda, M, N, K)
    whole = torch.full((M + 1, N), float("nan"), dtype=BF, device=cuda)
    lib.gemm_bf16(a, w, whole[:M])
    # (as in test_parts)
    bf16_close(whole[:M].cpu(), (a.double() @ w.double().t()).to(BF).cpu(), ulps=1.0, atol=2e-5 + K / 16 * 2.0 ** -24, what=f"{M} x {N} x {K}")
    assert torch.isnan(whole[M]).all() and L.b200q_wait_failures() == 0
    part, n = lib.gemm_bf16_splitk(a, w)
    assert n == parts
    y, res = torch.empty(M, N, dtype=BF, device=cuda), torch.zeros(M, N, dtype=BF, device=cuda)
    lib.add_rmsnorm_splitk(y, res, torch.ones(N, dtype=BF, device=cuda), part, n, 1e-5)
    assert torch.equal(res, whole[:M])
