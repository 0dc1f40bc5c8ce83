"""Products of more than 128 rows whose rounds are filled by tiles of 160 and 192 columns (csrc/gemm_tcgen05.cu: choose_tile): every width
that a last tile of a row can have, rows at the edges of the pair's 256, one row of pair tiles and several."""
import pytest
import torch

from tests.util import bf16_close

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def check(cuda, M, N, K, width):
    from llmq_b200 import lib
    assert lib.load().b200q_gemm_tile_n(M, N) == width, (M, N)
    g = torch.Generator(device=cuda).manual_seed(M + N + K)
    a = torch.randn(M, K, generator=g, device=cuda).to(BF)
    w = (torch.randn(N, K, generator=g, device=cuda) * K ** -0.5).to(BF)
    whole = torch.full((M + 1, N), float("nan"), dtype=BF, device=cuda)
    lib.gemm_bf16(a, w, whole[:M])
    ref = (a.double() @ w.double().t()).to(BF)
    # sums of K products of size K^-1/2 in fp32: order of summation moves them by about 1e-7 sqrt(K) K^-1/2, a rounding either way
    bf16_close(whole[:M].cpu(), ref.cpu(), ulps=1.0, atol=2e-5, what=f"{M} x {N} x {K}")
    assert torch.isnan(whole[M]).all()
    # every tile kernel adds in the same order
    for bn in (64, 128):
        lib.gemm_set_tile_n(bn)
        try:
            c = torch.empty(M, N, dtype=BF, device=cuda)
            if N % bn == 0:
                assert lib.load().b200q_gemm_tile_n(M, N) == bn
                lib.gemm_bf16(a, w, c)
                assert torch.equal(c, whole[:M])
        finally:
            lib.gemm_set_tile_n(0)


# 129 to 256 rows, one row of pair tiles: 160 columns from 9472 + 64 to 74 x 160 = 11840, 192 up to 74 x 192 = 14208
@pytest.mark.parametrize("M", [129, 255, 256])
@pytest.mark.parametrize("N,width", [(9536, 160), (9600, 160), (9664, 160), (9728, 160), (9792, 160), (11840, 160),      # last tile of 96, 160, 64, 128, 32, 160
                                     (11904, 192), (11968, 192), (12032, 192), (14208, 192)])                              # 192, 64, 128, 192
@pytest.mark.parametrize("K", [64, 1088])
def test_one_row_of_tiles(cuda, M, N, width, K):
    check(cuda, M, N, K, width)


# three rows of pair tiles and more
@pytest.mark.parametrize("M,N,width", [(513, 3392, 160), (750, 3584, 160), (768, 3712, 160), (768, 3840, 160), (640, 4096, 192), (513, 4608, 192),
                                       (1281, 2304, 192), (1500, 2304, 192), (512, 6144, 192), (1024, 6144, 192), (257, 6912, 192),
                                       (3000, 2048, 192)])
@pytest.mark.parametrize("K", [64, 1088])
def test_rows_of_tiles(cuda, M, N, width, K):
    check(cuda, M, N, K, width)
