"""Products of more than 128 rows whose rounds are filled by tiles of 160 and 192 columns (csrc/gemm_tcgen05.cu: choose_tile): columns
that those widths do not divide, a last tile of 32, 64 and 128 columns or without a half, rows at the edges of the pair's 256."""
import pytest
import torch

from tests.util import bf16_close

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


# 160 columns: 3584 = 22 x 160 + 64, 3392 = 21 x 160 + 32; 192: 4096 = 21 x 192 + 64, 2304 = 12 x 192, 6144 = 32 x 192, 3712 = 19 x 192 + 64,
# 8192 = 42 x 192 + 128
@pytest.mark.parametrize("M,N", [(513, 3584), (750, 3584), (768, 3392), (640, 4096), (768, 3712), (1281, 2304), (1500, 2304), (512, 6144), (1024, 6144),
                                 (513, 8192), (3000, 2048), (1537, 4096)])
@pytest.mark.parametrize("K", [64, 1088])
def test_ragged_tiles(cuda, M, N, K):
    from llmq_b200 import lib
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
                lib.gemm_bf16(a, w, c)
                assert torch.equal(c, whole[:M])
        finally:
            lib.gemm_set_tile_n(0)
