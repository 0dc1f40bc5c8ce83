"""Routing of a grouped mixture (csrc/prenorm_ops.cu) at the numbers of experts where its form changes: one to eight experts per lane
in registers, more than those read again for every pick; equal, infinite and masked choices; and the sums of routed rows whose choices
are read four at a time."""
import pytest
import torch

from oracle import fimilorn as O

pytestmark = pytest.mark.gpu


def route(cuda, z, corr, top, groups, keep):
    from llmq_b200 import lib as L
    lib = L.load()
    T, E = z.shape
    ints = lambda n: torch.full((n,), -1, dtype=torch.int32, device=cuda)
    idx, off, perm, pair, wts = ints(T * top), ints(E + 1), ints(T * top), ints(T * top), torch.zeros(T * top, device=cuda)
    zd, cd = z.to(cuda).contiguous(), corr.to(cuda).contiguous()
    L.check(lib.b200q_moe_route_gated(zd.data_ptr(), E, cd.data_ptr(), T, E, top, groups, keep, 0, idx.data_ptr(), wts.data_ptr(),
                                      off.data_ptr(), perm.data_ptr(), pair.data_ptr(), None, None, None))
    torch.cuda.synchronize()
    return idx.cpu().view(T, top), wts.cpu().view(T, top)


@pytest.mark.parametrize("E,groups,keep", [(32, 4, 2), (33, 3, 2), (64, 1, 1), (68, 4, 3), (128, 8, 2), (132, 2, 1), (256, 16, 5), (264, 8, 3), (1024, 4, 2)])
def test_picks(cuda, E, groups, keep):
    g = torch.Generator().manual_seed(E)
    T, top = 21, min(8, keep * (E // groups))
    z, corr = torch.randn(T, E, generator=g), torch.randn(E, generator=g) * 0.4 - 2.0
    idx, wts = route(cuda, z, corr, top, groups, keep)
    want_i, want_w = O.route(z.double(), corr.double(), top, groups, keep)
    for t in range(T):   # (the oracle's order of picks is that of their choices, as here)
        assert idx[t].tolist() == want_i[t].tolist()
    assert torch.allclose(wts.double(), want_w, atol=1e-6)
    # all choices equal: the lowest experts of the lowest groups; one infinite: picked first
    idx, _ = route(cuda, torch.zeros(1, E), torch.full((E,), -1.0), top, groups, keep)
    assert idx[0].tolist() == list(range(top))
    lifted = torch.full((E,), -1.0)
    lifted[E - 1] = float("inf")
    idx, _ = route(cuda, torch.zeros(1, E), lifted, top, groups, keep)
    assert idx[0, 0] == E - 1
    # minus infinity is a choice like any other, below all finite ones
    sunk = torch.full((E,), float("-inf"))
    sunk[0] = 0.0
    n = min(top, E // groups)
    idx, _ = route(cuda, torch.zeros(1, E), sunk, n, groups, 1)
    assert idx[0].tolist() == list(range(n))


@pytest.mark.parametrize("top", [1, 3, 4, 5, 8, 9])
@pytest.mark.parametrize("T,W", [(13, 8), (13, 2056), (1179, 2056), (1180, 2056)])   # four choices at a time, at last one
def test_sums_of_routed_rows(cuda, top, T, W):
    from llmq_b200 import lib as L
    lib = L.load()
    g = torch.Generator().manual_seed(top * W)
    real = 6
    x, eo = torch.randn(T, W, generator=g), torch.randn(T * top, W, generator=g).to(torch.bfloat16)
    h, wts = torch.randn(T, W, generator=g).to(torch.bfloat16), torch.rand(T * top, generator=g)
    idx, pair = torch.randint(0, real + 2, (T * top,), generator=g).to(torch.int32), torch.randperm(T * top, generator=g).to(torch.int32)
    d = [v.to(cuda) for v in (x, eo, pair, idx, wts, h)]
    L.check(lib.b200q_residual_add_routed(*[v.data_ptr() for v in d[:5]], top, real, d[5].data_ptr(), T, W, L.DTYPE_BF16, None))
    torch.cuda.synchronize()
    rows = torch.where((idx < real)[:, None], eo[pair.long()], h.repeat_interleave(top, 0)).double()
    want = x.double() + (wts.double()[:, None] * rows).view(T, top, W).sum(1)
    # top + 1 fp32 additions of terms of order 1
    assert float((d[0].cpu().double() - want).abs().max()) < 2e-6 * (top + 2)
