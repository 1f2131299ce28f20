"""The router's product and choice in one launch against fp64 and against the choice alone on the same logits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# an odd last token, rows that fill no warp, no cluster, several passes; widths below and beyond a warp's 256 columns
@pytest.mark.parametrize("T", [1, 2, 7, 64])
@pytest.mark.parametrize("N,E,D,top,groups,keep", [(3, 3, 64, 2, 0, 0), (128, 8, 2048, 2, 0, 0), (131, 130, 264, 5, 0, 0), (256, 256, 520, 8, 8, 3)])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_router(T, N, E, D, top, groups, keep, mode):
    from gpustack_b200 import ops
    from gpustack_b200.lib import load

    g = torch.Generator().manual_seed(T + N + D)
    x, w = torch.randn(T, D, generator=g).to(torch.bfloat16), (torch.randn(N, D, generator=g) * D ** -0.5).to(torch.bfloat16)
    corr = torch.randn(E, generator=g).cuda() if mode else None
    xd, wd, st = x.cuda(), w.cuda(), torch.cuda.current_stream().cuda_stream
    lg = torch.full((T, N + 5), 7.0, device="cuda")
    ids, wt, ids2, wt2 = (torch.zeros(T, top, dtype=t, device="cuda") for t in (torch.int32, torch.float32) * 2)
    cp = None if corr is None else corr.data_ptr()
    ops.check(load().b200_moe_router(xd.data_ptr(), D, wd.data_ptr(), D, N, D, lg.data_ptr(), lg.stride(0), cp, ids.data_ptr(), wt.data_ptr(), T, E,
                                     top, 1.3, mode, 1, groups, keep, st))
    ops.check(load().b200_moe_route_grouped(lg.data_ptr(), lg.stride(0), cp, ids2.data_ptr(), wt2.data_ptr(), T, E, top, 1.3, mode, 1, groups, keep,
                                            st))
    want = x.double() @ w.double().T
    # a lane's sum of D / 32 products and five steps of the butterfly, each rounded, against the sum of the terms' sizes
    bound = (D / 32 + 6) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)
    assert bool(((lg[:, :N].cpu().double() - want).abs() <= bound).all()) and bool((lg[:, N:] == 7.0).all())
    assert torch.equal(ids, ids2) and torch.equal(wt, wt2)


def test_router_of_the_narrowest_rows():
    """Eight columns: next to no work between a CTA's start and its stores into the cluster's first CTA."""
    for T in (1, 2, 33):
        test_router(T, 65, 64, 8, 3, 0, 0, 0)
