"""Linear layers on the CUDA cores at the edges of their tiles: rows, outputs and inner widths that fill no tile, results whose rows allow
wide stores and ones that do not, neighbours of the results untouched."""
import pytest
import torch

pytestmark = pytest.mark.gpu

F32, F64, BF = torch.float32, torch.float64, torch.bfloat16


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (63, 65, 15), (64, 64, 16), (65, 66, 17), (130, 68, 33), (3, 7, 100)])
@pytest.mark.parametrize("xd", [F32, BF])
@pytest.mark.parametrize("yd", [F32, BF])
@pytest.mark.parametrize("pad,shift", [(4, 0), (3, 0), (4, 1)])
@pytest.mark.parametrize("biased", [False, True])
def test_edges_of_tiles(M, N, K, xd, yd, pad, shift, biased):
    from gpustack_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x = torch.randn(M, K + 3, generator=g, device="cuda").to(xd)[:, 1:1 + K]
    w = torch.randn(N, K, generator=g, device="cuda").to(BF)
    b = torch.randn(N, generator=g, device="cuda").to(BF) if biased else None
    whole = torch.full((M, (N + 3) // 4 * 4 + pad), 7.0, device="cuda", dtype=yd)
    y = whole[:, shift:shift + N]
    ops.linear(x, w, y, bias=b, force_simt=True)
    want = x.to(F64) @ w.to(F64).T + (0.0 if b is None else b.to(F64))
    size = x.to(F64).abs() @ w.to(F64).abs().T + (0.0 if b is None else b.to(F64).abs())
    # K + 1 roundings of sums no larger than `size`, then that of the result
    assert bool(((y.to(F64) - want).abs() <= (K + 1) * 2.0 ** -24 * size + (2.0 ** -8 if yd == BF else 0.0) * want.abs() + 1e-30).all())
    assert bool((whole[:, :shift] == 7).all()) and bool((whole[:, shift + N:] == 7).all())
