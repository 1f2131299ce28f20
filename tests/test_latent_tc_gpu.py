"""Latent attention of prompt portions on CTA pairs, and the products of all heads in one launch, against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

F64, BF = torch.float64, torch.bfloat16
R, DR = 512, 64


def _rel(a, b):
    return float((a.cpu().to(F64) - b).norm() / b.norm())


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("M", [1, 33, 257, 700])
@pytest.mark.parametrize("H,N,K,pad", [(16, 512, 128, 64), (5, 128, 512, 0), (3, 192, 64, 64), (2, 72, 128, 8)])
def test_products_of_all_heads(H, N, K, pad, M, f32):
    from gpustack_b200.lib import check, load

    g = torch.Generator().manual_seed(M + N)
    x_head, y_head = K + pad, N + pad
    x = torch.randn(M, H * x_head, generator=g).to(BF)
    w = torch.randn(H, N, K, generator=g).to(BF)
    out = torch.full((M, H * y_head), 9.0, dtype=torch.float32 if f32 else BF, device="cuda")
    xd, wd = x.cuda(), w.cuda()
    check(load().b200_gemm_bf16_heads(xd.data_ptr(), wd.data_ptr(), out.data_ptr(), M, N, K, xd.stride(0), out.stride(0), H, x_head, y_head,
                                      int(f32), torch.cuda.current_stream().cuda_stream))
    want = torch.einsum("thk,hnk->thn", x.view(M, H, x_head)[..., :K].to(F64), w.to(F64))
    got = out.view(M, H, y_head).cpu()
    # fp32 sums of K exact products (K 2^-24 of the terms' norm at most), and one bf16 rounding
    assert float((got[..., :N].to(F64) - want).norm() / want.norm()) < (K * 2.0 ** -24 if f32 else 2.0 ** -8)
    assert bool((got[..., N:] == 9.0).all())                       # what lies between the heads is left alone
