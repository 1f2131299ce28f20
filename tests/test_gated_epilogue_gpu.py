"""The gated epilogue of the products against the product and the activation apart, where its quotients leave the branch-free range."""
import pytest
import torch

pytestmark = pytest.mark.gpu

BF = torch.bfloat16


# one token (16-column tiles), a remainder, whole tiles of 256, a second tile
@pytest.mark.parametrize("M,I", [(1, 128), (33, 104), (256, 512), (300, 136)])
def test_values_out_of_the_quotients_range(M, I):
    from gpustack_b200 import ops

    g = torch.Generator().manual_seed(M + I)
    x = torch.randn(M, 64, generator=g)
    x[:, 0] = 1.0
    wg, wu = torch.randn(I, 64, generator=g), torch.randn(I, 64, generator=g)
    # gates around the exponential's ends, beyond 2^100, subnormal, infinite and no number, each in a chunk with ordinary ones
    for i, v in enumerate([-87.0, -88.0, -89.0, -104.0, -1.0e4, 88.0, 1.0e4, 3.0e30, -3.0e30, 1.0e-39, -1.0e-39, float("inf"), -float("inf"),
                           float("nan")]):
        wg[3 + 7 * i] = 0.0
        wg[3 + 7 * i, 0] = v
    x, wg, wu = x.to(BF).cuda(), wg.to(BF).cuda(), wu.to(BF).cuda()
    fused = ops.gemm_silu_mul(x, ops.interleave_gate_up(wg, wu))
    apart = ops.silu_and_mul(ops.gemm(x, torch.cat([wg, wu], dim=0).contiguous()))
    assert torch.equal(fused.isnan(), apart.isnan())
    assert torch.equal(fused.nan_to_num(7.0), apart.nan_to_num(7.0))
