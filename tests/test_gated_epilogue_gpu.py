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


@pytest.mark.parametrize("M,I", [(1, 128), (33, 104), (256, 512), (300, 136)])
def test_clamped_values_out_of_the_quotients_range(M, I):
    """The clamped form, whose exponent is 1.702 gates and whose gates and values end at a limit, against fp64."""
    from gpustack_b200 import ops

    limit = 7.0
    g = torch.Generator().manual_seed(M + I)
    x = torch.randn(M, 64, generator=g)
    x[:, 0] = 1.0
    wg, wu = torch.randn(I, 64, generator=g), torch.randn(I, 64, generator=g)
    for i, v in enumerate([-51.0, -52.0, -52.5, -61.0, -1.0e4, 7.0, 52.0, 1.0e4, 3.0e30, -3.0e30, 1.0e-39, float("inf"), float("nan")]):
        wg[3 + 7 * i] = 0.0
        wg[3 + 7 * i, 0] = v
    for i, v in enumerate([-3.0e30, 3.0e30, float("inf"), -float("inf"), -7.0, 7.0]):
        wu[1 + 16 * i] = 0.0
        wu[1 + 16 * i, 0] = v
    x, wg, wu = x.to(BF), wg.to(BF), wu.to(BF)
    got = torch.empty(M, I, dtype=BF, device="cuda")
    ops.gated_linear(x.cuda(), ops.interleave_gate_up(wg.cuda(), wu.cuda()), got, "clamped_swish", limit)
    D = lambda t: t.double()   # noqa: E731
    prod = lambda w: torch.where(w[:, 1:].eq(0).all(-1)[None], D(w)[:, 0][None].expand(M, I), D(x) @ D(w).nan_to_num(0.0, 0.0, 0.0).T)   # noqa: E731
    # (a gate that is no number passes the smaller of itself and the limit: the limit)
    a = torch.fmin(prod(wg), torch.tensor(limit, dtype=torch.float64))
    want = a * torch.sigmoid(1.702 * a) * (prod(wu).clamp(-limit, limit) + 1.0)
    # fp32 sums of the products, 2^-22 of their terms each, through the form's slopes (at most 1.1 in the gate); the exponential and
    # the quotient, 2^-14 (an argument of 88 off by 2^-24 of itself); half a unit of bf16's 8 bits; quotients below fp32's range are zero
    terms = lambda w: 2.0 ** -22 * (D(x).abs() @ D(w).nan_to_num(0.0, 0.0, 0.0).abs().clamp(max=1.0e3).T)   # noqa: E731
    act, up = (a * torch.sigmoid(1.702 * a)).abs(), prod(wu).clamp(-limit, limit).abs() + 1.0
    bound = 2.0 ** -8 * want.abs() + 2.0 ** -14 * act * up + 1.1 * terms(wg) * up + terms(wu) * act + 2.0 ** -120
    assert bool(((got.cpu().double() - want).abs() <= bound).all())
