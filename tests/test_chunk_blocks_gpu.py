"""Chunks in blocks of four rows: channels cleared at each place of a block, rows that end inside one, values that are no number."""
import pytest
import torch

pytestmark = pytest.mark.gpu

F64 = torch.float64
# sums of at most 300 terms of one size without cancellation, each rounding by itself and by at most 2^-24 of the sum
TOL = 300 ** 0.5 * 2.0 ** -24


@pytest.mark.parametrize("rows", [61, 66, 131])
@pytest.mark.parametrize("H,dk,dv", [(2, 64, 64), (1, 64, 128), (1, 128, 128)])
def test_gated_linear_blocks(rows, H, dk, dv):
    from gpustack_b200 import ops

    def i32(v):
        return torch.tensor(v, dtype=torch.int32, device="cuda")

    g = torch.Generator().manual_seed(rows + dk + dv)
    x, z = torch.randn(rows, 2 * H * dk + H * dv, generator=g), torch.randn(rows, H * dk, generator=g) * 6
    for r in range(9, rows, 5):                     # every place of a block, another set of channels each time
        z[r, r % 7::7] = -float("inf") if r % 2 else -1.0e5
    S = torch.randn(1, H, dv, dk, generator=g)

    def scan(rows_):
        o, S_d = torch.zeros(rows, H * dv, device="cuda"), S.cuda()
        ops.gla_scan(rows_.cuda(), 0, H * dk, 2 * H * dk, z.cuda(), 1.0 / 16, i32([0, rows]), i32([5]), i32([0]), S_d, o, H, dk, dv, max_len=4096)
        return o.cpu(), S_d.cpu()

    q, k = x[:, :H * dk].view(rows, H, dk).to(F64), x[:, H * dk:2 * H * dk].view(rows, H, dk).to(F64)
    v = x[:, 2 * H * dk:].view(rows, H, dv).to(F64)
    alpha = torch.exp(torch.nn.functional.logsigmoid(z.to(F64)) / 16).view(rows, H, dk)
    want, Z = torch.zeros(rows, H, dv, dtype=F64), S[0].to(F64).clone()
    for t in range(rows):
        Z = alpha[t][:, None] * Z + v[t][:, :, None] * k[t][:, None]
        want[t] = torch.einsum("hvk,hk->hv", Z, q[t])
    o, S_end = scan(x)
    want = want.view(rows, -1)
    assert float((o.to(F64) - want).norm() / want.norm()) < TOL
    assert float((S_end[0].to(F64) - Z).norm() / Z.norm()) < TOL
    for bad in (13, 30, 60):                        # odd and even rows of a pair: a row's value reaches itself and later rows only
        y = x.clone()
        y[bad, 2 * H * dk:] = float("nan")
        got = scan(y)[0]
        assert torch.equal(got[:bad], o[:bad]) and got[bad:].isnan().all()
