"""Linear attention over chunks of 128 rows on the tensor cores against the recurrence in fp64: chunk edges, values that are bf16 numbers in
all, some or none of a chunk's halves (one term or three), and more items than CTAs."""
import pytest
import torch

pytestmark = pytest.mark.gpu

F64 = torch.float64
# fp32 sums of at most 128 + 128 terms and a chunk's share of the state, every rounding the same way, terms without cancellation beyond 2
TOL = 2 * 300 * 2.0 ** -24


@pytest.mark.parametrize("lens,H", [([128], 1), ([129], 1), ([255, 257], 2), ([700], 40)], ids=str)
@pytest.mark.parametrize("exact", ["all", "some", "none"])
@pytest.mark.parametrize("dk,dv", [(128, 128), (64, 64)])
def test_edges_and_terms(lens, H, exact, dk, dv):
    from gpustack_b200 import ops

    g = torch.Generator().manual_seed(sum(lens) + dk)
    T, n = sum(lens), len(lens)
    x, S = torch.randn(T, 2 * H * dk + H * dv, generator=g), torch.randn(n, H, dv, dk, generator=g)
    rows = {"all": T, "some": 70, "none": 0}[exact]
    x[:rows, 2 * H * dk:] = x[:rows, 2 * H * dk:].to(torch.bfloat16).float()
    cu = [sum(lens[:i]) for i in range(n + 1)]
    decay = torch.linspace(0.5, 0.999, H)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")   # noqa: E731
    o, S_d = torch.zeros(T, H * dv, device="cuda"), S.cuda()
    ops.linattn_scan(x.cuda(), 0, H * dk, 2 * H * dk, decay.cuda(), i32(cu), i32([9] * n), i32(list(range(n))), S_d, o, H, dk, dv, max_len=max(lens))
    q, k = x[:, :H * dk].view(T, H, dk).to(F64), x[:, H * dk:2 * H * dk].view(T, H, dk).to(F64)
    v, want = x[:, 2 * H * dk:].view(T, H, dv).to(F64), torch.zeros(T, H, dv, dtype=F64)
    for i in range(n):
        Z = S[i].to(F64)
        for t in range(cu[i], cu[i + 1]):
            Z = decay.to(F64)[:, None, None] * Z + v[t][:, :, None] * k[t][:, None]
            want[t] = torch.einsum("hvk,hk->hv", Z, q[t])
        assert float((S_d[i].cpu().to(F64) - Z).norm() / Z.norm()) < TOL
    assert float((o.cpu().to(F64) - want.view(T, -1)).norm() / want.norm()) < TOL
