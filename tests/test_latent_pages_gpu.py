"""Single rows over the latent cache: pages of 16 rows, each one copy, beside pages whose rows are copied one by one, against 64 bits.
Sequences end at every kind of place of a page, and what lies behind their end is no number."""
import pytest
import torch

pytestmark = pytest.mark.gpu

BF, F64 = torch.bfloat16, torch.float64
LENS = [1, 15, 16, 17, 31, 32, 33, 48, 49, 64, 65, 130, 0, 333]


@pytest.mark.parametrize("H,R,dr", [(16, 512, 64), (5, 128, 64), (1, 64, 64), (16, 384, 64), (8, 192, 64), (2, 256, 64), (4, 192, 32)])
@pytest.mark.parametrize("page", [16, 32])
@pytest.mark.parametrize("ranges", [1, 3])
def test_single_rows_by_pages(H, R, dr, page, ranges):
    from gpustack_b200 import ops

    g = torch.Generator().manual_seed(H + R)
    W, B = R + dr, len(LENS)
    need = [(n + page - 1) // page for n in LENS]
    order = torch.randperm(sum(need), generator=g).to(torch.int32) + 1
    table, at = torch.zeros(B, max(need) + 1, dtype=torch.int32), 0        # (page 0 belongs to nobody)
    cache = torch.full((sum(need) + 1, 1, page, W), float("nan"), dtype=BF)
    cache[:, :, 1::2] = float("inf")
    rows = [torch.randn(n, W, generator=g).to(BF) for n in LENS]
    for b, n in enumerate(LENS):
        for j in range(need[b]):
            table[b, j] = order[at]
            part = rows[b][j * page:(j + 1) * page]
            cache[int(order[at]), 0, :part.shape[0]] = part
            at += 1
    q, sink, scale = torch.randn(B, H, W, generator=g).to(BF), torch.randn(H, generator=g), W ** -0.5
    out = torch.full((B, H * R), 7.0, dtype=BF, device="cuda")
    ws = None
    if ranges > 1:
        ws = ops.latent_attn_decode_workspace(B, H, R, ranges, "cuda")
        ws.fill_(float("nan"))
    ops.latent_attn_decode(q.reshape(B, -1).cuda(), cache.cuda(), table.cuda(), torch.tensor(LENS, dtype=torch.int32, device="cuda"), sink.cuda(),
                           out, H, R, dr, scale, num_splits=ranges, workspace=ws)
    for b, n in enumerate(LENS):
        got = out[b].view(H, R).cpu().to(F64)
        if n == 0:
            assert bool((got == 0).all())
            continue
        s = torch.cat([q[b].to(F64) @ rows[b].to(F64).T * scale, sink.to(F64)[:, None]], 1)
        want = torch.softmax(s, 1)[:, :n] @ rows[b][:, :R].to(F64)
        # probabilities and results are rounded to 8 bits: 2^-9 each, and the scores' fp32 sums below that
        assert float((got - want).norm() / want.norm()) < 2 * 2.0 ** -8, n
