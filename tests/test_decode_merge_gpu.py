"""The merge of a decode row's key ranges: few and many of them, more than there are pages, a workspace off the 16-byte grid."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("splits,shift", [(2, 0), (9, 0), (32, 1), (300, 0)])
def test_ranges_meet_in_the_whole_softmax(D, splits, shift):
    from gpustack_b200 import ops

    B, Hq, Hkv = 3, 12, 3
    lens = [1, 161, 700]
    g = torch.Generator().manual_seed(D + splits)
    nb = (max(lens) + 15) // 16
    k, v = (torch.randn(B * nb, Hkv, 16, D, generator=g).to(torch.bfloat16).cuda() for _ in range(2))
    table = torch.randperm(B * nb, generator=g).to(torch.int32).view(B, nb).cuda()
    q = torch.randn(B, Hq * D, generator=g).to(torch.bfloat16).cuda()
    out = torch.empty(B, Hq * D, dtype=torch.bfloat16, device="cuda")
    lse = torch.empty(B, Hq, device="cuda")
    ws = ops.attn_decode_workspace(B, Hq, D, splits, "cuda")
    ws = torch.zeros(ws.numel() + 4, device="cuda")[shift:]
    for _ in range(2):                                   # the arrival counters reset themselves
        ops.paged_attn_decode(q, Hq * D, k, v, table, torch.tensor(lens, dtype=torch.int32, device="cuda"), out, Hq, Hkv, D, D ** -0.5,
                              num_splits=splits, workspace=ws, lse_out=lse)
        for b, n in enumerate(lens):
            rows = [c[table[b].long()].transpose(1, 2).reshape(-1, Hkv, D)[:n].double() for c in (k, v)]
            s = torch.einsum("hgd,nhd->hgn", q[b].double().view(Hkv, -1, D), rows[0]) * D ** -0.5
            want = torch.einsum("hgn,nhd->hgd", s.softmax(-1), rows[1]).reshape(-1)
            # bf16 probabilities and output, 2^-9 each
            assert float((out[b].double() - want).norm() / want.norm()) < 2 * 2.0 ** -9
            # fp32 scores of |s| < 8, D products each
            assert float((lse[b].double() - s.logsumexp(-1).reshape(-1)).abs().max()) < 8 * D * 2.0 ** -24
