"""Pairs of tokens and experts grouped by expert: every pair one row among its expert's, every other row marked as padding."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# around the CTA's 256 and 1024 threads, one warp of experts and several, experts without a pair, one expert with all of them
@pytest.mark.parametrize("n", [1, 255, 256, 257, 1024, 1025, 5000])
@pytest.mark.parametrize("E,block", [(1, 16), (8, 32), (33, 16), (256, 64)])
def test_every_pair_has_its_row(n, E, block):
    from gpustack_b200 import ops
    from gpustack_b200.lib import check, load

    g = torch.Generator().manual_seed(n + E)
    used = torch.randperm(E, generator=g)[:max(1, E // 2)]
    ids = used[torch.randint(0, len(used), (n,), generator=g)].to(torch.int32)
    if E == 8:
        ids[:] = 5
    w = torch.rand(n, generator=g) + 0.1
    cap = load().b200_moe_capacity_rows(n, E, block)
    i32 = lambda m: torch.full((m,), -7, dtype=torch.int32, device="cuda")   # noqa: E731
    pair_row, row_pair, tile_expert, num = i32(n), i32(cap), i32(cap // block), i32(2)
    row_weight = torch.full((cap,), float("nan"), device="cuda")
    ids_d, w_d = ids.cuda(), w.cuda()
    check(load().b200_moe_align(ids_d.data_ptr(), w_d.data_ptr(), n, E, block, cap, pair_row.data_ptr(), row_pair.data_ptr(), row_weight.data_ptr(),
                                tile_expert.data_ptr(), num.data_ptr(), ops._stream()), "moe_align")
    tiles = (torch.bincount(ids.long(), minlength=E) + block - 1) // block
    total = int(tiles.sum())
    assert num.tolist() == [total, total * block]
    assert torch.equal(tile_expert[:total].cpu().long(), torch.repeat_interleave(torch.arange(E), tiles))
    rows = pair_row.cpu().long()
    assert torch.equal(rows.sort().values, rows.unique()) and int(rows.min()) >= 0 and int(rows.max()) < total * block
    assert torch.equal(tile_expert.cpu()[rows // block], ids)
    want = torch.full((cap,), -1, dtype=torch.int32)
    want[rows] = torch.arange(n, dtype=torch.int32)
    weights = torch.zeros(cap)
    weights[rows] = w
    assert torch.equal(row_pair.cpu(), want) and torch.equal(row_weight.cpu(), weights)
