"""Latent attention of prompt portions on CTA pairs, and the products of all heads in one launch, against fp64."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

F64, BF = torch.float64, torch.bfloat16
R, DR = 512, 64


def _rel(a, b):
    return float((a.cpu().to(F64) - b).norm() / b.norm())


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


# portions around the item (256 / H rows), page (16), value unit (32) and block (96) edges, new and continued, several in one step
@pytest.mark.parametrize("H", [16, 32, 128])
@pytest.mark.parametrize("lens,ctx", [([1], [0]), ([16], [0]), ([17], [47]), ([96], [0]), ([97], [96]), ([65, 1, 200], [0, 127, 64]),
                                      ([33, 130], [300, 0])], ids=str)
def test_prompt_portions(H, lens, ctx):
    from gpustack_b200 import ops

    g = torch.Generator().manual_seed(H + sum(lens))
    T, total = sum(lens), [a + b for a, b in zip(lens, ctx)]
    need = [(n + 15) // 16 for n in total]
    order = torch.randperm(sum(need), generator=g).to(torch.int32)
    table = torch.zeros(len(lens), max(need) + 2, dtype=torch.int32)
    cache = torch.full((sum(need), 1, 16, R + DR), float("nan"), dtype=BF)      # what no sequence owns is no number
    rows, at = [], 0
    for i, n in enumerate(total):
        table[i, :need[i]] = order[at:at + need[i]]
        at += need[i]
        rows.append(torch.randn(n, R + DR, generator=g).to(BF))
        for j in range(n):
            cache[table[i, j // 16], 0, j % 16] = rows[i][j]
    q = torch.randn(T, H * (R + DR), generator=g).to(BF)
    sink, scale = torch.randn(H, generator=g), 1.5 * (R + DR) ** -0.5
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    ts, tq = ops.build_prefill_tiles(lens, ops.attn_sink_prefill_tile(), ctx)
    out = torch.zeros(T, H * R, dtype=BF, device="cuda")
    ops.latent_attn_prefill(q.cuda(), cache.cuda(), table.cuda(), _i32(cu), _i32(ctx), _i32(ts), _i32(tq), sink.cuda(), out, H, R, DR, scale)
    want = []
    for i, n in enumerate(lens):
        k = rows[i].to(F64)
        s = torch.einsum("thd,nd->htn", q[cu[i]:cu[i + 1]].to(F64).view(n, H, R + DR), k) * scale
        s.masked_fill_(torch.arange(total[i])[None] > ctx[i] + torch.arange(n)[:, None], -float("inf"))
        p = torch.cat([s, sink.to(F64)[:, None, None].expand(H, n, 1)], -1).softmax(-1)[..., :-1]
        want.append(torch.einsum("htn,nr->thr", p, k[:, :R]).reshape(n, -1))
    # bf16 probabilities and outputs: 2^-9 each, rounded independently
    assert _rel(out, torch.cat(want)) < 2 * 2.0 ** -9


def test_a_growing_maximum_moves_the_reference():
    """Scores that rise by far more than 2^8 from block to block: the accumulators are rescaled on the way."""
    from gpustack_b200 import ops

    H, n = 16, 520
    g = torch.Generator().manual_seed(2)
    C = torch.randn(n, R + DR, generator=g)
    C[:, R] = torch.arange(n) // 100 * 40.0
    q = torch.randn(1, H, R + DR, generator=g) * 0.02
    q[..., R] = 1.0
    C, q = C.to(BF), q.to(BF)
    cache = torch.zeros((n + 15) // 16, 1, 16, R + DR, dtype=BF)
    cache.view(-1, R + DR)[:n] = C
    out = torch.zeros(1, H * R, dtype=BF, device="cuda")
    ts, tq = ops.build_prefill_tiles([1], ops.attn_sink_prefill_tile(), [n - 1])
    ops.latent_attn_prefill(q.view(1, -1).cuda(), cache.cuda(), torch.arange(cache.shape[0], dtype=torch.int32).view(1, -1).cuda(), _i32([0, 1]),
                            _i32([n - 1]), _i32(ts), _i32(tq), None, out, H, R, DR, 1.0)
    p = (q[0].to(F64) @ C.to(F64).T).softmax(-1)
    assert _rel(out.view(H, R), p @ C[:, :R].to(F64)) < 2 * 2.0 ** -9


def test_the_largest_probability_is_exact():
    """A key that outweighs an earlier block's by 4 (1 + 2^-8), halfway between two bf16 numbers: relative to the earlier block's
    maximum its probability would be off by 2^-8, relative to its own it is 1."""
    from gpustack_b200 import ops

    H, n = 16, 200
    delta = 2.0 + math.log2(1 + 2.0 ** -8)                       # base-2 distance of the two scores
    C = torch.zeros(n, R + DR)
    C[:, R] = -100.0                                             # every other key's weight is 2^-200
    C[3, R], C[150, R] = 0.0, 1.0
    C[150, :R] = torch.randn(R, generator=torch.Generator().manual_seed(5))
    C = C.to(BF)
    q = torch.zeros(1, H, R + DR, dtype=BF)
    q[..., R] = 1.0
    cache = torch.zeros((n + 15) // 16, 1, 16, R + DR, dtype=BF)
    cache.view(-1, R + DR)[:n] = C
    out = torch.zeros(1, H * R, dtype=BF, device="cuda")
    ts, tq = ops.build_prefill_tiles([1], ops.attn_sink_prefill_tile(), [n - 1])
    ops.latent_attn_prefill(q.view(1, -1).cuda(), cache.cuda(), torch.arange(cache.shape[0], dtype=torch.int32).view(1, -1).cuda(), _i32([0, 1]),
                            _i32([n - 1]), _i32(ts), _i32(tq), None, out, H, R, DR, delta * math.log(2.0))
    want = (C[150, :R].to(F64) * (2.0 ** delta / (1 + 2.0 ** delta))).expand(H, R)
    # the output's rounding, at most 2^-9, and the smaller probability's, 2^-9 of a fifth of the weight
    assert _rel(out.view(H, R), want) < 1.2 * 2.0 ** -9


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


@pytest.mark.parametrize("splits", [1, 2, 7])
@pytest.mark.parametrize("H,R,dr", [(16, 512, 64), (9, 128, 16), (17, 384, 48), (1, 256, 0)])
def test_single_rows_at_the_edges_of_key_blocks(H, R, dr, splits):
    """One new row per sequence: lengths around the blocks of 32 keys and their halves, a row without keys, widths of an odd number of 16-column
    steps, 1 to 16 heads per CTA.  bf16 probabilities and outputs: each rounds by at most 2^-8 of its value (half a unit in the
    last of 8 bits), so the two together stay below 2 * 2^-8 of the output's norm."""
    from gpustack_b200 import ops

    lens = [1, 15, 16, 17, 31, 32, 33, 97, 0, 513]
    g = torch.Generator().manual_seed(H + R + dr)
    pages = [-(-max(n, 1) // 16) for n in lens]
    order = torch.randperm(sum(pages), generator=g).to(torch.int32)
    cache = torch.randn(sum(pages), 1, 16, R + dr, generator=g).to(torch.bfloat16)
    bt = torch.zeros(len(lens), max(pages), dtype=torch.int32)
    q = torch.randn(len(lens), H * (R + dr), generator=g).to(torch.bfloat16)
    scale, off, want = 1.3 / (R + dr) ** 0.5, 0, torch.zeros(len(lens), H, R, dtype=torch.float64)
    for b, n in enumerate(lens):
        bt[b, :pages[b]] = order[off:off + pages[b]]
        off += pages[b]
        if n:
            k = cache[bt[b, :pages[b]].long()].reshape(-1, R + dr)[:n].double()
            want[b] = torch.softmax(scale * q[b].view(H, -1).double() @ k.T, dim=-1) @ k[:, :R]
    for b, n in enumerate(lens):                       # what lies behind a sequence's last key is no number
        if n % 16:
            cache[bt[b, pages[b] - 1].long(), 0, n % 16:] = float("nan")
    out = torch.full((len(lens), H * R), 3.0, dtype=torch.bfloat16, device="cuda")
    ws = ops.latent_attn_decode_workspace(len(lens), H, R, splits, "cuda")
    ops.latent_attn_decode(q.cuda(), cache.cuda(), bt.cuda(), torch.tensor(lens, dtype=torch.int32, device="cuda"), None, out, H, R, dr, scale,
                           num_splits=splits, workspace=ws)
    got = out.view(len(lens), H, R).double().cpu()
    assert bool((got[lens.index(0)] == 0).all())
    for b, n in enumerate(lens):
        if n:
            assert float((got[b] - want[b]).norm() / want[b].norm()) < 2 * 2.0 ** -8, n


@pytest.mark.parametrize("half", [True, False])
@pytest.mark.parametrize("T,H", [(1, 1), (3, 8), (5, 17), (597, 16)])
def test_preparation_of_rows(T, H, half):
    """One warp per row: heads below, at and beyond a batch of eight, a remainder of rows in the last CTA, a padding row."""
    from gpustack_b200 import ops

    g = torch.Generator().manual_seed(T + H)
    dn, kv_col, mag, eps = 6, 8, 1.25, 1e-5
    proj, q = torch.randn(T, kv_col + R + DR + 8, generator=g).to(BF), torch.randn(T, H * (dn + DR), generator=g).to(BF)
    w, pos = torch.randn(R, generator=g).to(BF), torch.randint(0, 100000, (T,), generator=g, dtype=torch.int32)
    freq = 10000.0 ** (-torch.arange(DR // 2, dtype=F64) / 32)
    slots = torch.randperm(T + 16, generator=g)[:T].to(torch.int32)
    if T > 1:
        slots[T // 2] = -1
    pages = -(-(T + 16) // 16)
    cache, qa = torch.full((pages, 1, 16, R + DR), 9.0, dtype=BF, device="cuda"), torch.full((T, H * (R + DR)), 9.0, dtype=BF, device="cuda")
    ops.latent_prep(proj.cuda(), kv_col, q.cuda(), w.cuda(), pos.cuda(), slots.cuda(), cache, qa, H, dn, DR, R, DR, half, freq.cuda(), mag, eps)

    def turn(x):                                       # [..., T, 64]
        ang = pos.to(F64)[:, None] * freq
        c, s = torch.cos(ang) * mag, torch.sin(ang) * mag
        a, b = (x[..., :32], x[..., 32:]) if half else (x[..., ::2], x[..., 1::2])
        u, v = a * c - b * s, b * c + a * s
        return torch.cat([u, v], -1) if half else torch.stack([u, v], -1).flatten(-2)

    lat = proj[:, kv_col:kv_col + R].to(F64)
    want = torch.cat([lat / torch.sqrt((lat * lat).mean(-1, keepdim=True) + eps) * w.to(F64), turn(proj[:, kv_col + R:kv_col + R + DR].to(F64))], -1)
    live = slots >= 0
    got = cache.view(-1, R + DR)[slots[live].long().cuda()]
    # one rounding to bf16 (2^-9 of each value; an angle's reduction and the fp32 products are far below)
    assert float((got.cpu().to(F64) - want[live]).abs().max() / want.abs().max()) < 2.0 ** -8
    assert _rel(got, want[live]) < 2.0 ** -9
    rest = torch.ones(pages * 16, dtype=torch.bool)
    rest[slots[live].long()] = False
    assert bool((cache.view(-1, R + DR).cpu()[rest] == 9.0).all())
    parts = turn(q.view(T, H, dn + DR)[..., dn:].to(F64).transpose(0, 1)).transpose(0, 1)
    assert _rel(qa.view(T, H, R + DR)[..., R:], parts) < 2.0 ** -9
    assert bool((qa.view(T, H, R + DR)[..., :R] == 9.0).all())
