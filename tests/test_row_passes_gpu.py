"""The row passes beside the recurrences: convolved rows in items of 8 to 32 rows, rows without a rotation, values in pairs of pieces, the
closing step over many heads, and gates beyond the range of the polynomial -- each against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu

F32, F64, BF = torch.float32, torch.float64, torch.bfloat16


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


def _rel(a, b):
    return float((a.to(F64) - b).norm() / b.norm())


def _rnd(*s, seed, dtype=F32):
    return torch.randn(*s, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda").to(dtype)


# rows enough for items of 8, 16 and 32, ending inside an item; a second sequence that continues from its ring
@pytest.mark.parametrize("T,heads,taps", [(1190, 128, 4), (2381, 128, 2), (4747, 128, 4), (4747, 128, 1), (70, 3, 3)])
@pytest.mark.parametrize("dtype", [F32, BF])
def test_convolved_rows_in_long_items(T, heads, taps, dtype):
    from gpustack_b200 import ops

    W, R = 64, max(taps - 1, 1)
    C = 2 * heads * W
    lens, ctx, slots = [T - 37, 37], [0, 50], [1, 0]
    cu = [0, T - 37, T]
    u, w, ring = _rnd(T, C, seed=1, dtype=dtype), _rnd(taps, C, seed=2), _rnd(2, R, C, seed=3, dtype=dtype).float()
    tile = ops.attn_prefill_tile(16, 4)
    a, b = ops.build_prefill_tiles(lens, tile, ctx)
    x, after = torch.full((T, C), 7.0, device="cuda"), ring.clone()
    ops.conv_rec_prep(u, w, None, after, _i32(cu), _i32(ctx), _i32(slots), _i32(a), _i32(b), tile, 2, 0,
                      ((heads, W, 0.5), (heads // 2, W, None), (heads - heads // 2, W, None)), x)
    want, want_ring = torch.empty(T, C, dtype=F64, device="cuda"), ring.to(F64)
    for i, (n, c, s) in enumerate(zip(lens, ctx, slots)):
        rows = u[cu[i]:cu[i + 1]].to(F64)
        old = torch.zeros(taps - 1, C, dtype=F64, device="cuda")
        for j in range(min(taps - 1, c)):
            old[taps - 2 - j] = want_ring[s][(c - 1 - j) % R]
        full = torch.cat([old, rows])
        y = sum(w[j].to(F64) * full[j:j + n] for j in range(taps))
        want[cu[i]:cu[i + 1]] = torch.nn.functional.silu(y)
        for j in range(min(taps - 1, n)):
            want_ring[s][(c + n - 1 - j) % R] = rows[n - 1 - j]
    q = want[:, :heads * W].view(T, heads, W)
    want[:, :heads * W] = (q / (q.square().sum(-1, keepdim=True) + 1e-6).sqrt() * 0.5).flatten(1)
    assert _rel(x, want) < 1e-6                                        # taps products and a logistic, a rounding or two each
    if taps > 1:
        assert torch.equal(after.to(F64), want_ring)


@pytest.mark.parametrize("T", [1, 3, 600, 2501])
@pytest.mark.parametrize("src,dst", [(BF, F32), (BF, BF), (F32, F32)])
@pytest.mark.parametrize("H,G,dk,dv", [(3, 3, 24, 40), (8, 2, 64, 128)])
def test_rows_without_a_rotation_and_values_in_pairs(T, src, dst, H, G, dk, dv):
    from gpustack_b200 import ops

    nq, nk, nv = H * dk, G * dk, G * dv
    p = _rnd(T, 8 + nq + nk + nv, seed=T, dtype=src)
    pos, freq = torch.arange(T, dtype=torch.int32, device="cuda") * 7, torch.tensor([0.3 ** i for i in range(dk // 2)], dtype=F64, device="cuda")
    outs = [torch.zeros(T, n + 8, dtype=dst, device="cuda") for n in (nq, nk, nv)]
    q, k, v = p[:, 8:8 + nq].to(F64), p[:, 8 + nq:8 + nq + nk].to(F64), p[:, 8 + nq + nk:].to(F64)
    tol = 6e-8 if dst == F32 else 4e-3                                 # one rounding
    ops.rot_prep(p, 8, 8 + nq, 8 + nq + nk, pos, None, *outs, H, G, dk, dv, paged=False, q_mul=0.37, k_mul=1.5)
    assert _rel(outs[0][:, :nq], q * 0.37) < tol and _rel(outs[1][:, :nk], k * 1.5) < tol and torch.equal(outs[2][:, :nv].to(F64), v)
    ops.rot_prep(p, 8, 8 + nq, 8 + nq + nk, pos, None, *outs, H, G, dk, dv, paged=False, rot_dims=dk // 16 * 16, half_layout=True,
                 freq=freq[:dk // 16 * 8].contiguous(), unit_norm=True, eps=1e-6)
    half = dk // 16 * 8
    ang = pos.to(F64)[:, None, None] * freq[:half]
    for x, n, out in ((q, H, outs[0][:, :nq]), (k, G, outs[1][:, :nk])):
        x = x.view(T, n, dk)
        a, b = x[..., :half], x[..., half:2 * half]
        y = torch.cat([a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin(), x[..., 2 * half:]], -1)
        y = y / (y.square().mean(-1, keepdim=True) + 1e-6).sqrt()
        assert _rel(out, y.flatten(1)) < max(tol, 1e-6)
    assert torch.equal(outs[2][:, :nv].to(F64), v)
    assert not any(o[:, n:].any() for o, n in zip(outs, (nq, nk, nv)))


# a head per group of lanes; then several, from 5 * 740 CTAs on: of 4, 2 and 1 groups to a warp, rounds that end inside a warp and in the middle
# of a row
@pytest.mark.parametrize("T,H,dv", [(1, 1, 32), (5, 7, 64), (2601, 9, 32), (1201, 24, 128), (13200, 9, 32), (8600, 7, 64), (9867, 3, 128), (1235, 24, 128)])
@pytest.mark.parametrize("dtype", [F32, BF])
def test_closing_step_over_many_heads(T, H, dv, dtype):
    from gpustack_b200 import ops

    o, p, w = _rnd(T, H * dv, seed=1), _rnd(T, H * dv + 16, seed=2, dtype=dtype), 1 + _rnd(H * dv, seed=3) * 0.1
    w, out = w.to(BF), torch.zeros(T, H * dv + 4, dtype=dtype, device="cuda")
    p[:, 16::5] *= 40.0                                                # gates beyond +-64 beside others
    ops.mlstm_out(o, p, 16, w, out[:, :H * dv], H, dv, 1e-5)
    y = o.to(F64).view(T, H, dv)
    y = (y / (y.square().mean(-1, keepdim=True) + 1e-5).sqrt()).flatten(1) * w.to(F64) * torch.sigmoid(p[:, 16:].to(F64))
    assert _rel(out[:, :H * dv], y) < (1e-6 if dtype == F32 else 4e-3)
    assert not out[:, H * dv:].any()


def test_gates_out_of_range_and_no_numbers():
    from gpustack_b200 import ops

    z = torch.tensor([0.0, -0.0, 1e-30, -63.9, 63.9, -64.0, 64.0, -90.0, 200.0, 3e38, -3e38, float("inf"), -float("inf"), float("nan"), 5.0, -5.0],
                     device="cuda")
    z = torch.cat([z, torch.linspace(-70, 70, 48, device="cuda")])[None]
    y = torch.ones(1, 64, device="cuda")
    out = torch.zeros(1, 64, device="cuda")
    ops.gate_norm(y, z.contiguous(), 0, torch.ones(64, dtype=BF, device="cuda"), out, 1, 0.0, gate_after=True)
    want = torch.nn.functional.silu(z.to(F64))
    want[:, 12] = float("nan")                                         # -inf times zero
    bad = torch.isnan(want) | torch.isinf(want)
    assert torch.equal(torch.isnan(out), torch.isnan(want)) and torch.equal(torch.isinf(out), torch.isinf(want))
    # four units in the last place; below x = -88.73 the exponential is infinite in fp32 and the result zero, where it is x e^x: at most
    # 88.73 * 2^-128 < 2^-121
    assert bool(((out.to(F64) - want).abs() <= 4 * 2.0 ** -23 * want.abs() + 2.0 ** -121)[~bad].all())


# pieces of whole warps: one, several and an odd number of 128s, rows that end inside a pass of the block, the widest in registers and
# the next
@pytest.mark.parametrize("C,parts", [(256, 1), (2048, 2), (2048, 1), (1152, 3), (1792, 1), (2176, 1)])
@pytest.mark.parametrize("dtype", [F32, BF])
@pytest.mark.parametrize("after", [False, True])
def test_norm_of_wide_pieces(C, parts, dtype, after):
    from gpustack_b200 import ops

    T, W = 7, C // parts
    y, p, w = _rnd(T, C, seed=1), _rnd(T, C + 8, seed=2, dtype=dtype), (1 + _rnd(W if after else C, seed=3) * 0.1).to(BF)
    y[:, :W] *= 40.0                                                   # pieces of very different size
    p[:, 8::7] *= 40.0                                                 # gates beyond +-64 beside others
    out = torch.zeros(T, C + 4, dtype=dtype, device="cuda")
    ops.gate_norm(y, p, 8, w, out[:, :C], parts, 1e-5, gate_after=after)
    g, x = torch.nn.functional.silu(p[:, 8:].to(F64)), y.to(F64)
    x = (x if after else x * g).view(T, parts, W)
    x = (x / (x.square().mean(-1, keepdim=True) + 1e-5).sqrt() * w.to(F64).view(1 if after else parts, W)).flatten(1)
    assert _rel(out[:, :C], x * g if after else x) < (1e-6 if dtype == F32 else 4e-3)
    assert not out[:, C:].any()
