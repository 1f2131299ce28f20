"""Delta rule and state space over portions in blocks of four tokens (csrc/gated_scan.cu): every width of a warp's columns, portions that
end inside a block, a stage of four blocks and the ring of four stages, against a token-by-token walk in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu

F64 = torch.float64
LENS = [1, 3, 4, 5, 15, 16, 17, 48, 63, 64, 65, 131]


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


def _inputs(lens, H, G, dk, dv, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")   # noqa: E731
    T, n, kp, vp = sum(lens), len(lens), -(-dk // 4) * 4, -(-dv // 4) * 4
    q, k, v = r(T, G, dk), r(T, G, dk), r(T, H, dv)
    k /= k.norm(dim=-1, keepdim=True)
    x = torch.zeros(T, 2 * G * kp + H * vp, device="cuda")
    x[:, :G * kp].view(T, G, kp)[..., :dk], x[:, G * kp:2 * G * kp].view(T, G, kp)[..., :dk] = q, k
    x[:, 2 * G * kp:].view(T, H, vp)[..., :dv] = v
    S = torch.zeros(n, H, dv, kp, device="cuda")
    S[..., :dk] = r(n, H, dv, dk)
    return x, q, k, v, r(T, 2 * H), S, torch.linspace(0.1, 1.0, H, device="cuda"), torch.linspace(-2.5, -1.5, H, device="cuda")


def _scan(x, gates, rate, bias, skip, lens, ctx, S, H, G, dk, dv, delta):
    from gpustack_b200 import ops

    kp, n = -(-dk // 4) * 4, len(lens)
    cu = [sum(lens[:i]) for i in range(n + 1)]
    out = torch.full((x.shape[0], H * dv), 7.0, device="cuda")
    ops.gated_scan(x, 0, G * kp, 2 * G * kp, gates if delta else gates[:, :H].contiguous(), rate, bias, skip, _i32(cu), _i32(ctx),
                   _i32(list(range(n))[::-1]), S, out, H, G, dk, dv, delta, max_len=max(2, max(lens)))
    return out


def _walk(q, k, v, gates, rate, bias, skip, lens, ctx, S, H, G, dk, delta):
    q, k = (t.to(F64).repeat_interleave(H // G, 1) for t in (q, k))
    v, gates, S = v.to(F64), gates.to(F64), S.to(F64)
    sp = torch.nn.functional.softplus((gates[:, H:] if delta else gates[:, :H]) + bias.to(F64))
    decay, step = torch.exp(-rate.to(F64) * sp), torch.sigmoid(gates[:, :H]) if delta else sp
    n, out, at = len(lens), torch.empty_like(v), 0
    first = torch.tensor([sum(lens[:i]) for i in range(n)], device="cuda")
    live = torch.tensor(lens, device="cuda")
    Z = torch.stack([S[n - 1 - i, ..., :dk] * (1.0 if ctx[i] else 0.0) for i in range(n)])
    for at in range(max(lens)):                        # token `at` of every sequence that has one
        i = (live > at).nonzero()[:, 0]
        t = first[i] + at
        z = Z[i] * decay[t][..., None, None]
        u = v[t] - torch.einsum("nhvk,nhk->nhv", z, k[t]) if delta else v[t]
        z = z + (step[t][..., None] * u)[..., None] * k[t][:, :, None]
        Z[i], out[t] = z, torch.einsum("nhvk,nhk->nhv", z, q[t]) + (0.0 if skip is None else skip.to(F64)[:, None] * v[t])
    return out.flatten(1), Z


def _rel(a, b):
    return float((a.to(F64) - b).norm() / b.norm())


# heads and copies of the portions so that each of the widths that a number of CTAs chooses runs: (16, 64), (32, 128), (32, 256)
@pytest.mark.parametrize("H,G,dk,dv,copies", [(2, 1, 14, 17, 1), (2, 2, 32, 64, 1), (2, 1, 64, 33, 1), (4, 2, 52, 64, 6), (2, 1, 90, 70, 1),
                                              (1, 1, 128, 64, 1), (4, 2, 128, 60, 1), (8, 4, 124, 64, 2), (8, 4, 128, 128, 2), (1, 1, 256, 20, 1),
                                              (4, 4, 200, 128, 2), (1, 1, 400, 40, 1), (2, 1, 24, 33, 1), (2, 1, 12, 101, 1),
                                              (8, 4, 30, 64, 1)])
@pytest.mark.parametrize("delta", [True, False])
def test_blocks_of_four(H, G, dk, dv, copies, delta):
    lens = LENS * copies
    ctx = [9 * (i % 3) for i in range(len(lens))]
    x, q, k, v, gates, S, rate, bias = _inputs(lens, H, G, dk, dv, dk + dv)
    skip = None if delta else torch.linspace(-1.0, 1.0, H, device="cuda")
    want, Z = _walk(q, k, v, gates, rate, bias, skip, lens, ctx, S, H, G, dk, delta)
    out = _scan(x, gates, rate, bias, skip, lens, ctx, S, H, G, dk, dv, delta)
    # an entry of the state takes two roundings a step, 0.29 units of 2^-23 each and independent of one another, and the error of its
    # decays, two units at most and as independent from step to step: sqrt(131 (2 * 0.29^2 + 2^2 / 3)) of 2^-23 = 1.7e-6; an output
    # averages over the entries of its row, and over rows of all lengths: half of it
    assert _rel(out, want) < 8.5e-7
    for i in range(len(lens)):
        assert _rel(S[len(lens) - 1 - i, ..., :dk], Z[i]) < 1.7e-6, lens[i]
    assert not S[..., dk:].any()


@pytest.mark.parametrize("row", [4, 5, 6, 7])
@pytest.mark.parametrize("delta", [True, False])
def test_what_is_no_number_stays_behind_its_row(row, delta):
    """... also from the rows of its own block, each of them."""
    H, G, dk, dv, lens = 2, 1, 128, 64, [40]
    x, q, k, v, gates, S, rate, bias = _inputs(lens, H, G, dk, dv, 3)
    clean = _scan(x, gates, rate, bias, None, lens, [5], S.clone(), H, G, dk, dv, delta)
    bad = x.clone()
    bad[row, 2 * G * dk:] = float("nan")
    bad[row + 9, G * dk:2 * G * dk] = float("inf")
    out = _scan(bad, gates, rate, bias, None, lens, [5], S, H, G, dk, dv, delta)
    assert torch.equal(out[:row], clean[:row])
    assert bool(torch.isnan(out[row:]).all()) and bool(torch.isnan(S).all())


@pytest.mark.parametrize("H,G,dk,dv", [(16, 16, 120, 64), (16, 16, 24, 16), (16, 8, 60, 32), (4, 4, 256, 16)])   # (128 and 64 keys: chunks)
@pytest.mark.parametrize("delta", [True, False])
def test_a_state_left_alone_decays_as_exactly_as_its_entries_are_rounded(H, G, dk, dv, delta):
    """Keys of zero: after T tokens the state is its start times the decay to the power of T, whatever four decays' product rounds to."""
    T, n = 2048, 2
    x, q, k, v, gates, S, rate, bias = _inputs([T] * n, H, G, dk, dv, 8)
    x[:, G * dk:2 * G * dk] = 0
    gates[:] = torch.randn(2 * H, generator=torch.Generator().manual_seed(5)).cuda()
    bias -= 4.0                                         # a state keeps a fifth of itself or more over the rows
    one = torch.ones(1, H, dv, dk, device="cuda")       # the decays as the kernels form them
    zero, skip = torch.zeros(1, x.shape[1], device="cuda"), torch.zeros(H, device="cuda")
    from gpustack_b200 import ops
    ops.gated_scan(zero, 0, G * dk, 2 * G * dk, gates[:1] if delta else gates[:1, :H].contiguous(), rate, bias, skip, _i32([0, 1]), _i32([1]), _i32([0]),
                   one, torch.empty(1, H * dv, device="cuda"), H, G, dk, dv, delta, max_len=1)
    g, S0 = one[0, :, 0, 0].to(F64), S.to(F64)
    out = _scan(x, gates, rate, bias, None, [T] * n, [9] * n, S, H, G, dk, dv, delta)
    want = S0 * (g ** T)[:, None, None]
    rows = torch.arange(T - 64, T, device="cuda", dtype=F64) + 1
    Q = q.to(F64).repeat_interleave(H // G, 1).view(n, T, H, dk)[:, -64:]
    read = torch.einsum("nthk,nhvk->nthv", Q, S0.flip(0)) * (g ** rows[:, None])[..., None]
    out = out.view(n, T, H, dv)[:, -64:].to(F64)
    for h in range(H):
        # T / 4 roundings of every entry by itself, 0.29 units of 2^-23 each and independent of one another: 8e-7; three times that
        assert float((S[:, h].to(F64) - want[:, h]).norm() / want[:, h].norm()) < 2.4e-6, h
        assert float((out[:, :, h] - read[:, :, h]).norm() / read[:, :, h].norm()) < 2.4e-6, h


def _steps(gates, rate, bias, H, delta):
    """The decays and steps of every row as the kernels form them in fp32: rows as sequences of one, keys of zero over a state of ones,
    and keys and values of one over a state of zeros."""
    from gpustack_b200 import ops

    T, got = gates.shape[0], []
    for key in (0.0, 1.0):
        S = torch.full((T, H, 1, 4), 1.0 - key, device="cuda")
        x = torch.full((T, 8 + H * 4), key, device="cuda")
        ops.gated_scan(x, 0, 4, 8, gates if delta else gates[:, :H].contiguous(), rate, bias, None, _i32(list(range(T + 1))), _i32([1] * T),
                       _i32(list(range(T))), S, torch.empty(T, H, device="cuda"), H, 1, 4, 1, delta, max_len=1)
        got.append(S[:, :, 0, 0])
    return got


def _fma(a, b, c):
    return (a.to(F64) * b.to(F64) + c.to(F64)).float()


def _lanes(S, x, L=16):
    """Products summed as L lanes sum them: four neighbouring entries of a lane in pairs, one chain each, then over the lanes by halves."""
    pad = -S.shape[-1] % (4 * L)
    S, x = (torch.nn.functional.pad(t, (0, pad)).unflatten(-1, (-1, L, 2, 2)) for t in (S, x))
    p = torch.zeros_like(S[..., 0, :, 0, :])
    for i in range(S.shape[-4]):
        for h in range(2):
            p = _fma(S[..., i, :, h, :], x[..., i, :, h, :], p)
    p = p[..., 0] + p[..., 1]
    while p.shape[-1] > 1:
        p = p[..., 0::2] + p[..., 1::2]
    return p[..., 0]


@pytest.mark.parametrize("dk,dv", [(124, 64), (252, 16), (60, 64), (28, 32), (16, 64)])      # (64 and 128 keys: state space goes to chunks)
@pytest.mark.parametrize("one_sign", [True, False])
@pytest.mark.parametrize("delta", [True, False])
def test_blocks_are_no_further_off_than_tokens(dk, dv, one_sign, delta):
    """... than a walk of the same decays and steps token by token in fp32, both against 64 bits."""
    H, T = 32, 160
    x, q, k, v, gates, S, rate, bias = _inputs([T], H, H, dk, dv, dk)
    S *= 0.2
    if one_sign:
        x.abs_()
        q, k, v = q.abs(), k.abs(), v.abs()
    g, b = _steps(gates, rate, bias, H, delta)
    exact, walk = S[0].to(F64), S[0].clone()
    want, tokens = torch.empty(T, H, dv, dtype=F64, device="cuda"), torch.empty(T, H, dv, device="cuda")
    for t in range(T):
        kt, gt, bt = k[t][:, None], g[t][:, None], b[t][:, None]
        exact = exact * gt.to(F64)[..., None]
        u = v[t].to(F64) - (exact * kt.to(F64)).sum(-1) if delta else v[t].to(F64)
        exact = exact + (bt.to(F64) * u)[..., None] * kt.to(F64)
        want[t] = (exact * q[t][:, None].to(F64)).sum(-1)
        u = bt * _fma(-gt, _lanes(walk, kt.expand_as(walk)), v[t]) if delta else bt * v[t]
        walk = _fma(kt, u[..., None], gt[..., None] * walk)
        tokens[t] = _lanes(walk, q[t][:, None].expand_as(walk))
    out = _scan(x, gates, rate, bias, None, [T], [9], S, H, H, dk, dv, delta)
    # ratios of norms over 32 heads' 160 x dv outputs and dk x dv entries: from draw to draw they spread by 1 % and, with 16 keys, 4 %.  Delta rule
    # over rows of one sign 0.95 to 1.015 (without the last sums' rests 1.03 to 1.16), state space 0.84 to 0.97 (without 1.09; with
    # the state scaled by rounded products 1.02 to 1.33)
    assert _rel(out.view(T, H, dv), want) < 1.02 * _rel(tokens, want)
    assert _rel(S[0], exact) < 1.04 * _rel(walk, exact)
