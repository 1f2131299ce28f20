"""The recurrences with all chunks of a prompt portion side by side, against the recurrences themselves in fp64: chunk edges, short
and single rows beside long portions, states carried in slots, value widths that fill no tile, a skipped sequence."""
import pytest
import torch

pytestmark = pytest.mark.gpu

F64 = torch.float64
# rows of a step's sequences: one chunk, its edges, a remainder of one row, portions that stay one-pass beside long ones
LENS = [[64], [65], [127], [17, 128, 16, 1, 300], [1, 1, 449], [63, 64, 65]]
# fp32 sums of at most dk + 64 + (a chunk's share of the state) terms of one size, each rounded: |error| <= 300 * 2^-24 of the
# terms' norm when all roundings point the same way; the outputs are sums of that kind without cancellation beyond a factor of 2
TOL = 2 * 300 * 2.0 ** -24


def _rel(a, b):
    return float((a.cpu().to(F64) - b).norm() / b.norm())


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


def _layout(lens):
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    ctx = [0 if i % 2 else 40 for i in range(len(lens))]
    slots = list(range(len(lens)))[::-1]
    return cu, ctx, slots


@pytest.mark.parametrize("lens", LENS, ids=str)
@pytest.mark.parametrize("H,dk,dv", [(2, 64, 64), (1, 128, 128), (2, 64, 132), (1, 128, 36)])
def test_linear_chunks(lens, H, dk, dv):
    from gpustack_b200 import ops

    g = torch.Generator().manual_seed(sum(lens) + dk + dv)
    cu, ctx, slots = _layout(lens)
    T = cu[-1]
    x = torch.randn(T, 2 * H * dk + H * dv, generator=g)
    S = torch.randn(len(lens), H, dv, dk, generator=g)
    decay = torch.tensor([0.98, 0.5][:H])
    o, S_d = torch.zeros(T, H * dv, device="cuda"), S.cuda()
    ops.linattn_scan(x.cuda(), 0, H * dk, 2 * H * dk, decay.cuda(), _i32(cu), _i32(ctx), _i32(slots), S_d, o, H, dk, dv, max_len=4096)
    q, k = x[:, :H * dk].view(T, H, dk).to(F64), x[:, H * dk:2 * H * dk].view(T, H, dk).to(F64)
    v = x[:, 2 * H * dk:].view(T, H, dv).to(F64)
    want, S_want = torch.zeros(T, H, dv, dtype=F64), S.to(F64)
    for i in range(len(lens)):
        Z = S_want[slots[i]].clone() * (1.0 if ctx[i] else 0.0)
        for t in range(cu[i], cu[i + 1]):
            Z = decay.to(F64)[:, None, None] * Z + v[t][:, :, None] * k[t][:, None]
            want[t] = torch.einsum("hvk,hk->hv", Z, q[t])
        S_want[slots[i]] = Z
    assert _rel(o, want.view(T, -1)) < TOL
    assert _rel(S_d, S_want) < TOL


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("lens", LENS, ids=str)
@pytest.mark.parametrize("H,dk,dv", [(2, 64, 64), (1, 128, 128), (2, 64, 132), (1, 128, 36)])
def test_mlstm_chunks(lens, H, dk, dv, dtype):
    from gpustack_b200 import ops
    from oracle import vodavik_oracle as O

    g = torch.Generator().manual_seed(sum(lens) + dk + dv)
    cu, ctx, slots = _layout(lens)
    T, n_seq, Z, cap = cu[-1], len(lens), ops.mlstm_state_slices(dv), 6.0
    proj = torch.randn(T, 2 * H * dk + H * dv, generator=g).to(dtype)
    gates = torch.randn(T, 2 * H, generator=g) * 3.0
    bias = torch.cat([torch.randn(H, generator=g), 2 + torch.randn(H, generator=g)]).to(torch.bfloat16)
    S = torch.randn(n_seq, H, dv, dk, generator=g)
    n = torch.randn(n_seq, H, 1, dk, generator=g).expand(n_seq, H, Z, dk).contiguous()
    m = torch.rand(n_seq, H, 1, generator=g).expand(n_seq, H, Z).contiguous()
    o, S_d, n_d, m_d = torch.zeros(T, H * dv, device="cuda"), S.cuda(), n.cuda(), m.cuda()
    ops.mlstm_scan(proj.cuda(), 0, H * dk, 2 * H * dk, gates.cuda(), bias.cuda(), _i32(cu), _i32(ctx), _i32(slots), S_d, n_d, m_d, o, H, dk,
                   dv, cap, max_len=4096)
    p = proj.to(F64)
    q, k = p[:, :H * dk].view(T, H, dk) * dk ** -0.5, p[:, H * dk:2 * H * dk].view(T, H, dk)
    v = p[:, 2 * H * dk:].view(T, H, dv)
    a = cap * torch.tanh((gates.to(F64) + bias.to(F64)) / cap)
    li, lf = a[:, :H], torch.nn.functional.logsigmoid(a[:, H:])
    want = torch.zeros(T, H, dv, dtype=F64)
    for i in range(n_seq):
        rows, at = slice(cu[i], cu[i + 1]), slots[i]
        state = (S[at].to(F64).transpose(1, 2), n[at, :, 0].to(F64), m[at, :, 0].to(F64)) if ctx[i] else None
        want[rows], (Sw, nw, mw) = O.mlstm_scan(q[rows], k[rows], v[rows], li[rows], lf[rows], state)
        assert _rel(S_d[at], Sw.transpose(1, 2)) < TOL
        assert all(_rel(n_d[at, :, z], nw) < TOL for z in range(Z)) and all(_rel(m_d[at, :, z], mw) < TOL for z in range(Z))
    # a denominator |n . q| cancels: its error is of the size of the terms, so rows are compared by the same norm as a whole
    assert _rel(o, want.reshape(T, -1)) < 20 * TOL


@pytest.mark.parametrize("lens", LENS, ids=str)
@pytest.mark.parametrize("H,dk,dv", [(2, 64, 128), (1, 128, 64), (2, 64, 132)])
def test_gated_linear_chunks(lens, H, dk, dv):
    """Decays per key channel from nearly 1 to exactly 0 (a channel cleared in the middle of a chunk)."""
    from gpustack_b200 import ops

    g = torch.Generator().manual_seed(sum(lens) + dk + dv)
    cu, ctx, slots = _layout(lens)
    T = cu[-1]
    x, z = torch.randn(T, 2 * H * dk + H * dv, generator=g), torch.randn(T, H * dk, generator=g) * 4 + 1
    z[T // 2, ::3] = -1.0e5
    S = torch.randn(len(lens), H, dv, dk, generator=g)
    o, S_d = torch.zeros(T, H * dv, device="cuda"), S.cuda()
    ops.gla_scan(x.cuda(), 0, H * dk, 2 * H * dk, z.cuda(), 1.0 / 16, _i32(cu), _i32(ctx), _i32(slots), S_d, o, H, dk, dv, max_len=4096)
    q, k = x[:, :H * dk].view(T, H, dk).to(F64), x[:, H * dk:2 * H * dk].view(T, H, dk).to(F64)
    v = x[:, 2 * H * dk:].view(T, H, dv).to(F64)
    alpha = torch.exp(torch.nn.functional.logsigmoid(z.to(F64)) / 16).view(T, H, dk)
    want, S_want = torch.zeros(T, H, dv, dtype=F64), S.to(F64)
    for i in range(len(lens)):
        Z = S_want[slots[i]].clone() * (1.0 if ctx[i] else 0.0)
        for t in range(cu[i], cu[i + 1]):
            Z = alpha[t][:, None] * Z + v[t][:, :, None] * k[t][:, None]
            want[t] = torch.einsum("hvk,hk->hv", Z, q[t])
        S_want[slots[i]] = Z
    assert _rel(o, want.view(T, -1)) < TOL
    assert _rel(S_d, S_want) < TOL


@pytest.mark.parametrize("lens", LENS, ids=str)
@pytest.mark.parametrize("H,G,dk,dv,skip", [(4, 2, 128, 64, True), (2, 1, 64, 128, False), (2, 2, 128, 36, True)])
def test_state_space_chunks(lens, H, G, dk, dv, skip):
    from gpustack_b200 import ops

    g = torch.Generator().manual_seed(sum(lens) + dk + dv)
    cu, ctx, slots = _layout(lens)
    T = cu[-1]
    x = torch.randn(T, 2 * G * dk + H * dv, generator=g)
    gates, rate, dt = torch.randn(T, H, generator=g), torch.rand(H, generator=g), torch.randn(H, generator=g) - 2
    D = torch.randn(H, generator=g) if skip else None
    S = torch.randn(len(lens), H, dv, dk, generator=g)
    o, S_d = torch.zeros(T, H * dv, device="cuda"), S.cuda()
    ops.gated_scan(x.cuda(), 0, G * dk, 2 * G * dk, gates.cuda(), rate.cuda(), dt.cuda(), None if D is None else D.cuda(), _i32(cu), _i32(ctx),
                   _i32(slots), S_d, o, H, G, dk, dv, False, max_len=4096)
    q, k = (x[:, c:c + G * dk].view(T, G, dk).to(F64).repeat_interleave(H // G, 1) for c in (0, G * dk))
    v = x[:, 2 * G * dk:].view(T, H, dv).to(F64)
    step = torch.nn.functional.softplus(gates.to(F64) + dt.to(F64))
    want, S_want = torch.zeros(T, H, dv, dtype=F64), S.to(F64)
    for i in range(len(lens)):
        Z = S_want[slots[i]].clone() * (1.0 if ctx[i] else 0.0)
        for t in range(cu[i], cu[i + 1]):
            Z = torch.exp(-rate.to(F64) * step[t])[:, None, None] * Z + (step[t][:, None] * v[t])[:, :, None] * k[t][:, None]
            want[t] = torch.einsum("hvk,hk->hv", Z, q[t]) + (D.to(F64)[:, None] * v[t] if skip else 0.0)
        S_want[slots[i]] = Z
    assert _rel(o, want.view(T, -1)) < TOL
    assert _rel(S_d, S_want) < TOL


def test_no_row_reaches_an_earlier_one_and_negative_slots_are_skipped():
    from gpustack_b200 import ops

    H, dk, dv, T = 1, 64, 64, 200
    x = torch.randn(T, 2 * dk + dv, generator=torch.Generator().manual_seed(5))
    x[70, 2 * dk:] = float("nan")
    x[130, dk:2 * dk] = float("inf")
    S = torch.full((2, H, dv, dk), 3.0, device="cuda")
    o = torch.full((T + 100, H * dv), 7.0, device="cuda")
    xx = torch.cat([x, torch.randn(100, 2 * dk + dv, generator=torch.Generator().manual_seed(6))]).cuda()
    ops.linattn_scan(xx, 0, dk, 2 * dk, torch.tensor([0.9]).cuda(), _i32([0, T, T + 100]), _i32([0, 5]), _i32([1, -1]), S, o, H, dk, dv, max_len=T)
    assert bool(torch.isfinite(o[:70]).all()) and bool(torch.isnan(o[70:T]).all())
    assert bool((o[T:] == 7.0).all()) and bool((S[0] == 3.0).all())


def _scans(x, gates, z, cu, ctx, slots, H, dk, dv, max_len, n_seq=None):
    """Every recurrence over the same rows; state slots start alike.  -> {name: (outputs, *states)}"""
    from gpustack_b200 import ops

    T, n, Z = x.shape[0], n_seq or len(slots), ops.mlstm_state_slices(dv)
    cols, idx, out = (0, H * dk, 2 * H * dk), (_i32(cu), _i32(ctx), _i32(slots)), {}
    g = torch.Generator().manual_seed(11)
    S0, n0, m0 = torch.randn(n, H, dv, dk, generator=g), torch.randn(n, H, 1, dk, generator=g), torch.rand(n, H, 1, generator=g)
    vec = lambda lo: torch.linspace(lo, lo + 0.3, H).cuda()   # noqa: E731
    bias = torch.linspace(-1, 3, 2 * H).to(torch.bfloat16).cuda()
    for name in ("linear", "mlstm", "gated_linear", "state_space"):
        o, S = torch.full((T, H * dv), 7.0, device="cuda"), S0.cuda()
        more = ()
        if name == "linear":
            ops.linattn_scan(x, *cols, vec(0.6), *idx, S, o, H, dk, dv, max_len=max_len)
        elif name == "mlstm":
            more = (n0.expand(n, H, Z, dk).contiguous().cuda(), m0.expand(n, H, Z).contiguous().cuda())
            ops.mlstm_scan(x, *cols, gates, bias, *idx, S, *more, o, H, dk, dv, 6.0, max_len=max_len)
        elif name == "gated_linear":
            ops.gla_scan(x, *cols, z, 1.0 / 16, *idx, S, o, H, dk, dv, max_len=max_len)
        else:
            ops.gated_scan(x, *cols, gates[:, :H].contiguous(), vec(0.3), vec(-2.0), vec(0.5), *idx, S, o, H, H, dk, dv, False, max_len=max_len)
        out[name] = (o, S) + more
    return out


def _rows(T, H, dk, dv, seed):
    g = torch.Generator().manual_seed(seed)
    return tuple(torch.randn(T, w, generator=g).cuda() for w in (2 * H * dk + H * dv, 2 * H, H * dk))


@pytest.mark.parametrize("n", [1, 10, 16, 17, 70])
def test_one_sequence_in_a_longer_buffer(n):
    """The buffer's rows say nothing about the sequence's: a short one beside nothing is not left out."""
    H, dk, dv, T = 2, 64, 64, 600
    x, gates, z = _rows(T, H, dk, dv, n)
    long = _scans(x, gates, z, [0, n], [5], [0], H, dk, dv, T)
    alone = _scans(x[:n].contiguous(), gates[:n].contiguous(), z[:n].contiguous(), [0, n], [5], [0], H, dk, dv, n)
    for name, got in long.items():
        assert bool((got[0][n:] == 7.0).all())
        assert _rel(got[0][:n], alone[name][0].cpu().to(F64)) < (20 if name == "mlstm" else 1) * TOL, name
        for a, b in zip(got[1:], alone[name][1:]):
            assert _rel(a, b.cpu().to(F64)) < TOL, name


def test_mlstm_stabilisers_of_more_value_slices_than_keys():
    """Every slice's copy of the stabiliser is written, also where there are more slices (value columns / 32) than key columns."""
    H, dk, dv, T = 1, 64, 2084, 130
    x, gates, z = _rows(T, H, dk, dv, 3)
    for n in (T, 90):
        m = _scans(x, gates, z, [0, n], [5], [0], H, dk, dv, 4096)["mlstm"][3]
        assert bool((m == m[..., :1]).all())


@pytest.mark.parametrize("row", [70, 71])
def test_what_is_no_number_reaches_no_earlier_row(row):
    """A gate (or, without gates, a key) that is no number and an infinite value behind it: rows before stay as they are."""
    H, dk, dv, T = 2, 64, 64, 400
    x, gates, z = _rows(T, H, dk, dv, 7)
    clean = _scans(x, gates, z, [0, T], [5], [0], H, dk, dv, 4096)
    gates[row], z[row] = float("nan"), float("nan")
    x[row + 60, 2 * H * dk:] = float("inf")
    xk = x.clone()
    xk[row, H * dk:2 * H * dk] = float("nan")
    got = _scans(x, gates, z, [0, T], [5], [0], H, dk, dv, 4096)
    got["linear"] = _scans(xk, gates, z, [0, T], [5], [0], H, dk, dv, 4096)["linear"]
    for name, out in got.items():
        assert torch.equal(out[0][:row], clean[name][0][:row]), name
        assert bool(torch.isnan(out[0][row:]).all()) and bool(torch.isnan(out[1]).all()), name


def test_a_state_space_row_that_clears_the_state():
    """A step whose rate times size overflows fp32 clears the state; what comes behind it knows only what came behind it."""
    from gpustack_b200 import ops

    dk, dv, T = 64, 64, 300
    g = torch.Generator().manual_seed(9)
    x, gates, S = torch.randn(T, 2 * dk + dv, generator=g), torch.randn(T, 1, generator=g) * 0.5 - 87.0, torch.randn(1, 1, dv, dk, generator=g)
    gates[100] = 50.0
    rate, dt = torch.tensor([1.0e38]), torch.zeros(1)
    o, S_d = torch.zeros(T, dv, device="cuda"), S.cuda()
    ops.gated_scan(x.cuda(), 0, dk, 2 * dk, gates.cuda(), rate.cuda(), dt.cuda(), None, _i32([0, T]), _i32([9]), _i32([0]), S_d, o, 1, 1, dk, dv,
                   False, max_len=4096)
    step, Z, want = torch.nn.functional.softplus(gates.to(F64))[:, 0], S[0, 0].to(F64), torch.zeros(T, dv, dtype=F64)
    x = x.to(F64)
    for t in range(T):
        Z = torch.exp(-1.0e38 * step[t]) * Z + step[t] * x[t, 2 * dk:, None] * x[t, None, dk:2 * dk]
        want[t] = Z @ x[t, :dk]
    # the steps are formed from numbers of 2^-126, whose rounding is 2^-22 of them, and scaled by the rate in the exponent
    for a, b in ((0, 100), (100, 104)):
        assert _rel(o[a:b], want[a:b]) < TOL
    assert bool(torch.isfinite(o).all()) and bool(torch.isfinite(S_d).all())


# beyond the carry's eight chunks in flight, with its remainder and a second walk; more sequences than a warp looks up at once, long
# ones before, between and behind single rows
@pytest.mark.parametrize("lens", [[513], [577, 1100], [1] * 3 + [150] + [1] * 40 + [200, 17] + [1] * 20, [1] * 33 + [130]], ids=lambda v: str(len(v)))
def test_long_portions_and_many_sequences(lens):
    """The chunk form against the one-pass form, sequence by sequence (which the other tests hold against fp64)."""
    H, dk, dv = 2, 64, 64
    cu, ctx, slots = _layout(lens)
    x, gates, z = _rows(cu[-1], H, dk, dv, len(lens))
    got = _scans(x, gates, z, cu, ctx, slots, H, dk, dv, 4096)
    for i, n in enumerate(lens):
        a, b = cu[i], cu[i + 1]
        want = _scans(x[a:b].contiguous(), gates[a:b].contiguous(), z[a:b].contiguous(), [0, n], [ctx[i]], [slots[i]], H, dk, dv, min(n, 30),
                      n_seq=len(lens))
        for name in got:
            # both sides' sums are rounded, and an output's error is of the size of the sequence's outputs
            assert _rel(got[name][0][a:b], want[name][0].cpu().to(F64)) < (40 if name == "mlstm" else 2) * TOL, (name, i)
            for p, q in zip(got[name][1:], want[name][1:]):
                assert _rel(p[slots[i]], q[slots[i]].cpu().to(F64)) < 2 * TOL, (name, i)
