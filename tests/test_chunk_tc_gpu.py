"""Linear attention and mLSTM over chunks of 128 rows on the tensor cores against the recurrences in fp64: chunk edges, values that are
bf16 numbers in all, some or none of a chunk's halves (one term or three), and many items per CTA."""
import pytest
import torch

pytestmark = pytest.mark.gpu

F64 = torch.float64
# fp32 sums of at most 128 + 128 terms and a chunk's share of the state, every rounding the same way, terms without cancellation beyond 2
TOL = 2 * 300 * 2.0 ** -24
# ... as they come out, roundings of both signs: four per chunk and sum.  A product without its smallest terms (2^-17 of a number and
# more) is ten times further off.
CLOSE = 8 * 2.0 ** -24


def _linear_exact(x, S, decay, dk, dv):
    """Outputs [H, n, dv] and the state behind the rows of one sequence, in fp64, without chunks."""
    n, H, t = x.shape[0], decay.shape[0], torch.arange(x.shape[0], device="cuda", dtype=F64)
    q, k, v = (x[:, a:b].to(F64).view(n, H, -1).transpose(0, 1) for a, b in ((0, H * dk), (H * dk, 2 * H * dk), (2 * H * dk, x.shape[1])))
    d, Z = decay.to(F64)[:, None, None], S.to(F64)
    o, back = torch.empty(H, n, dv, device="cuda", dtype=F64), (t[:, None] - t).clamp(min=0)
    for h in range(H):
        D = torch.where(t[:, None] >= t, d[h] ** back, 0.0)
        o[h] = (q[h] @ k[h].mT * D) @ v[h] + d[h] ** (t[:, None] + 1) * (q[h] @ Z[h].mT)
    return o, d ** n * Z + (d ** (n - 1 - t[:, None]) * v).mT @ k


# the last three: more than six items for each of 148 CTAs, and more chunks than a table of the carry holds
@pytest.mark.parametrize("lens,H", [([128], 1), ([129], 1), ([255, 257], 2), ([700], 40), ([700, 65, 1400], 60), ([4400, 64], 3)], ids=str)
@pytest.mark.parametrize("exact", ["all", "some", "nearly", "none"])
@pytest.mark.parametrize("dk,dv", [(128, 128), (64, 64)])
def test_edges_and_terms(lens, H, exact, dk, dv):
    from gpustack_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(sum(lens) + dk)
    T, n = sum(lens), len(lens)
    x, S = torch.randn(T, 2 * H * dk + H * dv, generator=g, device="cuda"), torch.randn(n, H, dv, dk, generator=g, device="cuda")
    rows = {"all": T, "some": 70, "nearly": T, "none": 0}[exact]
    x[:rows, 2 * H * dk:] = x[:rows, 2 * H * dk:].to(torch.bfloat16).float()
    if exact == "nearly":                               # bf16 numbers but for the last bits
        x[:, 2 * H * dk:] = (x[:, 2 * H * dk:].view(torch.int32) | 0x3f).view(torch.float32)
    cu = [sum(lens[:i]) for i in range(n + 1)]
    decay = torch.linspace(0.5, 0.999, H, device="cuda")
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")   # noqa: E731
    o, S_d = torch.zeros(T, H * dv, device="cuda"), S.clone()
    ops.linattn_scan(x, 0, H * dk, 2 * H * dk, decay, i32(cu), i32([9] * n), i32(list(range(n))), S_d, o, H, dk, dv, max_len=max(lens))
    for i in range(n):
        want, Z = _linear_exact(x[cu[i]:cu[i + 1]], S[i], decay, dk, dv)
        got = o[cu[i]:cu[i + 1]].view(-1, H, dv).transpose(0, 1)
        for a, b in ((got, want), (S_d[i], Z)):         # per head
            assert float(((a.to(F64) - b).flatten(1).norm(dim=1) / b.flatten(1).norm(dim=1)).max()) < CLOSE


# chunks of 128 rows, 1, 48, 64 and 65 rows at a sequence's end, more chunks of one than a table of the carry holds (32)
MANY = [4400, 129, 300, 17, 193, 640, 1, 128]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("sign", ["both", "one"])
def test_mlstm_beyond_the_second_item_of_a_cta(dtype, sign):
    """Buffers of a CTA's items are used again from its third item on: eight items per CTA (148 of them) and more.  With queries and keys
    of one sign no denominator cancels, and the outputs are as close as the states."""
    from gpustack_b200 import ops
    from oracle import vodavik_oracle as O

    H, dk, dv, cap, n = 24, 128, 128, 6.0, len(MANY)
    cu = [sum(MANY[:i]) for i in range(n + 1)]
    T, Z = cu[-1], ops.mlstm_state_slices(dv)
    g = torch.Generator().manual_seed(3)
    proj = torch.randn(T, 2 * H * dk + H * dv, generator=g)
    if sign == "one":
        proj[:, :2 * H * dk] = proj[:, :2 * H * dk].abs()
    proj[:T // 2, 2 * H * dk:] = proj[:T // 2, 2 * H * dk:].bfloat16().float()
    proj, gates = proj.to(dtype).cuda(), (torch.randn(T, 2 * H, generator=g) * 3.0).cuda()
    bias = torch.cat([torch.randn(H, generator=g), 2 + torch.randn(H, generator=g)]).bfloat16().cuda()
    S, nn, m = (torch.randn(n, H, *w, generator=g).cuda() for w in ((dv, dk), (1, dk), (1,)))
    if sign == "one":
        nn = nn.abs()
    nn, m = nn.expand(n, H, Z, dk).contiguous(), m.abs().expand(n, H, Z).contiguous()
    o, S_d, n_d, m_d = torch.zeros(T, H * dv, device="cuda"), S.clone(), nn.clone(), m.clone()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")   # noqa: E731
    ctx = [i % 2 for i in range(n)]
    ops.mlstm_scan(proj, 0, H * dk, 2 * H * dk, gates, bias, i32(cu), i32(ctx), i32(list(range(n))), S_d, n_d, m_d, o, H, dk, dv, cap,
                   max_len=max(MANY))
    p = proj.to(F64)
    q, k, v = p[:, :H * dk].view(T, H, dk) * dk ** -0.5, p[:, H * dk:2 * H * dk].view(T, H, dk), p[:, 2 * H * dk:].view(T, H, dv)
    a = cap * torch.tanh((gates.to(F64) + bias.to(F64)) / cap)
    li, lf = a[:, :H], torch.nn.functional.logsigmoid(a[:, H:])
    for i in range(n):
        rows = slice(cu[i], cu[i + 1])
        state = (S[i].to(F64).transpose(1, 2), nn[i, :, 0].to(F64), m[i, :, 0].to(F64)) if ctx[i] else None
        with torch.device("cuda"):
            want, (Sw, nw, mw) = O.mlstm_scan(q[rows], k[rows], v[rows], li[rows], lf[rows], state)
        Sw = Sw.transpose(1, 2)
        # per head: one chunk's wrong factors are not lost among the others.  A log gate up to 6 in fp32, twice in an exponent, is 12 x 2^-24
        # of a weight; a denominator |n . q| cancels, its error is of the size of the terms
        for got, ref, tol in ((S_d[i], Sw, 17 * 2.0 ** -24), (n_d[i, :, 0], nw, 17 * 2.0 ** -24),
                              (o[rows].view(-1, H, dv).transpose(0, 1), want.transpose(0, 1),
                               17 * 2.0 ** -24 if sign == "one" else 20 * TOL)):
            err = (got.to(F64) - ref).flatten(1).norm(dim=1) / ref.flatten(1).norm(dim=1)
            assert float(err.max()) < tol, (i, MANY[i])
        assert bool((m_d[i].to(F64) - mw[:, None]).abs().max() < 17 * 2.0 ** -24 * mw.abs().max().clamp(min=6.0))


@pytest.mark.parametrize("where", ["query", "key", "value", "state", "largest key", "largest value"])
@pytest.mark.parametrize("kind,dtype", [("linear", torch.float32), ("mlstm", torch.float32), ("mlstm", torch.bfloat16)])
@pytest.mark.parametrize("H,dk,dv", [(2, 128, 128), (2, 64, 36), (160, 64, 36)])       # the last: in a CTA's second to fourth item
def test_infinite_numbers(where, kind, dtype, H, dk, dv):
    """An infinite number, and one that is infinite as a bf16 number only, gives what fp32 arithmetic gives.  Numbers of one sign in every
    column: no sum has infinities of both."""
    from gpustack_b200 import ops
    from oracle import vodavik_oracle as O

    T, cap = 300, 6.0
    g = torch.Generator().manual_seed(dk)
    q, k, v = (0.1 + 0.8 * torch.rand(T, H, w, generator=g) for w in (dk, dk, dv))
    sign = torch.tensor([1.0, -1.0]).repeat(dv)[:dv]
    v, S = v * sign, (0.1 + torch.rand(H, dv, dk, generator=g)) * sign[:, None]
    n, m = 0.1 + torch.rand(H, 1, dk, generator=g), torch.zeros(H, 1)
    if where == "query":
        q[70, -1, 3] = float("inf")
    elif where == "key":
        k[70, -1, 3] = float("inf")
    elif where == "value":
        v[200, -1, 5] = -float("inf")
    elif where == "state":
        S[-1, 7, 9] = -float("inf")
    elif where == "largest key":
        k[70, -1, 3], q[:, -1, 3] = 3.4e38, 1e-3
    else:
        v[200, -1, 5], k[200, -1] = -3.4e38, 1e-3
    x = torch.cat([t.reshape(T, -1) for t in (q, k, v)], 1).to(dtype)
    i32 = lambda t: torch.tensor(t, dtype=torch.int32, device="cuda")   # noqa: E731
    idx, o, S_d = (i32([0, T]), i32([9]), i32([0])), torch.zeros(T, H * dv, device="cuda"), S[None].cuda()
    q, k, v = (x[:, a:b].view(T, H, -1).to(F64) for a, b in ((0, H * dk), (H * dk, 2 * H * dk), (2 * H * dk, x.shape[1])))
    more = []
    if kind == "linear":
        decay = torch.linspace(0.5, 0.98, H)
        ops.linattn_scan(x.cuda(), 0, H * dk, 2 * H * dk, decay.cuda(), *idx, S_d, o, H, dk, dv, max_len=T)
        Z, want = S.to(F64), torch.zeros(T, H, dv, dtype=F64)
        for t in range(T):
            Z = decay.to(F64)[:, None, None] * Z + v[t][:, :, None] * k[t][:, None]
            want[t] = torch.einsum("hvk,hk->hv", Z, q[t])
    else:
        slices = ops.mlstm_state_slices(dv)
        gates, bias = torch.randn(T, 2 * H, generator=g), torch.cat([torch.zeros(H), torch.linspace(3, 5, H)]).bfloat16()
        n_d, m_d = n.expand(H, slices, dk)[None].contiguous().cuda(), m.expand(H, slices)[None].contiguous().cuda()
        ops.mlstm_scan(x.cuda(), 0, H * dk, 2 * H * dk, gates.cuda(), bias.cuda(), *idx, S_d, n_d, m_d, o, H, dk, dv, cap, max_len=T)
        a = cap * torch.tanh((gates.to(F64) + bias.to(F64)) / cap)
        want, (Z, nw, _) = O.mlstm_scan(q * dk ** -0.5, k, v, a[:, :H], torch.nn.functional.logsigmoid(a[:, H:]),
                                        (S.to(F64).transpose(1, 2), n[:, 0].to(F64), m[:, 0].to(F64)))
        Z, more = Z.transpose(1, 2), [(n_d[0, :, 0], nw)]
    for got, ref in [(o, want.reshape(T, -1)), (S_d[0], Z)] + more:
        got = got.cpu().to(F64)
        assert torch.equal(got.isnan(), ref.isnan()) and torch.equal(got == float("inf"), ref == float("inf"))
        assert torch.equal(got == -float("inf"), ref == -float("inf"))
        a, b = (t[ref.isfinite()] for t in (got, ref))
        assert bool(((a - b).abs() <= TOL * b.abs()).all())


@pytest.mark.parametrize("kind,dtype", [("linear", torch.float32), ("mlstm", torch.float32), ("mlstm", torch.bfloat16)])
@pytest.mark.parametrize("how", ["one after the other", "captured"])
def test_launches_that_begin_early(kind, dtype, how):
    """Steps of other lengths over one workspace with nothing between them, or in one captured graph, give what they give alone."""
    from gpustack_b200 import config, ops

    H, dk, dv = 3, 128, 128
    steps = [[130], [700, 40], [64, 65, 1], [300] + [1] * 20, [2500], [129]] * 4       # chunks also beside a one-pass kernel
    g = torch.Generator(device="cuda").manual_seed(1)
    draw = lambda *s: torch.randn(*s, generator=g, device="cuda")   # noqa: E731
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")   # noqa: E731
    ws = torch.empty(config.chunk_scan_floats(4096, 32, H, dk, dv), device="cuda")
    calls, states = [], []
    for lens in steps:
        T, n, Z = sum(lens), len(lens), ops.mlstm_state_slices(dv)
        x, o, gates = draw(T, 3 * H * dk).to(dtype), torch.zeros(T, H * dv, device="cuda"), draw(T, 2 * H)
        idx = (i32([sum(lens[:i]) for i in range(n + 1)]), i32([9] * n), i32(list(range(n))))
        S, more = draw(n, H, dv, dk), [draw(n, H, 1, dk).expand(n, H, Z, dk).contiguous(), torch.zeros(n, H, Z, device="cuda")]
        decay, bias = torch.linspace(0.9, 0.999, H, device="cuda"), torch.linspace(-1, 3, 2 * H).bfloat16().cuda()
        cols = (0, H * dk, 2 * H * dk)
        if kind == "linear":
            more = []
            call = lambda x=x, i=idx, S=S, o=o, L=max(lens), d=decay: ops.linattn_scan(x, *cols, d, *i, S, o, H, dk, dv, max_len=L,   # noqa: E731
                                                                                       workspace=ws)
        else:
            call = lambda x=x, i=idx, S=S, o=o, L=max(lens), m=more, b=bias, gt=gates: ops.mlstm_scan(   # noqa: E731
                x, *cols, gt, b, *i, S, *m, o, H, dk, dv, 6.0, max_len=L, workspace=ws)
        calls.append(call)
        states.append([o, S] + more)
    start = [[t.clone() for t in s] for s in states]
    real, ops.chunk_scan_pays = ops.chunk_scan_pays, lambda *a: True
    try:
        want = []
        for call, s, s0 in zip(calls, states, start):
            call()
            torch.cuda.synchronize()
            want.append([t.clone() for t in s])
            [a.copy_(b) for a, b in zip(s, s0)]
        torch.cuda.synchronize()
        if how == "captured":
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                for call in calls:
                    call()
            graph.replay()
        else:
            for call in calls:
                call()
        torch.cuda.synchronize()
    finally:
        ops.chunk_scan_pays = real
    assert all(torch.equal(a, b) for s, w in zip(states, want) for a, b in zip(s, w))


@pytest.mark.parametrize("dk,dv", [(128, 128), (64, 64)])
def test_sums_of_one_sign(dk, dv):
    """What the products cut from a sum does not add up: over rows of one sign the mean deviation of outputs and states is below half a
    unit of fp32's last place (2^-24), and their error that of a few roundings."""
    from gpustack_b200 import ops

    H, lens = 2, [2048, 300]
    T, cu = sum(lens), [0, lens[0], sum(lens)]
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(T, H * (2 * dk + dv), generator=g, device="cuda").abs()
    S, decay = torch.randn(2, H, dv, dk, generator=g, device="cuda").abs(), torch.tensor([0.9, 0.99], device="cuda")
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")   # noqa: E731
    o, S_d = torch.zeros(T, H * dv, device="cuda"), S.clone()
    ops.linattn_scan(x, 0, H * dk, 2 * H * dk, decay, i32(cu), i32([9, 9]), i32([0, 1]), S_d, o, H, dk, dv, max_len=lens[0])
    for i, n in enumerate(lens):
        rows = slice(cu[i], cu[i + 1])
        want_o, want_S = _linear_exact(x[rows], S[i], decay, dk, dv)
        for got, want in ((o[rows].view(n, H, dv).transpose(0, 1), want_o), (S_d[i], want_S)):
            off = got.to(F64) - want
            assert float((off.flatten(1).sum(1).abs() / want.flatten(1).sum(1)).max()) < 2.0 ** -24
            assert float((off.flatten(1).norm(dim=1) / want.flatten(1).norm(dim=1)).max()) < 2.0 ** -23


@pytest.mark.parametrize("kind", ["linear", "mlstm"])
@pytest.mark.parametrize("lens,H", [([64] * 20 + [33] * 10, 2), ([17] * 70 + [200], 1), ([40], 1), ([40, 41], 1), ([1] * 30 + [130] * 3, 3)],
                         ids=["short", "shortest", "one", "two", "singles"])
def test_a_workspace_of_the_documented_size(kind, lens, H):
    """Portions too short for all sequences' chunks to fit at once: in groups, within the workspace, with the same results."""
    from gpustack_b200 import config, ops

    dk = dv = 64
    T, n, Z = sum(lens), len(lens), ops.mlstm_state_slices(dv)
    floats = config.chunk_scan_floats(T, n, H, dk, dv)
    g = torch.Generator(device="cuda").manual_seed(T)
    draw = lambda *s: torch.randn(*s, generator=g, device="cuda")   # noqa: E731
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")   # noqa: E731
    x, gates, S0, n0 = draw(T, 3 * H * dk), draw(T, 2 * H), draw(n, H, dv, dk), draw(n, H, 1, dk)
    idx = (i32([sum(lens[:i]) for i in range(n + 1)]), i32([i % 3 for i in range(n)]), i32(list(range(n))[::-1]))
    real, out = ops.chunk_scan_pays, []
    for chunks in (True, False):
        ws = torch.full((floats + 4096,), 7.0, device="cuda")
        o, S, more = torch.zeros(T, H * dv, device="cuda"), S0.clone(), []
        ops.chunk_scan_pays = lambda *a: chunks
        try:
            if kind == "linear":
                ops.linattn_scan(x, 0, H * dk, 2 * H * dk, torch.linspace(0.9, 0.99, H, device="cuda"), *idx, S, o, H, dk, dv, max_len=max(lens),
                                 workspace=ws[:floats])
            else:
                more = [n0.expand(n, H, Z, dk).contiguous(), torch.zeros(n, H, Z, device="cuda")]
                ops.mlstm_scan(x, 0, H * dk, 2 * H * dk, gates, torch.linspace(-1, 3, 2 * H).bfloat16().cuda(), *idx, S, *more, o, H, dk, dv, 6.0,
                               max_len=max(lens), workspace=ws[:floats])
        finally:
            ops.chunk_scan_pays = real
        assert bool((ws[floats:] == 7.0).all()) and bool((ws[:floats] == 7.0).all()) == (not chunks or lens == [40])
        out.append([o, S] + more)
    for a, b in zip(*out):                              # two roundings' worth of either side's
        assert float((a - b).norm() / b.norm().clamp(min=1.0)) < (40 if kind == "mlstm" else 2) * TOL
