"""What the engine is measured on: the layers that a serving step spends its time in, each through the entry point that the
model runners call, and one whole engine step sequence.  `listed()` is the fixed list, `draw()` gives more of the same kinds
and ranges; sizes are those of the model families' benchmark (width 2048: 16 / 4 heads of 128, the latent, recurrent and
routed layers beside them) and of the 8-billion-parameter serving benchmark (width 4096, 32 / 8 heads of 128, 512-token
prompts, 256 sequences).

kinds:
  attention_prefill   causal attention of prompt portions over the paged cache
  attention_decode    one new row per sequence over the paged cache, keys split over CTAs
  mlp                 add + RMS norm -> gate / up product with SiLU -> down product (split sums) -> add + RMS norm
  routed              router product -> choice -> grouping -> expert products -> combine
  latent_prefill      latent cache rows and rotations -> per-head absorption -> attention -> per-head values
  latent_decode       the same for one new row per sequence
  mlstm               matrix-memory recurrence with its gates -> head norm and output gate
  linear              rotation -> linear attention with a fixed decay -> head norm and gate
  gated_linear        factors -> decay projection -> linear attention with a decay per channel -> head norm and gate
  delta               short convolution and unit norms -> gated delta rule -> head norm and gate
  state_space         short convolution -> state-space recurrence -> gated norm
  engine              prompts, then decode steps, through the engine; returns every step's logits
"""
from __future__ import annotations

import math

import torch

from gpustack_b200 import ops

BF, F32, F64 = torch.bfloat16, torch.float32, torch.float64
PAGE = 16
MLP = {2048: 8192, 4096: 14336}                      # width -> feed-forward width
HEADS = {"8b": (32, 8, 128), "2k": (16, 4, 128), "half": (14, 2, 64)}
LATENT = (16, 512, 64, 128, 128)                     # heads, latent, rotated part, unrotated part, value width
ROUTED = (2048, 2048, 8, 2)                          # width, expert width, experts, chosen
RECURRENT = (8, 128, 128)                            # heads, key width, value width
GATED = (8, 64, 128, 16)                             # heads, key width, value width, rank of the decay projection
DELTA = (16, 8, 128, 128, 4)                         # value heads, key heads, key width, value width, taps
SPACE = (32, 2, 128, 64, 4)                          # heads, groups, state, head width, taps
ENGINE = (2048, 8192, 2, 16, 4, 128, 32000)          # width, feed-forward, layers, heads, kv heads, head width, vocabulary


def listed():
    return [
        # a chat's next tokens, few sequences: launches and latency count more than bytes
        {"name": "engine 3 requests", "kind": "engine", "seqs": 3, "tokens": 243, "steps": 4},
        # the smallest call of the list: one sequence's next token over its own cache
        {"name": "attention decode 1", "kind": "attention_decode", "heads": "8b", "seqs": 1, "context": 3001},
        # the serving benchmark's decode step: 256 sequences in the middle of their answers
        {"name": "attention decode 256", "kind": "attention_decode", "heads": "8b", "seqs": 256, "context": 576},
        # the serving benchmark's prompt step
        {"name": "attention prefill 16x512", "kind": "attention_prefill", "heads": "8b", "seqs": 16, "tokens": 8192, "ragged": False,
         "context": 0},
        # the feed-forward of the benchmark's decode step
        {"name": "mlp 256", "kind": "mlp", "width": 4096, "tokens": 256},
        # a routed layer's decode step
        {"name": "routed 64", "kind": "routed", "tokens": 64},
        # prompts of a latent-attention layer
        {"name": "latent prefill 4x2048", "kind": "latent_prefill", "seqs": 4, "tokens": 8192, "ragged": False, "context": 0},
        # its decode step
        {"name": "latent decode 64", "kind": "latent_decode", "seqs": 64, "context": 2048},
        # recurrent layers over prompts of mixed lengths, some of them continued from a state
        {"name": "mlstm ragged", "kind": "mlstm", "seqs": 7, "tokens": 7919, "ragged": True, "context": 640, "f32": False},
        {"name": "linear prefill 4x2048", "kind": "linear", "seqs": 4, "tokens": 8192, "ragged": False, "context": 0, "f32": False},
        {"name": "gated linear ragged", "kind": "gated_linear", "seqs": 5, "tokens": 6007, "ragged": True, "context": 512, "f32": False},
        {"name": "delta prefill 4x2048", "kind": "delta", "seqs": 4, "tokens": 8192, "ragged": False, "context": 0, "f32": False},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 50)


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(["attention_prefill", "attention_decode", "mlp", "routed", "latent_prefill", "latent_decode", "mlstm", "linear",
                           "gated_linear", "delta", "state_space", "engine"])
        c = {"kind": kind}
        if kind == "engine":
            c.update(seqs=rng.randint(1, 8), steps=rng.randint(1, 6))
            c["tokens"] = c["seqs"] * _log(rng, 8, 300) + rng.randint(0, c["seqs"])
        elif kind == "mlp":
            c.update(width=rng.choice(sorted(MLP)), tokens=_log(rng, 1, 4096))
        elif kind == "routed":
            c.update(tokens=_log(rng, 1, 4096))
        elif kind in ("attention_decode", "latent_decode"):
            c.update(seqs=_log(rng, 1, 256), context=_log(rng, 16, 8000))
            if kind == "attention_decode":
                c["heads"] = rng.choice(sorted(HEADS))
        else:
            c.update(seqs=rng.randint(1, 16), ragged=rng.random() < 0.6, context=rng.choice([0, _log(rng, 1, 2048)]))
            c["tokens"] = c["seqs"] * _log(rng, 1, 4096 // min(c["seqs"], 4)) if rng.random() < 0.8 else c["seqs"]
            if c["ragged"]:
                c["tokens"] += rng.randint(0, 2 * c["seqs"])
            c["tokens"] = min(c["tokens"], 8192)
            if kind == "attention_prefill":
                c["heads"] = rng.choice(sorted(HEADS))
            elif kind != "latent_prefill":
                c["f32"] = rng.random() < 0.15
        if _cost(c) <= most:
            return c


# ------------------------------------------------------------------------------------------- shared layout
def _lens(case):
    """New rows of every sequence: equal, or mixed in a fixed way; at least one each."""
    n, total = case["seqs"], case["tokens"]
    if not case.get("ragged"):
        return [total // n + (1 if i < total % n else 0) for i in range(n)]
    w = [1 + (5 * i + 3) % 7 for i in range(n)]
    out = [1 + (total - n) * x // sum(w) for x in w]
    out[0] += total - sum(out)
    return out


def _contexts(case):
    """Rows that came before: none for every other sequence, so that new and continued ones share a step."""
    c = case.get("context", 0)
    return [0 if c == 0 or i % 2 else max(1, c * (i + 2) // (case["seqs"] + 1)) for i in range(case["seqs"])]


class _Random:
    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(seed)

    def __call__(self, *shape, scale=1.0, dtype=BF):
        return (torch.randn(*shape, generator=self.g, device="cuda", dtype=F32) * scale).to(dtype)

    def uniform(self, *shape, low=0.0, high=1.0):
        return torch.rand(*shape, generator=self.g, device="cuda", dtype=F32) * (high - low) + low

    def order(self, n):
        return torch.randperm(n, generator=self.g, device="cuda").to(torch.int32)


def _i32(x):
    return torch.as_tensor(x, dtype=torch.int32, device="cuda")


def _starts(lens):
    out = [0]
    for n in lens:
        out.append(out[-1] + n)
    return out


def _pages(r, totals):
    """A block table over pages in a mixed order (page 0 stays empty), and the number of pages."""
    need = [(n + PAGE - 1) // PAGE for n in totals]
    order = r.order(sum(need)) + 1
    table = torch.zeros(len(totals), max(need), dtype=torch.int32, device="cuda")
    at = 0
    for i, n in enumerate(need):
        table[i, :n] = order[at:at + n]
        at += n
    return table, sum(need) + 1


def _slots(table, lens, contexts):
    rows = [table[i].long()[torch.arange(c, c + n, device="cuda") // PAGE] * PAGE + torch.arange(c, c + n, device="cuda") % PAGE
            for i, (n, c) in enumerate(zip(lens, contexts))]
    return torch.cat(rows).to(torch.int32)


def _positions(lens, contexts):
    return torch.cat([torch.arange(c, c + n, device="cuda") for n, c in zip(lens, contexts)]).to(torch.int32)


def _freq(dims, base):
    return torch.tensor([base ** (-2.0 * i / dims) for i in range(dims // 2)], dtype=F64, device="cuda")


def _inputs(case, seed):
    """Everything that comes from the seed, in plain torch."""
    return _INPUTS[case["kind"]](case, _Random(seed))


def _act(case):
    return F32 if case.get("f32") else BF


# ------------------------------------------------------------------------------------------- attention over the paged cache
def _in_prefill(case, r):
    H, G, D = HEADS[case["heads"]]
    lens, ctx = _lens(case), _contexts(case)
    table, blocks = _pages(r, [a + b for a, b in zip(lens, ctx)])
    s = {"H": H, "G": G, "D": D, "lens": lens, "ctx": ctx, "table": table, "q": r(sum(lens), (H + 2 * G) * D), "k": r(blocks, G, PAGE, D),
         "v": r(blocks, G, PAGE, D), "scale": D ** -0.5}
    s["k"][0], s["v"][0] = 0, 0
    return s


def _prepare_prefill(s):
    tile = ops.attn_prefill_tile(s["H"], s["G"])
    a, b = ops.build_prefill_tiles(s["lens"], tile, s["ctx"])
    s.update(cu=_i32(_starts(s["lens"])), ctx_d=_i32(s["ctx"]), ts=_i32(a), tq=_i32(b),
             out=torch.empty(s["q"].shape[0], s["H"] * s["D"], dtype=BF, device="cuda"))


def _run_prefill(s):
    return ops.paged_attn_prefill(s["q"], s["q"].shape[1], s["k"], s["v"], s["table"], s["cu"], s["ctx_d"], s["ts"], s["tq"], s["out"],
                                  s["H"], s["G"], s["D"], s["scale"])


def _rows_of(cache, table, i, n):
    """The first n rows [n, G, D] of sequence i in a paged cache [blocks, G, page, D]."""
    need = (n + PAGE - 1) // PAGE
    return cache[table[i, :need].long()].transpose(1, 2).flatten(0, 1)[:n]


def _softmax_attention(q, k, v, scale, first):
    """q [T, H, D] at positions first ..., k / v [n, G, *] -> [T, H, Dv], in 64 bits, in slices of the rows."""
    T, H = q.shape[:2]
    G = k.shape[1]
    k, v = k.to(F64), v.to(F64)
    out = []
    for a in range(0, T, 512):
        x = q[a:a + 512].to(F64).reshape(-1, G, H // G, q.shape[2])
        s = torch.einsum("tghd,ngd->ghtn", x, k) * scale
        pos = first + a + torch.arange(x.shape[0], device="cuda")
        s.masked_fill_(torch.arange(k.shape[0], device="cuda")[None] > pos[:, None], -math.inf)
        out.append(torch.einsum("ghtn,ngd->tghd", s.softmax(-1), v).reshape(x.shape[0], H, v.shape[2]))
    return torch.cat(out)


def _exact_prefill(s):
    out, H, D, cu = [], s["H"], s["D"], _starts(s["lens"])
    for i, (n, c) in enumerate(zip(s["lens"], s["ctx"])):
        q = s["q"][cu[i]:cu[i + 1], :H * D].reshape(n, H, D)
        out.append(_softmax_attention(q, _rows_of(s["k"], s["table"], i, n + c), _rows_of(s["v"], s["table"], i, n + c), s["scale"], c))
    return torch.cat(out).flatten(1)


def _pairs(case):
    return sum(n * c + n * (n + 1) // 2 for n, c in zip(_lens(case), _contexts(case)))


def _work_prefill(case):
    H, G, D = HEADS[case["heads"]]
    T, keys = case["tokens"], sum(_lens(case)) + sum(_contexts(case))
    return 4.0 * T * H * D + 4.0 * keys * G * D, 4.0 * _pairs(case) * H * D


def _decode_lens(case):
    return [max(1, case["context"] - (13 * i) % 64) for i in range(case["seqs"])]


def _in_decode(case, r):
    H, G, D = HEADS[case["heads"]]
    lens = _decode_lens(case)
    table, blocks = _pages(r, lens)
    return {"H": H, "G": G, "D": D, "lens": lens, "table": table, "q": r(len(lens), (H + 2 * G) * D), "k": r(blocks, G, PAGE, D),
            "v": r(blocks, G, PAGE, D), "scale": D ** -0.5}


def _prepare_decode(s):
    B = len(s["lens"])
    s["splits"] = ops.attn_decode_splits(B, s["G"], max(s["lens"]))
    s.update(n=_i32(s["lens"]), ws=ops.attn_decode_workspace(B, s["H"], s["D"], s["splits"], "cuda"),
             out=torch.empty(B, s["H"] * s["D"], dtype=BF, device="cuda"))


def _run_decode(s):
    return ops.paged_attn_decode(s["q"], s["q"].shape[1], s["k"], s["v"], s["table"], s["n"], s["out"], s["H"], s["G"], s["D"], s["scale"],
                                 num_splits=s["splits"], workspace=s["ws"])


def _exact_decode(s):
    H, D = s["H"], s["D"]
    return torch.cat([_softmax_attention(s["q"][i:i + 1, :H * D].reshape(1, H, D), _rows_of(s["k"], s["table"], i, n),
                                         _rows_of(s["v"], s["table"], i, n), s["scale"], n - 1) for i, n in enumerate(s["lens"])]).flatten(1)


def _work_decode(case):
    H, G, D = HEADS[case["heads"]]
    keys = sum(_decode_lens(case))
    return 4.0 * keys * G * D + 4.0 * case["seqs"] * H * D, 4.0 * keys * H * D


# ------------------------------------------------------------------------------------------- feed-forwards
def _in_mlp(case, r):
    T, D = case["tokens"], case["width"]
    ff = MLP[D]
    return {"x": r(T, D), "res": r(T, D), "w1": 1 + r(D, scale=0.1), "w2": 1 + r(D, scale=0.1), "gate_up": r(2 * ff, D, scale=D ** -0.5),
            "down": r(D, ff, scale=ff ** -0.5), "eps": 1e-5}


def _prepare_mlp(s):
    T, D = s["x"].shape
    ff = s["down"].shape[1]
    e = lambda *n, dt=BF: torch.empty(*n, dtype=dt, device="cuda")   # noqa: E731
    s["splits"] = ops.gemm_suggest_splits(T, D, ff) if T <= 256 else 1
    s.update(xn=e(T, D), r1=e(T, D), act=e(T, ff), parts=e(s["splits"], T, D, dt=F32), h=e(T, D), y=e(T, D), r2=e(T, D))


def _run_mlp(s):
    ops.fused_add_rms_norm(s["x"], s["res"], s["w1"], s["eps"], out=s["xn"], residual_out=s["r1"])
    ops.gemm_silu_mul(s["xn"], s["gate_up"], out=s["act"])
    if s["splits"] > 1:
        ops.gemm(s["act"], s["down"], out=s["parts"], splits=s["splits"])
        ops.fused_add_rms_norm_partials(s["parts"], s["r1"], s["w2"], s["eps"], s["y"], s["r2"])
    else:
        ops.gemm(s["act"], s["down"], out=s["h"])
        ops.fused_add_rms_norm(s["h"], s["r1"], s["w2"], s["eps"], out=s["y"], residual_out=s["r2"])
    return s["y"], s["r2"]


def _rms(x, eps):
    return x * (x.square().mean(-1, keepdim=True) + eps).rsqrt()


def _exact_mlp(s):
    d = lambda n: s[n].to(F64)   # noqa: E731
    r1 = d("x") + d("res")
    gu = (_rms(r1, s["eps"]) * d("w1")) @ d("gate_up").T
    r2 = r1 + (torch.nn.functional.silu(gu[:, ::2]) * gu[:, 1::2]) @ d("down").T
    return _rms(r2, s["eps"]) * d("w2"), r2


def _work_mlp(case):
    T, D = case["tokens"], case["width"]
    ff = MLP[D]
    return 6.0 * D * ff + 8.0 * T * D, 6.0 * T * D * ff


def _in_routed(case, r):
    D, ff, E, _ = ROUTED
    router = torch.zeros(128, D, dtype=BF, device="cuda")
    router[:E] = r(E, D, scale=D ** -0.5)
    return {"x": r(case["tokens"], D), "router": router, "w13": r(E * 2 * ff, D, scale=D ** -0.5), "w2": r(E * D, ff, scale=ff ** -0.5)}


def _prepare_routed(s):
    D, ff, E, top = ROUTED
    T = s["x"].shape[0]
    s.update(ws=ops.RoutedWorkspace(T, top, E, D, ff, BF, "cuda"), out=torch.empty(T, D, device="cuda"))


def _run_routed(s):
    _, ff, E, top = ROUTED
    return ops.routed_experts(s["x"], s["router"], None, s["w13"], s["w2"], s["ws"], s["out"], E, 0, top, 1.0, ff, 0.0, act="silu")


def _exact_routed(s):
    D, ff, E, top = ROUTED
    x = s["x"].to(F64)
    p = (x @ s["router"][:E].to(F64).T).softmax(-1)
    w, ids = p.topk(top, -1)
    w = w / w.sum(-1, keepdim=True)
    out = torch.zeros_like(x)
    for e in range(E):
        t, j = (ids == e).nonzero(as_tuple=True)
        gu = x[t] @ s["w13"].view(E, 2 * ff, D)[e].to(F64).T
        out.index_add_(0, t, (torch.nn.functional.silu(gu[:, ::2]) * gu[:, 1::2]) @ s["w2"].view(E, D, ff)[e].to(F64).T * w[t, j][:, None])
    return out


def _work_routed(case):
    D, ff, E, top = ROUTED
    T = case["tokens"]
    return 6.0 * D * ff * min(E, T * top) + 6.0 * T * D, 6.0 * T * top * D * ff


# ------------------------------------------------------------------------------------------- latent attention
def _in_latent(case, r):
    H, R, dr, dn, dv = LATENT
    if case["kind"] == "latent_decode":
        total = _decode_lens(case)
        lens, ctx = [1] * len(total), [n - 1 for n in total]
    else:
        lens, ctx = _lens(case), _contexts(case)
    table, blocks = _pages(r, [a + b for a, b in zip(lens, ctx)])
    s = {"lens": lens, "ctx": ctx, "table": table, "proj": r(sum(lens), H * (dn + dr) + R + dr), "cache": r(blocks, 1, PAGE, R + dr),
         "kv_norm": 1 + r(R, scale=0.1), "uk": r(H, R, dn, scale=dn ** -0.5), "uv": r(H * dv, R, scale=R ** -0.5), "sink": r(H, dtype=F32),
         "freq": _freq(dr, 1e6), "scale": (dn + dr) ** -0.5}
    s["cache"][0] = 0
    return s


def _prepare_latent(s):
    H, R, dr, dn, dv = LATENT
    T = s["proj"].shape[0]
    e = lambda *n: torch.empty(*n, dtype=BF, device="cuda")   # noqa: E731
    s.update(pos=_positions(s["lens"], s["ctx"]), slots=_slots(s["table"], s["lens"], s["ctx"]), qa=e(T, H * (R + dr)), lat=e(T, H * R),
             out=e(T, H * dv), decode=all(n == 1 for n in s["lens"]))
    if s["decode"]:
        n = [c + 1 for c in s["ctx"]]
        s["splits"] = ops.latent_attn_decode_splits(len(n), H, max(n))
        s.update(n=_i32(n), ws=ops.latent_attn_decode_workspace(len(n), H, R, 16, "cuda"))
    else:
        a, b = ops.build_prefill_tiles(s["lens"], ops.attn_sink_prefill_tile(), s["ctx"])
        s.update(cu=_i32(_starts(s["lens"])), ctx_d=_i32(s["ctx"]), ts=_i32(a), tq=_i32(b))


def _run_latent(s):
    H, R, dr, dn, dv = LATENT
    q = s["proj"][:, :H * (dn + dr)]
    ops.latent_prep(s["proj"], H * (dn + dr), q, s["kv_norm"], s["pos"], s["slots"], s["cache"], s["qa"], H, dn, dr, R, dr, False, s["freq"],
                    1.0, 1e-6)
    ops.head_linear(q, s["uk"], s["qa"], H, n=R, k=dn, x_head=dn + dr, out_head=R + dr)
    if s["decode"]:
        ops.latent_attn_decode(s["qa"], s["cache"], s["table"], s["n"], s["sink"], s["lat"], H, R, dr, s["scale"], num_splits=s["splits"],
                               workspace=s["ws"])
    else:
        ops.latent_attn_prefill(s["qa"], s["cache"], s["table"], s["cu"], s["ctx_d"], s["ts"], s["tq"], s["sink"], s["lat"], H, R, dr,
                                s["scale"])
    ops.head_linear(s["lat"], s["uv"], s["out"], H, n=dv, k=R, x_head=R, out_head=dv)
    return s["out"], s["cache"]


def _rotate(x, pos, freq, dims, half):
    """Rotation of the first `dims` entries of x [T, heads, width] at positions pos."""
    ang = pos.to(F64)[:, None] * freq
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    y = x.clone()
    a, b = (slice(0, dims // 2), slice(dims // 2, dims)) if half else (slice(0, dims, 2), slice(1, dims, 2))
    y[..., a], y[..., b] = x[..., a] * c - x[..., b] * s, x[..., b] * c + x[..., a] * s
    return y


def _exact_latent(s):
    H, R, dr, dn, dv = LATENT
    T = s["proj"].shape[0]
    pos, slots, proj = _positions(s["lens"], s["ctx"]), _slots(s["table"], s["lens"], s["ctx"]), s["proj"].to(F64)
    q = proj[:, :H * (dn + dr)].view(T, H, dn + dr)
    kv = proj[:, H * (dn + dr):]
    row = torch.cat([_rms(kv[:, :R], 1e-6) * s["kv_norm"].to(F64), _rotate(kv[:, None, R:], pos, s["freq"], dr, False)[:, 0]], -1)
    cache = s["cache"].to(F64)
    cache.view(-1, R + dr)[slots.long()] = row
    qa = torch.cat([torch.einsum("thd,hrd->thr", q[..., :dn], s["uk"].to(F64)), _rotate(q[..., dn:], pos, s["freq"], dr, False)], -1)
    cu, out = _starts(s["lens"]), []
    for i, (n, c) in enumerate(zip(s["lens"], s["ctx"])):
        k = _rows_of(cache, s["table"], i, n + c)[:, 0]
        for a in range(0, n, 512):
            x = qa[cu[i] + a:cu[i] + min(n, a + 512)]
            sc = torch.einsum("thd,nd->htn", x, k) * s["scale"]
            at = c + a + torch.arange(x.shape[0], device="cuda")
            sc.masked_fill_(torch.arange(n + c, device="cuda")[None] > at[:, None], -math.inf)
            p = torch.cat([sc, s["sink"].to(F64)[:, None, None].expand(H, x.shape[0], 1)], -1).softmax(-1)[..., :-1]
            out.append(torch.einsum("htn,nr->thr", p, k[:, :R]))
    o = torch.einsum("thr,hvr->thv", torch.cat(out), s["uv"].view(H, dv, R).to(F64))
    return o.flatten(1), cache


def _work_latent(case):
    H, R, dr, dn, dv = LATENT
    if case["kind"] == "latent_decode":
        n = _decode_lens(case)
        T, keys, pairs = len(n), sum(n), sum(n)
    else:
        T, keys, pairs = case["tokens"], sum(_contexts(case)) + case["tokens"], _pairs(case)
    flops = 2.0 * pairs * H * (2 * R + dr) + 2.0 * T * H * R * (dn + dv)
    return 2.0 * (keys * (R + dr) + T * (H * (dn + dr + dv) + 2 * (R + dr)) + H * R * (dn + dv)), flops


# ------------------------------------------------------------------------------------------- recurrences
def _sequences(case):
    lens, ctx = _lens(case), _contexts(case)
    return {"lens": lens, "ctx": ctx, "act": _act(case)}


def _prepare_sequences(s):
    lens = s["lens"]
    s.update(cu=_i32(_starts(lens)), ctx_d=_i32(s["ctx"]), pos=_positions(lens, s["ctx"]), slot=_i32(list(range(len(lens)))[::-1]),
             longest=1 if max(lens) == 1 else sum(lens))


def _states(s, name):
    """Per sequence, its state at the start in 64 bits (slots are handed out in reverse order)."""
    n = len(s["lens"])
    return [s[name][n - 1 - i].to(F64) * (1.0 if s["ctx"][i] else 0.0) for i in range(n)]


def _in_mlstm(case, r):
    H, dk, dv = RECURRENT
    s = _sequences(case)
    T, n, Z = sum(s["lens"]), len(s["lens"]), (dv + 31) // 32
    norm = r(n, H, 1, dk, dtype=F32).expand(n, H, Z, dk).contiguous()
    m = r.uniform(n, H, 1, low=-1.0, high=1.0).expand(n, H, Z).contiguous()
    s.update(proj=r(T, 2 * H * dk + 2 * H * dv, dtype=s["act"]), gates=r(T, 2 * H, dtype=F32),
             bias=torch.cat([r(H, scale=0.5), 3 + r(H, scale=0.5)]), S=r(n, H, dv, dk, dtype=F32), n=norm, m=m, w=1 + r(H * dv, scale=0.1))
    return s


def _prepare_mlstm(s):
    H, dk, dv = RECURRENT
    _prepare_sequences(s)
    T = s["proj"].shape[0]
    s.update(o=torch.empty(T, H * dv, device="cuda"), out=torch.empty(T, H * dv, dtype=s["act"], device="cuda"))


def _run_mlstm(s):
    H, dk, dv = RECURRENT
    ops.mlstm_scan(s["proj"], 0, H * dk, 2 * H * dk, s["gates"], s["bias"], s["cu"], s["ctx_d"], s["slot"], s["S"], s["n"], s["m"], s["o"],
                   H, dk, dv, 15.0, max_len=s["longest"])
    ops.mlstm_out(s["o"], s["proj"], 2 * H * dk + H * dv, s["w"], s["out"], H, dv, 1e-5)
    return s["out"], s["S"], s["n"], s["m"]


def _exact_mlstm(s):
    H, dk, dv = RECURRENT
    p, cu = s["proj"].to(F64), _starts(s["lens"])
    T = p.shape[0]
    q = p[:, :H * dk].view(T, H, dk) * dk ** -0.5
    k, v = p[:, H * dk:2 * H * dk].view(T, H, dk), p[:, 2 * H * dk:2 * H * dk + H * dv].view(T, H, dv)
    a = 15.0 * torch.tanh((s["gates"].to(F64) + s["bias"].to(F64)) / 15.0)
    li, lf = a[:, :H], torch.nn.functional.logsigmoid(a[:, H:])
    S2, n2, m2 = s["S"].to(F64), s["n"].to(F64), s["m"].to(F64)
    S0, n0, m0 = _states(s, "S"), _states(s, "n"), _states(s, "m")
    o = torch.empty(T, H, dv, dtype=F64, device="cuda")
    for i in range(len(s["lens"])):
        S, n, m = S0[i], n0[i][:, 0], m0[i][:, 0]
        for t in range(cu[i], cu[i + 1]):
            new = torch.maximum(lf[t] + m, li[t])
            f, g = torch.exp(lf[t] + m - new)[:, None], torch.exp(li[t] - new)[:, None]
            m = new
            S = f[..., None] * S + v[t][:, :, None] * (g * k[t])[:, None]
            n = f * n + g * k[t]
            den = torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-m)) + 1e-6
            o[t] = torch.einsum("hvk,hk->hv", S, q[t]) / den[:, None]
        at = len(s["lens"]) - 1 - i
        S2[at], n2[at], m2[at] = S, n[:, None], m[:, None]
    gate = torch.sigmoid(p[:, 2 * H * dk + H * dv:])
    return (_rms(o, 1e-5).flatten(1) * s["w"].to(F64) * gate), S2, n2, m2


def _in_linear(case, r):
    H, dk, dv = RECURRENT
    s = _sequences(case)
    T, n = sum(s["lens"]), len(s["lens"])
    s.update(proj=r(T, 2 * H * dk + 2 * H * dv, dtype=s["act"]), S=r(n, H, dv, dk, dtype=F32), freq=_freq(dk, 1e6),
             decay=torch.tensor([1.0 - 2.0 ** (-5 - 5 * i / (H - 1)) for i in range(H)], device="cuda"))
    return s


def _prepare_linear(s):
    H, dk, dv = RECURRENT
    _prepare_sequences(s)
    T = s["proj"].shape[0]
    s.update(x=torch.empty(T, 2 * H * dk + H * dv, device="cuda"), o=torch.empty(T, H * dv, device="cuda"),
             out=torch.empty(T, H * dv, dtype=s["act"], device="cuda"))


def _run_linear(s):
    H, dk, dv = RECURRENT
    kc, vc, x = H * dk, 2 * H * dk, s["x"]
    ops.rot_prep(s["proj"], 0, kc, vc, s["pos"], None, x, x[:, kc:], x[:, vc:], H, H, dk, dv, paged=False, rot_dims=dk, half_layout=True,
                 freq=s["freq"], k_mul=dk ** -0.5)
    ops.linattn_scan(x, 0, kc, vc, s["decay"], s["cu"], s["ctx_d"], s["slot"], s["S"], s["o"], H, dk, dv, max_len=s["longest"])
    ops.linattn_out(s["o"], s["proj"], vc + H * dv, None, s["out"], H, dv, 1e-5, False, "silu")
    return s["out"], s["S"]


def _decayed(s, q, k, v, decay):
    """o_t = S_t^T q_t with S_t = decay_t S_(t-1) + k_t v_t^T; decay broadcasts against [T, H, dk]."""
    cu, S2, S0 = _starts(s["lens"]), s["S"].to(F64), _states(s, "S")
    o = torch.empty_like(v)
    for i in range(len(s["lens"])):
        S = S0[i]
        for t in range(cu[i], cu[i + 1]):
            S = decay[t][:, None] * S + v[t][:, :, None] * k[t][:, None]
            o[t] = torch.einsum("hvk,hk->hv", S, q[t])
        S2[len(s["lens"]) - 1 - i] = S
    return o, S2


def _exact_linear(s):
    H, dk, dv = RECURRENT
    p = s["proj"].to(F64)
    T, pos = p.shape[0], _positions(s["lens"], s["ctx"])
    q = _rotate(p[:, :H * dk].view(T, H, dk), pos, s["freq"], dk, True)
    k = _rotate(p[:, H * dk:2 * H * dk].view(T, H, dk), pos, s["freq"], dk, True) * dk ** -0.5
    v = p[:, 2 * H * dk:2 * H * dk + H * dv].view(T, H, dv)
    o, S = _decayed(s, q, k, v, s["decay"].to(F64)[None, :, None].expand(T, H, 1))
    return _rms(o, 1e-5).flatten(1) * torch.nn.functional.silu(p[:, 2 * H * dk + H * dv:]), S


def _in_gated_linear(case, r):
    H, dk, dv, rank = GATED
    s = _sequences(case)
    T, n = sum(s["lens"]), len(s["lens"])
    s.update(proj=r(T, 2 * H * dk + 2 * H * dv + rank, dtype=s["act"]), S=r(n, H, dv, dk, dtype=F32), up=r(H * dk, rank, scale=rank ** -0.5),
             bias=2 + r(H * dk, scale=0.5), w=1 + r(dv, scale=0.1))
    return s


def _prepare_gated_linear(s):
    H, dk, dv, rank = GATED
    _prepare_sequences(s)
    T = s["proj"].shape[0]
    s.update(x=torch.empty(T, 2 * H * dk + H * dv, device="cuda"), z=torch.empty(T, H * dk, device="cuda"),
             o=torch.empty(T, H * dv, device="cuda"), out=torch.empty(T, H * dv, dtype=s["act"], device="cuda"))


def _run_gated_linear(s):
    H, dk, dv, rank = GATED
    kc, vc, x, ac = H * dk, 2 * H * dk, s["x"], 2 * H * dk + 2 * H * dv
    ops.rot_prep(s["proj"], 0, kc, vc, s["pos"], None, x, x[:, kc:], x[:, vc:], H, H, dk, dv, paged=False, q_mul=dk ** -0.5)
    ops.linear(s["proj"][:, ac:ac + rank], s["up"], s["z"], bias=s["bias"])
    ops.gla_scan(x, 0, kc, vc, s["z"], 1.0 / 16.0, s["cu"], s["ctx_d"], s["slot"], s["S"], s["o"], H, dk, dv, max_len=s["longest"])
    ops.linattn_out(s["o"], s["proj"], vc + H * dv, s["w"], s["out"], H, dv, 1e-5, False, "silu")
    return s["out"], s["S"]


def _exact_gated_linear(s):
    H, dk, dv, rank = GATED
    p = s["proj"].to(F64)
    T, ac = p.shape[0], 2 * H * dk + 2 * H * dv
    z = p[:, ac:] @ s["up"].to(F64).T + s["bias"].to(F64)
    alpha = torch.exp(torch.nn.functional.logsigmoid(z) / 16.0).view(T, H, dk)
    q, k = p[:, :H * dk].view(T, H, dk) * dk ** -0.5, p[:, H * dk:2 * H * dk].view(T, H, dk)
    o, S = _decayed(s, q, k, p[:, 2 * H * dk:2 * H * dk + H * dv].view(T, H, dv), alpha)
    gate = torch.nn.functional.silu(p[:, 2 * H * dk + H * dv:ac])
    return (_rms(o, 1e-5) * s["w"].to(F64)).flatten(1) * gate, S


def _scan_shape(kind):
    """heads, key heads, key width, value width, taps, convolved channels, and the segments of conv_rec_prep."""
    if kind == "delta":
        H, G, dk, dv, taps = DELTA
        return H, G, dk, dv, taps, 2 * G * dk + H * dv, ((G, dk, dk ** -0.5), (G, dk, 1.0), (H, dv, None))
    H, G, dk, dv, taps = SPACE
    return H, G, dk, dv, taps, H * dv + 2 * G * dk, ((H, dv, None), (G, dk, None), (G, dk, None))


def _in_scan(case, r):
    H, G, dk, dv, taps, C, segments = _scan_shape(case["kind"])
    s = _sequences(case)
    T, n, delta = sum(s["lens"]), len(s["lens"]), case["kind"] == "delta"
    s.update(kind=case["kind"], proj=r(T, C + H * dv, dtype=s["act"]), conv=r(taps, C, scale=0.5, dtype=F32),
             conv_bias=None if delta else r(C, scale=0.1, dtype=F32), ring=r(n, taps - 1, C, dtype=F32), gates=r(T, (2 if delta else 1) * H, dtype=F32),
             rate=r.uniform(H, low=0.1, high=1.0), dt=r(H, scale=0.5, dtype=F32) - 2.0, skip=None if delta else r(H, dtype=F32),
             S=r(n, H, dv, dk, scale=0.2, dtype=F32), w=1 + r(dv if delta else H * dv, scale=0.1))
    return s


def _prepare_scan(s):
    H, G, dk, dv, taps, C, segments = _scan_shape(s["kind"])
    _prepare_sequences(s)
    T, single = s["proj"].shape[0], max(s["lens"]) == 1
    s["tile"] = ops.attn_prefill_tile(16, 4)
    a, b = ([], []) if single else ops.build_prefill_tiles(s["lens"], s["tile"], s["ctx"])
    s.update(ts=None if single else _i32(a), tq=None if single else _i32(b), n_prompt=0 if single else len(s["lens"]),
             n_single=len(s["lens"]) if single else 0, x=torch.empty(T, C, device="cuda"), o=torch.empty(T, H * dv, device="cuda"),
             out=torch.empty(T, H * dv, dtype=s["act"], device="cuda"))


def _run_scan(s):
    H, G, dk, dv, taps, C, segments = _scan_shape(s["kind"])
    delta = s["kind"] == "delta"
    ops.conv_rec_prep(s["proj"], s["conv"], s["conv_bias"], s["ring"], s["cu"], s["ctx_d"], s["slot"], s["ts"], s["tq"], s["tile"],
                      s["n_prompt"], s["n_single"], segments, s["x"])
    q, k, v = (0, G * dk, 2 * G * dk) if delta else (H * dv + G * dk, H * dv, 0)
    ops.gated_scan(s["x"], q, k, v, s["gates"], s["rate"], s["dt"], s["skip"], s["cu"], s["ctx_d"], s["slot"], s["S"], s["o"], H, G, dk, dv,
                   delta, max_len=s["longest"])
    ops.gate_norm(s["o"], s["proj"], C, s["w"], s["out"], H if delta else G, 1e-5, gate_after=delta)
    return s["out"], s["S"], s["ring"]


def _exact_scan(s):
    H, G, dk, dv, taps, C, segments = _scan_shape(s["kind"])
    delta, p, cu, n = s["kind"] == "delta", s["proj"].to(F64), _starts(s["lens"]), len(s["lens"])
    T, R = p.shape[0], taps - 1
    ring, rows = s["ring"].to(F64), []
    for i in range(n):
        c, u, slot = s["ctx"][i], p[cu[i]:cu[i + 1], :C], n - 1 - i
        old = torch.zeros(R, C, dtype=F64, device="cuda")
        for j in range(min(R, c)):                           # the input at position c - 1 - j
            old[R - 1 - j] = ring[slot][(c - 1 - j) % R]
        full = torch.cat([old, u])
        rows.append(sum(s["conv"][j].to(F64) * full[j:j + u.shape[0]] for j in range(taps)))
        for j in range(min(R, u.shape[0])):
            ring[slot][(c + u.shape[0] - 1 - j) % R] = u[u.shape[0] - 1 - j]
    y = torch.cat(rows)
    y = torch.nn.functional.silu(y if delta else y + s["conv_bias"].to(F64))
    if delta:
        unit = lambda x: x / (x.square().sum(-1, keepdim=True) + 1e-6).sqrt()   # noqa: E731
        q, k = unit(y[:, :G * dk].view(T, G, dk)) * dk ** -0.5, unit(y[:, G * dk:2 * G * dk].view(T, G, dk))
        v = y[:, 2 * G * dk:].view(T, H, dv)
        beta, a = torch.sigmoid(s["gates"][:, :H].to(F64)), s["gates"][:, H:].to(F64)
    else:
        v, k, q = y[:, :H * dv].view(T, H, dv), y[:, H * dv:H * dv + G * dk].view(T, G, dk), y[:, H * dv + G * dk:].view(T, G, dk)
        a = s["gates"].to(F64)
    q, k = q.repeat_interleave(H // G, 1), k.repeat_interleave(H // G, 1)
    step = torch.nn.functional.softplus(a + s["dt"].to(F64))
    g = torch.exp(-s["rate"].to(F64) * step)
    if not delta:
        beta = step
    o, S2, S0 = torch.empty(T, H, dv, dtype=F64, device="cuda"), s["S"].to(F64), _states(s, "S")
    for i in range(n):
        S = S0[i]
        for t in range(cu[i], cu[i + 1]):
            S = g[t][:, None, None] * S
            u = beta[t][:, None] * (v[t] - torch.einsum("hvk,hk->hv", S, k[t]) if delta else v[t])
            S = S + u[:, :, None] * k[t][:, None]
            o[t] = torch.einsum("hvk,hk->hv", S, q[t])
        S2[n - 1 - i] = S
    z = torch.nn.functional.silu(p[:, C:])
    if delta:
        out = (_rms(o, 1e-5) * s["w"].to(F64)).flatten(1) * z
    else:
        o = (o + s["skip"].to(F64)[:, None] * v).flatten(1) * z
        out = _rms(o.view(T, G, -1), 1e-5).flatten(1) * s["w"].to(F64)
    return out, S2, ring


def _work_recurrence(case):
    """Rows and gate in, output rows out, states in and out; the recurrence's own products."""
    kind, T, n, a = case["kind"], case["tokens"], case["seqs"], 4 if case.get("f32") else 2
    if kind in ("mlstm", "linear"):
        H, dk, dv = RECURRENT
        width, G, per = 2 * H * dk + 2 * H * dv, H, 4.0
    elif kind == "gated_linear":
        H, dk, dv, rank = GATED
        width, G, per = 2 * H * dk + 2 * H * dv + rank, H, 5.0
    else:
        H, G, dk, dv = _scan_shape(kind)[:4]
        width, per = 2 * G * dk + 2 * H * dv, 6.0 if kind == "delta" else 4.0
    return a * T * (width + H * dv) + 8.0 * n * H * dk * dv, per * T * H * dk * dv


# ------------------------------------------------------------------------------------------- the engine
def _in_engine(case, r):
    D, ff, L, H, G, hd, V = ENGINE
    w = {"model.embed_tokens.weight": r(V, D), "model.norm.weight": 1 + r(D, scale=0.1), "lm_head.weight": r(V, D, scale=D ** -0.5)}
    for i in range(L):
        p = "model.layers.%d." % i
        for name, rows, cols in (("self_attn.q_proj", H * hd, D), ("self_attn.k_proj", G * hd, D), ("self_attn.v_proj", G * hd, D),
                                 ("self_attn.o_proj", D, H * hd), ("mlp.gate_proj", ff, D), ("mlp.up_proj", ff, D), ("mlp.down_proj", D, ff)):
            w[p + name + ".weight"] = r(rows, cols, scale=cols ** -0.5)
        w[p + "input_layernorm.weight"], w[p + "post_attention_layernorm.weight"] = 1 + r(D, scale=0.1), 1 + r(D, scale=0.1)
    lens = _lens(case)
    ids = torch.randint(0, V, (sum(lens) + case["steps"] * len(lens),), generator=r.g, device="cuda").cpu().tolist()
    cu = _starts(lens)
    return {"weights": w, "lens": lens, "prompts": [ids[cu[i]:cu[i + 1]] for i in range(len(lens))],
            "next": [ids[cu[-1] + j * len(lens):cu[-1] + (j + 1) * len(lens)] for j in range(case["steps"])]}


def _prepare_engine(s):
    from gpustack_b200.config import EngineConfig, ModelConfig
    from gpustack_b200.engine import LLMEngine

    D, ff, L, H, G, hd, V = ENGINE
    n = len(s["lens"])
    cfg = ModelConfig(vocab_size=V, hidden_size=D, intermediate_size=ff, num_hidden_layers=L, num_attention_heads=H, num_key_value_heads=G,
                      head_dim=hd, max_position_embeddings=1024, eos_token_id=2, bos_token_id=1)
    s["engine"] = LLMEngine.from_engine_config(
        EngineConfig(max_model_len=1024, max_num_seqs=8, max_num_batched_tokens=2560, num_gpu_blocks=600, enable_prefix_caching=False,
                     cuda_graph_sizes=[n]), mcfg=cfg, state_dict=s.pop("weights"))


def _run_engine(s):
    """Prompts in one step, then one given token per request and step (a recorded trace); the logits of every step."""
    e, n = s["engine"], len(s["lens"])
    end = [str(i) for i in range(n)]
    out = [e.replay_step([(str(i), p, [len(p) - 1]) for i, p in enumerate(s["prompts"])], [] if s["next"] else end)]
    for j, row in enumerate(s["next"]):
        out.append(e.replay_step([(str(i), [t], [0]) for i, t in enumerate(row)], end if j + 1 == len(s["next"]) else []))
    return out


def _exact_engine(s):
    D, ff, L, H, G, hd, V = ENGINE
    w, freq = {k: v.to(F64) for k, v in s["weights"].items()}, _freq(hd, 500000.0)
    rows = []
    for i, p in enumerate(s["prompts"]):
        ids = torch.tensor(p + [row[i] for row in s["next"]], device="cuda")
        T = ids.shape[0]
        pos = torch.arange(T, device="cuda")
        x = w["model.embed_tokens.weight"][ids]
        for l in range(L):
            g = lambda name: w["model.layers.%d.%s.weight" % (l, name)]   # noqa: B023, E731
            h = _rms(x, 1e-5) * g("input_layernorm")
            q, k, v = ((h @ g("self_attn.%s_proj" % a).T).view(T, -1, hd) for a in "qkv")
            q, k = _rotate(q, pos, freq, hd, True), _rotate(k, pos, freq, hd, True)
            x = x + _softmax_attention(q, k, v, hd ** -0.5, 0).flatten(1) @ g("self_attn.o_proj").T
            h = _rms(x, 1e-5) * g("post_attention_layernorm")
            x = x + (torch.nn.functional.silu(h @ g("mlp.gate_proj").T) * (h @ g("mlp.up_proj").T)) @ g("mlp.down_proj").T
        rows.append((_rms(x[len(p) - 1:], 1e-5) * w["model.norm.weight"]) @ w["lm_head.weight"].T)
    return [torch.stack([r[j] for r in rows]) for j in range(1 + len(s["next"]))]


def _work_engine(case):
    D, ff, L, H, G, hd, V = ENGINE
    T, n, k = case["tokens"], case["seqs"], case["steps"]
    layer = D * (H + 2 * G) * hd + H * hd * D + 3 * D * ff
    return (1 + k) * 2.0 * (L * layer + V * D) + 4.0 * (1 + k) * n * V, 2.0 * (T + k * n) * L * layer + 2.0 * (1 + k) * n * V * D


_INPUTS = {"attention_prefill": _in_prefill, "attention_decode": _in_decode, "mlp": _in_mlp, "routed": _in_routed, "latent_prefill": _in_latent,
           "latent_decode": _in_latent, "mlstm": _in_mlstm, "linear": _in_linear, "gated_linear": _in_gated_linear, "delta": _in_scan,
           "state_space": _in_scan, "engine": _in_engine}
_PREPARE = {"attention_prefill": _prepare_prefill, "attention_decode": _prepare_decode, "mlp": _prepare_mlp, "routed": _prepare_routed,
            "latent_prefill": _prepare_latent, "latent_decode": _prepare_latent, "mlstm": _prepare_mlstm, "linear": _prepare_linear,
            "gated_linear": _prepare_gated_linear, "delta": _prepare_scan, "state_space": _prepare_scan, "engine": _prepare_engine}
_RUN = {"attention_prefill": _run_prefill, "attention_decode": _run_decode, "mlp": _run_mlp, "routed": _run_routed, "latent_prefill": _run_latent,
        "latent_decode": _run_latent, "mlstm": _run_mlstm, "linear": _run_linear, "gated_linear": _run_gated_linear, "delta": _run_scan,
        "state_space": _run_scan, "engine": _run_engine}
_EXACT = {"attention_prefill": _exact_prefill, "attention_decode": _exact_decode, "mlp": _exact_mlp, "routed": _exact_routed,
          "latent_prefill": _exact_latent, "latent_decode": _exact_latent, "mlstm": _exact_mlstm, "linear": _exact_linear,
          "gated_linear": _exact_gated_linear, "delta": _exact_scan, "state_space": _exact_scan, "engine": _exact_engine}
_WORK = {"attention_prefill": _work_prefill, "attention_decode": _work_decode, "mlp": _work_mlp, "routed": _work_routed,
         "latent_prefill": _work_latent, "latent_decode": _work_latent, "engine": _work_engine}


def prepare(case, seed):
    s = _inputs(case, seed)
    _PREPARE[case["kind"]](s)
    s["run"] = _RUN[case["kind"]]
    return s


def run(state):
    return state["run"](state)


def work(case):
    b, f = _WORK.get(case["kind"], _work_recurrence)(case)
    return {"bytes": b, "flops": f}


def tolerance(case):
    if case.get("f32"):
        return {"rel": 1e-5, "max": 4e-3}
    return {"rel": 1e-2, "max": 0.1} if case["kind"] != "engine" else {"rel": 2e-2, "max": 0.2}


def exact(case, seed):
    with torch.no_grad():
        return _EXACT[case["kind"]](_inputs(case, seed))
