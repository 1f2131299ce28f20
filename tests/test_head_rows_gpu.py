"""The closing norm and gate of recurrent heads in registers, against fp64, and rotations of several rows per CTA against fewer rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu

F64, BF = torch.float64, torch.bfloat16


# heads of 8, 16 and 32 lanes; items that fill no warp, no CTA; 48: the general kernel
@pytest.mark.parametrize("dtype", [torch.float32, BF])
@pytest.mark.parametrize("dv", [32, 64, 128, 48])
@pytest.mark.parametrize("T,H", [(1, 1), (5, 3), (67, 8)])
def test_head_norm_and_gate(T, H, dv, dtype):
    from gpustack_b200 import ops

    g = torch.Generator().manual_seed(T + dv)
    o, proj = torch.randn(T, H * dv, generator=g) * 3, (torch.randn(T, 8 + H * dv, generator=g) * 30).to(dtype)
    proj[0, 8:11] = torch.tensor([-1.0e4, 1.0e4, -90.0])               # gates whose quotients leave the branch-free range
    w = torch.randn(H * dv, generator=g).to(BF)
    # bf16: half a unit in the last of 8 bits is at most 2^-8 of a value, and so of the norm; fp32: a few operations each
    tol = 2.0 ** -8 if dtype == BF else 64 * 2.0 ** -24
    z, x = proj[:, 8:].to(F64), o.to(F64).view(T, H, dv)
    n = (x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5)).reshape(T, -1)

    def check(got, want):
        assert float((got.cpu().to(F64) - want).norm() / want.norm()) < tol

    for act in ("sigmoid", "silu"):
        out = torch.zeros(T, H * dv, dtype=dtype, device="cuda")
        ops.linattn_out(o.cuda(), proj.cuda(), 8, None, out, H, dv, 1e-5, False, act)
        check(out, n * torch.sigmoid(z) * (z if act == "silu" else 1.0))
    out = torch.zeros(T, H * dv, dtype=dtype, device="cuda")
    ops.mlstm_out(o.cuda(), proj.cuda(), 8, w.cuda(), out, H, dv, 1e-5)
    check(out, n * w.to(F64) * torch.sigmoid(z))


@pytest.mark.parametrize("half", [True, False])
@pytest.mark.parametrize("T", [4736, 4737, 4739])                      # the first count with four rows per CTA, remainders of one and three
def test_rotations_of_four_rows_per_cta(T, half):
    from gpustack_b200 import ops

    H, dk, dv = 2, 64, 64
    kc, vc = H * dk, 2 * H * dk
    g = torch.Generator().manual_seed(T)
    proj = torch.randn(T, vc + H * dv, generator=g).to(BF).cuda()
    pos = torch.randint(0, 50000, (T,), generator=g, dtype=torch.int32).cuda()
    freq = (10000.0 ** (-torch.arange(dk // 2, dtype=F64) / 32)).cuda()

    def run(a, b):
        x = torch.zeros(b - a, vc + H * dv, device="cuda")
        ops.rot_prep(proj[a:b], 0, kc, vc, pos[a:b], None, x, x[:, kc:], x[:, vc:], H, H, dk, dv, paged=False, feature="silu", rot_dims=dk,
                     half_layout=half, freq=freq, k_mul=0.5)
        return x

    assert torch.equal(run(0, T), torch.cat([run(0, 2000), run(2000, 4000), run(4000, T)]))


@pytest.mark.parametrize("src,dst", [(BF, BF), (torch.float32, torch.float32), (BF, torch.float32)])
@pytest.mark.parametrize("half", [True, False])
@pytest.mark.parametrize("T", [4737, 4739])
def test_rotations_of_four_rows_per_cta_into_pages(T, half, src, dst):
    """Every instance, paged, with a norm, factors, an unrotated rest, fewer key heads and rows that have no slot."""
    from gpustack_b200 import ops

    H, G, dk, dv, dims, page = 3, 2, 96, 64, 64, 16
    kc, vc = H * dk, (H + G) * dk
    g = torch.Generator().manual_seed(T + half)
    proj = torch.randn(T, vc + G * dv, generator=g).to(src).cuda()
    pos = torch.randint(0, 50000, (T,), generator=g, dtype=torch.int32).cuda()
    slots = torch.randperm(T + 40, generator=g)[:T].to(torch.int32)
    slots[::97] = -1
    slots = slots.cuda()
    freq = (10000.0 ** (-torch.arange(dims // 2, dtype=F64) / (dims // 2))).cuda()
    mul = torch.rand(H, generator=g).cuda()

    def run(cuts):
        q = torch.full((T, H * dk), 7.0, dtype=dst, device="cuda")
        k, v = (torch.full(((T + 40 + page - 1) // page, G, page, w), 7.0, dtype=dst, device="cuda") for w in (dk, dv))
        for a, b in zip(cuts, cuts[1:]):
            ops.rot_prep(proj[a:b], 0, kc, vc, pos[a:b], slots[a:b], q[a:b], k, v, H, G, dk, dv, paged=True, rot_dims=dims, half_layout=half,
                         freq=freq, unit_norm=True, eps=1e-6, q_mul=0.5, k_mul=2.0, q_head_mul=mul)
        return q, k, v

    for a, b in zip(run([0, T]), run([0, 2000, 4000, T])):
        assert torch.equal(a, b)
