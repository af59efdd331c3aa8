"""QK-norm + rotary kernels where the split of a token's heads over warps and the width of the loads change: one token, odd head
counts, more tokens than resident warps, views that start on an 8-byte boundary, and the scatter into the paged cache."""
import pytest
import torch

from miles_b200.ops import reference as R

pytestmark = pytest.mark.gpu
DEV, D = "cuda", 128


@pytest.fixture(scope="module")
def ext():
    from miles_b200.ops import _ext

    return _ext.load(required=True)


def _shifted(t, by):
    """The same values in a tensor whose first element lies ``by`` elements into its storage."""
    buf = torch.empty(t.numel() + by, dtype=t.dtype, device=t.device)
    buf[by:].copy_(t.reshape(-1))
    return buf[by:].view(t.shape)


def _rel(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-20)).item()


@pytest.mark.parametrize("T,Hq,Hk", [(1, 3, 1), (1, 32, 4), (64, 32, 4), (2371, 5, 1), (19001, 2, 1)])
@pytest.mark.parametrize("shift", [0, 4])
@pytest.mark.parametrize("use_norm", [True, False])
def test_every_split_of_the_heads(ext, T, Hq, Hk, shift, use_norm):
    torch.manual_seed(T + Hq + shift)
    qkv = _shifted(torch.randn(T, (Hq + 2 * Hk) * D, device=DEV).bfloat16(), shift)
    pos = torch.randint(0, 9000, (T,), device=DEV, dtype=torch.int32)
    qw, kw = ((torch.randn(D, device=DEV) * 0.1 + 1).bfloat16() if use_norm else None for _ in range(2))
    slots = torch.randperm(T + 7, device=DEV)[:T].to(torch.int32)
    slots[T // 2] = -1  # a row that is not stored
    kc, vc = (torch.full((T + 7, Hk, D), 7.0, device=DEV, dtype=torch.bfloat16) for _ in range(2))
    q, k, qr, kr = ext.qk_norm_rope_fwd(qkv, qw, kw, pos, Hq, Hk, 1e6, 1e-6, kc, vc, slots, True)
    f = qkv.double().requires_grad_(True)
    qwd, kwd = ((w.double().requires_grad_(True) if use_norm else None) for w in (qw, kw))
    q_ref, k_ref, v_ref = R.qk_norm_rope(f, qwd, kwd, pos, Hq, Hk, D, 1e6, 1e-6)
    # bf16 results: a rounding of 2^-9 after the norm and one after the rotation; angles up to 9000 in fp32 add 9000 * 2^-24
    assert _rel(q, q_ref) < 5e-3 and _rel(k, k_ref) < 5e-3
    kept = slots >= 0
    assert torch.equal(kc[slots[kept].long()], k[kept]) and torch.equal(vc[slots[kept].long()], qkv.view(T, -1, D)[:, Hq + Hk:][kept])
    rest = torch.ones(T + 7, dtype=torch.bool, device=DEV)
    rest[slots[kept].long()] = False
    assert (kc[rest] == 7).all() and (vc[rest] == 7).all()
    dq, dk, dv = (_shifted(torch.randn(T, h, D, device=DEV).bfloat16(), shift) for h in (Hq, Hk, Hk))
    ((q_ref * dq.double()).sum() + (k_ref * dk.double()).sum() + (v_ref * dv.double()).sum()).backward()
    dqw, dkw = (torch.zeros(D, device=DEV) if use_norm else None for _ in range(2))
    got = ext.qk_norm_rope_bwd(dq, dk, dv, qkv, qw, kw, pos, qr if use_norm else None, kr if use_norm else None, dqw, dkw, Hq, Hk, 1e6)
    assert _rel(got, f.grad) < 5e-3
    if use_norm:
        # the summands' own error is the rotation's, about 1e-3 at these angles
        assert _rel(dqw, qwd.grad) < 5e-3 and _rel(dkw, kwd.grad) < 5e-3


def _fma(a, b, c):  # one rounding: the product is exact in 64 bits, the sum then almost always rounds to 32 bits as it would from infinite precision
    return (a.double() * b.double() + c.double()).float()


def _tree(t):  # [.., 32] -> [..]: the value 16 places further is added, then 8, 4, 2 and 1
    for o in (16, 8, 4, 2, 1):
        t = t[..., :o] + t[..., o:2 * o]
    return t[..., 0]


@pytest.mark.parametrize("T,Hq,Hk", [(1, 3, 1), (517, 8, 2)])
@pytest.mark.parametrize("rotary", [128, 64])
def test_order_of_sums_and_roundings(ext, T, Hq, Hk, rotary):
    torch.manual_seed(T + rotary)
    heads, half = Hq + Hk, rotary // 2
    qkv = torch.randn(T, (Hq + 2 * Hk) * D, device=DEV).bfloat16()
    pos = torch.randint(0, 9000, (T,), device=DEV, dtype=torch.int32)
    qw, kw = ((torch.randn(D, device=DEV) * 0.1 + 1).bfloat16() for _ in range(2))
    tab = (1e6 ** (-torch.arange(half, device=DEV).float() / half)).contiguous()
    q, k, qr, kr = ext.qk_norm_rope_fwd_scaled(qkv, qw, kw, pos, Hq, Hk, 1e6, 1e-6, None, None, None, True, tab, rotary)
    x = qkv.view(T, -1, D)[:, :heads].float()
    s = x.view(T, heads, 32, 4).square()  # (exact: bf16 squares have 16 bits)
    r = torch.rsqrt(_tree(s[..., 0] + s[..., 1] + s[..., 2] + s[..., 3]) / D + 1e-6)
    assert torch.equal(torch.cat([qr.view(T, Hq), kr.view(T, Hk)], 1), r)
    w = torch.cat([qw.expand(Hq, D), kw.expand(Hk, D)]).float()
    n = (x * r[..., None] * w).bfloat16().float()
    ang = pos.float()[:, None] * tab
    c, sn = ang.cos()[:, None], ang.sin()[:, None]
    a, b = n[..., :half], n[..., half:rotary]
    want = torch.cat([_fma(a, c, -(b * sn)), _fma(a, sn, b * c), n[..., rotary:]], -1).bfloat16()
    assert torch.equal(torch.cat([q, k], 1), want)
    dq, dk, dv = (torch.randn(T, h, D, device=DEV).bfloat16() for h in (Hq, Hk, Hk))
    dqw, dkw = (torch.zeros(D, device=DEV) for _ in range(2))
    got = ext.qk_norm_rope_bwd_scaled(dq, dk, dv, qkv, qw, kw, pos, qr, kr, dqw, dkw, Hq, Hk, 1e6, tab, rotary).view(T, -1, D)[:, :heads]
    g = torch.cat([dq, dk], 1).float()
    a, b = g[..., :half], g[..., half:rotary]
    dn = torch.cat([_fma(b, sn, a * c), _fma(b, c, -(a * sn)), g[..., rotary:]], -1)
    t, rr = (dn * w * x).view(T, heads, 32, 4), r[..., None].expand(T, heads, 32)
    lane = torch.zeros(T, heads, 32, device=DEV)
    for i in range(4):
        lane = _fma(t[..., i], rr, lane)
    dot = _tree(lane)[..., None] / D
    want = (r[..., None] * _fma(-(x * r[..., None]), dot.expand_as(x), dn * w)).bfloat16()
    assert torch.equal(got, want)
