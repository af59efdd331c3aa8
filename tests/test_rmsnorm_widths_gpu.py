"""RMSNorm where the pieces of a row that a thread keeps change: one, two and four of them, rows that end inside one, rows too wide."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("T, H", [(1, 8), (3, 2048), (700, 2056), (5, 4096), (300, 4104), (2, 6144), (3, 8192), (5, 8200), (297, 520)])
@pytest.mark.parametrize("residual", [False, True])
def test_against_64_bits(T, H, residual):
    from miles_b200.ops import _ext

    C = _ext.load(required=True)
    g = torch.Generator(device=DEV).manual_seed(T + H)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g).bfloat16()  # noqa: E731
    x, w, dy = rnd(T, H), (1 + 0.1 * rnd(H)).bfloat16(), rnd(T, H)
    res = rnd(T, H) if residual else None
    y, rstd, *rest = C.rmsnorm_fwd(x, res, w, 1e-6)
    h = (x.float() + res.float()).bfloat16() if residual else x
    if residual:
        assert torch.equal(rest[0], h)
    hd, wd = h.double().requires_grad_(True), w.double().requires_grad_(True)
    ref = hd * torch.rsqrt(hd.square().mean(-1, keepdim=True) + 1e-6) * wd
    # one rounding to bf16 (half a unit of 7 fraction bits: 2^-8 of the value) of what is computed in fp32
    assert ((y.double() - ref).abs() <= 2 ** -8 * ref.abs() + 1e-6).all()
    ref.backward(dy.double())
    dw = torch.ones(H, device=DEV)
    dx = C.rmsnorm_bwd(dy, h, w, rstd, res, dw, True)
    want = hd.grad + (res.double() if residual else 0)
    assert ((dx.double() - want).abs() <= 2 ** -8 * want.abs() + 1e-4).all()
    assert ((dw.double() - 1 - wd.grad).norm() <= 1e-5 * wd.grad.norm() + 1e-5 * H ** 0.5).item()
