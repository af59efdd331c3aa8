"""Rows of the experts in their order and back, where they fit into half of L2 and where they pass it by: the same values."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("T, align", [(2047, 1), (2049, 1), (1800, 64), (4100, 64)])
def test_rows_above_and_below_half_of_l2(T, align):
    from miles_b200.ops import _ext

    C = _ext.load(required=True)
    E, K, H = 16, 8, 2048
    g = torch.Generator(device=DEV).manual_seed(T)
    ids = torch.rand(T, E, device=DEV, generator=g).topk(K, -1).indices.int().contiguous()
    R = T * K + E * (align - 1)
    _, _, dest, src, _, nt = C.moe_build_permutation(ids, E, R, align)
    x, w = torch.randn(T, H, device=DEV, generator=g).bfloat16(), torch.rand(T, K, device=DEV, generator=g)
    y = torch.randn(R, H, device=DEV, generator=g).bfloat16()
    xp = C.moe_permute(x, src, nt, K)
    live = int(nt[1])
    has = src[:live] >= 0
    assert torch.equal(xp[:live][has], x[(src[:live][has] // K).long()]) and not xp[:live][~has].any()
    out = C.moe_combine(y, dest, w, T, K, x)
    half = T // 2  # (fewer tokens at a time stay below)
    parts = [C.moe_combine(y, d.contiguous(), v.contiguous(), v.shape[0], K, r.contiguous())
             for d, v, r in zip(dest.view(T, K).split([half, T - half]), w.split([half, T - half]), x.split([half, T - half]))]
    assert torch.equal(out, torch.cat(parts))
    dy, dw = C.moe_combine_bwd(x, y, src, nt, w)
    at = src[:live][has].long()
    want = (w.flatten()[at, None] * x[at // K].float()).bfloat16()
    assert torch.equal(dy[:live][has], want) and not dy[:live][~has].any()
    dots = (x[at // K].double() * y[:live][has].double()).sum(-1)
    # sums of 2048 products in fp32: 2^-24 of the sum of their sizes for each of some 70 additions in a row
    size = (x[at // K].double() * y[:live][has].double()).abs().sum(-1)
    assert ((dw.flatten()[at] - dots).abs() <= 70 * 2 ** -24 * size).all()
