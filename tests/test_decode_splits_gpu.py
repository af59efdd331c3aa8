"""Decode attention where its paths part: pages of whole chunks, smaller and larger ones, one split, clusters up to 16, more
splits through scratch, slices without a token, lengths at the edges of a chunk, and a page outside the cache."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV, D = "cuda", 128


@pytest.mark.parametrize("page_size", [16, 48, 64, 128])
@pytest.mark.parametrize("splits", [1, 2, 3, 8, 13, 16, 17, 24])
@pytest.mark.parametrize("Hq,Hk", [(8, 1), (8, 2), (4, 2), (3, 3)])
def test_splits_and_pages(page_size, splits, Hq, Hk):
    from miles_b200.ops import _ext

    ext = _ext.load(required=True)
    g = torch.Generator().manual_seed(page_size + splits)
    lens = [1, 63, 64, 65, 200, 1025, 0]
    pages = [-(-n // page_size) for n in lens]
    slots = (sum(pages) + 2) * page_size
    kc, vc = (torch.randn(slots, Hk, D, generator=g).bfloat16() for _ in range(2))
    order, at = torch.randperm(sum(pages), generator=g), 0
    table = torch.zeros(len(lens), max(pages) + 1, dtype=torch.int32)
    for b, n in enumerate(pages):
        table[b, :n] = order[at:at + n].int()
        at += n
    used = torch.zeros(slots, dtype=torch.bool)
    for b, n in enumerate(lens):
        t = torch.arange(n)
        used[table[b].long()[t // page_size] * page_size + t % page_size] = True
    kc[~used], vc[~used] = float("nan"), float("nan")  # what no sequence holds must not be looked at
    q = torch.randn(len(lens), Hq, D, generator=g).bfloat16()
    want = torch.zeros(len(lens), Hq, D, dtype=torch.float64)
    for b, n in enumerate(lens):
        if n:
            t = torch.arange(n)
            s = table[b].long()[t // page_size] * page_size + t % page_size
            k, v = (c[s].double().repeat_interleave(Hq // Hk, 1) for c in (kc, vc))
            want[b] = torch.einsum("ht,thd->hd", torch.softmax(torch.einsum("hd,thd->ht", q[b].double(), k) * D ** -0.5, -1), v)
    out = torch.full((len(lens), Hq, D), 7.0, device=DEV, dtype=torch.bfloat16)
    scratch = torch.empty(len(lens) * Hq * splits * 130, device=DEV)
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    args = (scratch, page_size, splits, D ** -0.5, st)
    ext.paged_decode_attention(q.to(DEV), kc.to(DEV), vc.to(DEV), table.to(DEV), torch.tensor(lens, dtype=torch.int32).to(DEV), out, *args)
    # probabilities and the result are rounded to bf16 (2^-9 each) around values of size one
    assert st.item() == 0 and (out.cpu().double() - want).abs().max() < 2.5e-2
    table[3, 0] = slots  # a page that does not exist reads as zeros and is reported
    ext.paged_decode_attention(q.to(DEV), kc.to(DEV), vc.to(DEV), table.to(DEV), torch.tensor(lens, dtype=torch.int32).to(DEV), out, *args)
    assert st.item() == 9 and torch.isfinite(out).all()
