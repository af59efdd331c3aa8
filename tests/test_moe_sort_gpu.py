"""The expert sort where its split over warps and blocks changes: one entry, part of a warp, the last size of the one-block
variant and the first of the other, more experts than a block has threads; ids outside the experts and too little room."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ext():
    from miles_b200.ops import _ext

    return _ext.load(required=True)


def _expected(ids, E, max_rows, align):
    flat = ids.reshape(-1).tolist()
    counts = [0] * E
    for e in flat:
        if 0 <= e < E:
            counts[e] += 1
    cap = max_rows // align * align
    off, run = [], 0
    for c in counts:
        off.append(min(run, cap))
        run += -(-c // align) * align
    off.append(min(run, cap))
    dest, src, seen = [], [-1] * max_rows, [0] * E
    for i, e in enumerate(flat):
        row = -1
        if 0 <= e < E:
            if seen[e] < off[e + 1] - off[e]:
                row = off[e] + seen[e]
                src[row] = i
            seen[e] += 1
        dest.append(row)
    tiles = [[e, off[e] + j, min(128, off[e + 1] - off[e] - j), 0] for e in range(E) for j in range(0, off[e + 1] - off[e], 128)]
    return counts, off, dest, src, tiles


@pytest.mark.parametrize("T,K,E", [(1, 1, 1), (1, 8, 128), (16, 8, 128), (43, 3, 5), (64, 8, 128), (65, 8, 128), (512, 8, 512), (513, 8, 128),
                                   (2049, 8, 1500), (9001, 8, 160), (700, 8, 12288), (700, 8, 12289), (700, 8, 14500)])
@pytest.mark.parametrize("align", [1, 64])
@pytest.mark.parametrize("short", [False, True])
def test_expert_sort_equals_a_sequential_one(ext, T, K, E, align, short):
    g = torch.Generator().manual_seed(T * 31 + K + E)
    ids = (torch.rand(T, K, generator=g) ** 2 * E).long().clamp_max(E - 1).to(torch.int32)  # low experts are popular
    if T > 8:
        ids[3, 0], ids[T - 1, K - 1] = -1, E
    max_rows = T * K + E * (align - 1)
    if short:
        max_rows = max(align, max_rows // 2)
    counts, off, dest, src, tiles = _expected(ids, E, max_rows, align)
    got = ext.moe_build_permutation(ids.to(DEV), E, max_rows, align)
    assert got[0].tolist() == counts and got[1].tolist() == off and got[2].tolist() == dest and got[3].tolist() == src
    assert got[5].tolist() == [len(tiles), off[-1]] and got[4][:len(tiles)].tolist() == tiles


def test_more_experts_than_shared_memory_holds_are_refused(ext):
    ids = torch.zeros(700, 8, dtype=torch.int32, device=DEV)
    with pytest.raises(RuntimeError, match="20000 experts"):
        ext.moe_build_permutation(ids, 20000, 5600, 1)
    assert ext.moe_build_permutation(ids, 16, 5600, 1)[0].tolist() == [5600] + [0] * 15  # the refusal leaves no error behind


@pytest.mark.parametrize("T,E,K", [(1, 16, 1), (1, 128, 8), (8, 128, 8), (5, 160, 6), (8, 1024, 32)])
def test_small_router_lists(ext, T, E, K):
    g = torch.Generator().manual_seed(T + E)
    logits = torch.randn(T, E, generator=g).to(DEV)
    logits[:, 1] = logits[:, 0]  # ties go to the lower expert
    ids, w = torch.empty(T, K, dtype=torch.int32, device=DEV), torch.empty(T, K, device=DEV)
    active, count, lists = (torch.full((n,), -1, dtype=torch.int32, device=DEV) for n in (1 + E, E, 8 * E))
    ext.router_small(logits, K, True, ids, w, active, count, lists)
    order = sorted(range(E), key=lambda e: e)
    for t in range(T):
        row = logits[t].tolist()
        assert ids[t].tolist() == sorted(order, key=lambda e: -row[e])[:K]
    p = torch.softmax(logits.double(), -1).gather(1, ids.long())
    assert torch.allclose(w.double(), p / p.sum(-1, keepdim=True), rtol=1e-5)  # fast exponentials: about 2^-20 each
    used = sorted(set(ids.flatten().tolist()))
    assert active[:1 + len(used)].tolist() == [len(used)] + used
    for e in range(E):
        pairs = [t * K + k for t in range(T) for k in range(K) if int(ids[t, k]) == e]
        assert int(count[e]) == len(pairs) and lists[8 * e:8 * e + len(pairs)].tolist() == pairs


@pytest.mark.parametrize("T,K,H", [(1, 8, 2048), (5, 1, 64), (300, 16, 1032), (7, 6, 72)])
def test_permute_and_combine_at_odd_widths(ext, T, K, H):
    g = torch.Generator().manual_seed(T + H)
    E = 16
    ids = torch.stack([torch.randperm(E, generator=g)[:K] for _ in range(T)]).to(torch.int32).to(DEV)
    x, res = (torch.randn(T, H, generator=g).bfloat16().to(DEV) for _ in range(2))
    w = torch.rand(T, K, generator=g).to(DEV)
    _, _, dest, src, _, nt = ext.moe_build_permutation(ids, E, T * K + E * 7, 8)
    xp = ext.moe_permute(x, src, nt, K)
    live = int(nt[1])
    want = torch.where(src[:live, None] >= 0, x[(src[:live].long() // K).clamp_min(0)], 0)
    assert torch.equal(xp[:live], want)
    y = torch.randn(xp.shape, generator=g).bfloat16().to(DEV)
    dest[K - 1] = -1  # a choice without a row
    rows = y[dest.long().clamp_min(0)].double().view(T, K, H) * (dest >= 0).view(T, K, 1)
    want = (rows * w.double()[..., None]).sum(1) + res.double()
    got = ext.moe_combine(y, dest, w, T, K, res)
    assert (got.double() - want).abs().max() <= 2 ** -8 * want.abs().max()  # one bf16 rounding of fp32 sums
    dout = torch.randn(T, H, generator=g).bfloat16().to(DEV)
    dy, dw = ext.moe_combine_bwd(dout, y, src, nt, w)
    at = src[:live].long()
    pick = at.clamp_min(0)
    assert torch.equal(dy[:live], torch.where(at[:, None] >= 0, (dout[pick // K].float() * w.view(-1)[pick][:, None]).bfloat16(), 0))
    dots = (dout[pick // K].double() * y[:live].double()).sum(-1)
    size = (dout[pick // K].double() * y[:live].double()).abs().sum(-1)
    assert ((dw.view(-1)[pick].double() - dots).abs() <= 1e-5 * size)[at >= 0].all()
