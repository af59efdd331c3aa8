"""Log-probabilities and entropies that leave with the LM head's product, against its logits in 64 bits and the kernel over whole rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


# vocabularies below a tile, ending inside a chunk, a half and a tile; rows with remainders, a pair's second CTA empty; targets outside
@pytest.mark.parametrize("T, V, K", [(1, 40, 64), (129, 128, 64), (300, 1000, 136), (256, 1160, 512), (33, 151936, 64), (700, 4096, 2048)])
@pytest.mark.parametrize("pair", [1, 2])
@pytest.mark.parametrize("keep", [False, True])
def test_against_logits(T, V, K, pair, keep):
    from miles_b200.ops import _ext

    C = _ext.load(required=True)
    g = torch.Generator(device=DEV).manual_seed(T + V)
    h, w = torch.randn(T, K, device=DEV, generator=g).bfloat16(), (torch.randn(V, K, device=DEV, generator=g) * 3 * K ** -0.5).bfloat16()
    tg = torch.randint(0, V, (T,), device=DEV, generator=g).int()
    tg[0], tg[-1] = V - 1, (-1 if T > 1 else 0)
    inv_t = 1 / 0.7
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    want = torch.empty(T, V, device=DEV)
    C.gemm(h, w, want, False, False, False, 256, st, pair=1)
    buf = torch.full((T, V + 4), 5.0, device=DEV)
    lp, ent, lse, px = C.score_rows(h, w, tg, inv_t, buf[:, :V] if keep else None, st, pair=pair)
    assert st.item() == 0
    if keep:
        assert torch.equal(buf[:, :V], want) and (buf[:, V:] == 5).all()
    x = want.double() * inv_t
    ref_lse = torch.logsumexp(x, -1)
    ref_px = (torch.softmax(x, -1) * x).sum(-1)
    ref_lp = torch.where(tg >= 0, x.gather(1, tg.clamp(min=0).long()[:, None])[:, 0] - ref_lse, 0.0)
    # an exponential's weight is off by 2^-22 for itself and for every unit of its argument (rounded to 24 bits), a mean of x by that
    # times the spread of x; and no further off, over the rows, than the kernel that reads the logits
    tol = 2 ** -22 * (1 + x.abs().max().item()) ** 2
    one = C.logprob_entropy_fwd(want, tg, inv_t)
    for got, ref, old in zip((lp, ent, lse, px), (ref_lp, ref_lse - ref_px, ref_lse, ref_px), one):
        assert (got.double() - ref).abs().max().item() < tol
        assert (got.double() - ref).norm().item() <= 1.5 * (old.double() - ref).norm().item() + 1e-6 * T ** 0.5


def test_no_rows_and_wide_scores():
    from miles_b200.ops import _ext

    C = _ext.load(required=True)
    w = torch.zeros(512, 64, device=DEV).bfloat16()
    w[7, 0], w[300, 0] = 1e4, -1e4
    h = torch.zeros(3, 64, device=DEV).bfloat16()
    h[0, 0], h[1, 0] = 1.0, -1.0
    tg = torch.tensor([7, 7, 0], dtype=torch.int32, device=DEV)
    lp, ent, lse, _ = C.score_rows(h, w, tg, 1.0, None, None)
    big = float(w[7, 0])
    assert lp[0] == 0 and lse[0] == big and ent[0] == 0 and lp[1] == -2 * big and lse[1] == big
    assert abs(lse[2].item() - torch.log(torch.tensor(512.0)).item()) < 1e-5 and abs(ent[2].item() - lse[2].item()) < 1e-5
    assert all(t.numel() == 0 for t in C.score_rows(h[:0], w, tg[:0], 1.0, None, None))


@pytest.mark.parametrize("vocab", [4096, 31992, 32000])
def test_a_row_scores_the_same_in_any_company(vocab):
    """However many rows there are, are scored at a time, or keep their logits. (Up to 32 rows, heads below SCORE_VOCAB take the
    engine's products, whose sums are split.)"""
    from miles_b200.models import ParamStore, build_model, get_config

    cfg = get_config("qwen3-smoke")
    cfg.vocab_size = vocab
    model = build_model(cfg, ParamStore(cfg, torch.device(DEV), torch.bfloat16, init_std=0.05, seed=3), "b200")
    g = torch.Generator(device=DEV).manual_seed(vocab)
    h = torch.randn(3000, cfg.hidden_size, device=DEV, generator=g).bfloat16()
    tg = torch.randint(0, vocab, (3000,), device=DEV, generator=g)
    want = model.logprobs_entropy(h, tg, 1.0, keep_stats=True)
    assert model._fused_scores(vocab) == (vocab == 32000)
    for n in (33, 128, 129, 2048, 2999) + ((1, 8, 32) if vocab == 32000 else ()):
        for kw in (dict(), dict(keep_logits=[]), dict(chunk=128), dict(chunk=128, keep_logits=[])):
            if n % kw.get("chunk", 2048) in range(1, 33) and vocab < 32000:
                continue
            got = model.logprobs_entropy(h[:n], tg[:n], 1.0, keep_stats=True, **kw)
            assert all(torch.equal(a, b[:n]) for a, b in zip(got, want)), (n, kw)
    model.check_status()
