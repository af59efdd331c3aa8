"""The attention backward's tiles at their edges: sequences that end inside a tile, share one with a neighbour, or are shorter than a
tile, and rows that another sequence's tile reaches."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SCALE = 128 ** -0.5
EPS = 2.0 ** -8  # rounding to bf16, 8 significant bits: half of 2^-7, relative to a value of 1 up to 2


def _inputs(T, Hq, Hk):
    g = torch.Generator(device="cuda").manual_seed(11)
    return [torch.randn(T, h, 128, device="cuda", generator=g).bfloat16() for h in (Hq, Hk, Hk, Hq)]


def _run(q, k, v, do, lens, split=1):
    from miles_b200.ops import _ext
    from miles_b200.ops.attention import build_bwd_blocks, build_tiles

    C = _ext.load(required=True)
    st = torch.zeros(1, dtype=torch.int32, device="cuda")
    o, lse = C.flash_attn_fwd(q, k, v, build_tiles(lens).cuda(), SCALE, st)
    grads = C.flash_attn_bwd(q, k, v, o, do, lse, build_bwd_blocks(lens).cuda(), SCALE, st, split=split)
    assert int(st.item()) == 0
    return o, grads


def _check(q, k, v, do, o, grads, a, b):
    """Gradients of rows a:b, one sequence, against 64 bits. P and dS are rounded to bf16 before their products and D is summed from the
    rounded O: that and the result's own rounding bound the error, with a tenth more for the 32-bit sums and the exponential."""
    Hq, Hk = q.shape[1], k.shape[1]
    n, rep = b - a, q.shape[1] // k.shape[1]
    Q, DO, O = (t[a:b].double().transpose(0, 1) for t in (q, do, o))
    K, V = (t[a:b].double().transpose(0, 1).repeat_interleave(rep, 0) for t in (k, v))
    S = (Q @ K.transpose(1, 2) * SCALE).masked_fill(~torch.ones(n, n, dtype=torch.bool, device="cuda").tril(), float("-inf"))
    P = S.softmax(-1)
    D = (DO * (P @ V)).sum(-1, keepdim=True)
    dS = P * (DO @ V.transpose(1, 2) - D)
    e_ds = EPS * (dS.abs() + P * (DO.abs() * O.abs()).sum(-1, keepdim=True))
    heads = lambda t: t.view(Hk, rep, n, 128).sum(1)
    want = (SCALE * dS @ K, heads(SCALE * dS.transpose(1, 2) @ Q), heads(P.transpose(1, 2) @ DO))
    err = (SCALE * e_ds @ K.abs(), heads(SCALE * e_ds.transpose(1, 2) @ Q.abs()), heads(EPS * P.transpose(1, 2) @ DO.abs()))
    for got, w, e in zip(grads, want, err):
        off = (got[a:b].double().transpose(0, 1) - w).abs()
        assert (off <= 1.1 * (e + EPS * w.abs()) + 1e-6).all(), float((off - 1.1 * (e + EPS * w.abs())).max())


@pytest.mark.parametrize("lens", [[1], [63, 65], [64, 128, 1], [127, 129, 200], [5, 700, 128, 1, 300]])
@pytest.mark.parametrize("Hq,Hk", [(4, 1), (2, 2), (8, 4)])
def test_edges_of_tiles(lens, Hq, Hk):
    q, k, v, do = _inputs(sum(lens), Hq, Hk)
    o, grads = _run(q, k, v, do, lens)
    a = 0
    for n in lens:
        _check(q, k, v, do, o, grads, a, a + n)
        a += n


@pytest.mark.parametrize("first", [1, 40, 100, 129])
def test_a_sequence_leaves_the_next_one_alone(first):
    lens = [first, 150]
    q, k, v, do = _inputs(sum(lens), 4, 2)
    for t in (q, k, v, do):
        t[:first] = float("nan")
    o, grads = _run(q, k, v, do, lens)
    _check(q, k, v, do, o, grads, first, first + 150)


def test_rows_that_start_off_a_16_byte_boundary():
    from miles_b200.ops import _ext
    from miles_b200.ops.attention import build_bwd_blocks, build_tiles

    C = _ext.load(required=True)
    q, k, v, do = _inputs(100, 4, 2)
    st = torch.zeros(1, dtype=torch.int32, device="cuda")
    o, lse = C.flash_attn_fwd(q, k, v, build_tiles([100]).cuda(), SCALE, st)
    shifted = torch.empty(o.numel() + 4, dtype=o.dtype, device="cuda")[4:].view(o.shape)
    shifted.copy_(o)
    blocks = build_bwd_blocks([100]).cuda()
    _check(q, k, v, do, o, C.flash_attn_bwd(q, k, v, shifted, do, lse, blocks, SCALE, st), 0, 100)


# a lone row, a block's edges, more blocks than the device has room for at once; every number of CTAs that divides the heads
@pytest.mark.parametrize("lens", [[1], [127, 129], [200] * 12])
@pytest.mark.parametrize("Hq,Hk,split", [(8, 4, 2), (16, 2, 1), (16, 2, 2), (16, 2, 4), (12, 1, 4)])
def test_heads_shared_by_a_cluster(lens, Hq, Hk, split):
    q, k, v, do = _inputs(sum(lens), Hq, Hk)
    o, grads = _run(q, k, v, do, lens, split)
    a = 0
    for n in lens:
        _check(q, k, v, do, o, grads, a, a + n)
        a += n


@pytest.mark.parametrize("which", ["q", "k", "v", "d_o"])
def test_misaligned_operands_are_refused_before_anything_reads_them(which):
    """Nothing is launched: the refusal comes from the host, and what follows on the stream runs."""
    from miles_b200.ops import _ext
    from miles_b200.ops.attention import build_bwd_blocks, build_tiles

    C = _ext.load(required=True)
    t = dict(zip(("q", "k", "v", "d_o"), _inputs(100, 4, 2)))
    o, lse = C.flash_attn_fwd(t["q"], t["k"], t["v"], build_tiles([100]).cuda(), SCALE, None)
    off = torch.empty(t[which].numel() + 8, dtype=torch.bfloat16, device="cuda")[4:-4].view(t[which].shape)
    assert off.data_ptr() % 16 == 8 and off.is_contiguous()
    t[which] = off.copy_(t[which])
    with pytest.raises(RuntimeError, match="16-byte aligned"):
        C.flash_attn_bwd(t["q"], t["k"], t["v"], o, t["d_o"], lse, build_bwd_blocks([100]).cuda(), SCALE, None)
    torch.cuda.synchronize()
