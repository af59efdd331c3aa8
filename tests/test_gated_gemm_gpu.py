"""Products with SwiGLU in the epilogue against the product and the activation kernel: the same bits, and gate and up beside them."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


# widths below, at and above a tile's 128 columns, with remainders; rows with remainders and a pair's second CTA empty; one and many tiles
@pytest.mark.parametrize("M, I, K", [(1, 8, 64), (129, 128, 512), (300, 200, 136), (256, 1032, 64), (3000, 776, 2048), (5000, 2560, 256)])
@pytest.mark.parametrize("pair", [1, 2])
def test_dense(M, I, K, pair):
    from miles_b200.ops import _ext

    C = _ext.load(required=True)
    g = torch.Generator(device=DEV).manual_seed(M + I)
    x, w = torch.randn(M, K, device=DEV, generator=g).bfloat16(), (torch.randn(2 * I, K, device=DEV, generator=g) * 0.1).bfloat16()
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    want = torch.empty(M, 2 * I, device=DEV, dtype=torch.bfloat16)
    C.gemm(x, w, want, False, False, False, 256, st, pair=1)
    guard = torch.full((M, 2 * I + 8), 7.0, device=DEV, dtype=torch.bfloat16)  # (rows with a pitch, nothing behind them touched)
    act = torch.full((M, I + 8), 7.0, device=DEV, dtype=torch.bfloat16)
    C.gated_gemm(x, w, act[:, :I], guard[:, :2 * I], None, None, st, pair=pair)
    assert st.item() == 0
    assert torch.equal(guard[:, :2 * I], want) and torch.equal(act[:, :I], C.swiglu_fwd(want))
    assert (guard[:, 2 * I:] == 7).all() and (act[:, I:] == 7).all()
    only = torch.empty(M, I, device=DEV, dtype=torch.bfloat16)
    C.gated_gemm(x, w, only, None, None, None, st, pair=pair)
    assert torch.equal(only, act[:, :I])


@pytest.mark.parametrize("T, E, K, I, align", [(5, 16, 2, 96, 1), (64, 128, 8, 768, 1), (700, 8, 2, 136, 64), (2000, 128, 8, 256, 1)])
def test_grouped(T, E, K, I, align):
    from miles_b200.ops import _ext

    C = _ext.load(required=True)
    H = 256
    g = torch.Generator(device=DEV).manual_seed(T)
    ids = torch.rand(T, E, device=DEV, generator=g).topk(K, -1).indices.int()
    rows = T * K + E * (align - 1)
    _, _, _, _, tg, nt = C.moe_build_permutation(ids, E, rows, align)
    x, w = torch.randn(rows, H, device=DEV, generator=g).bfloat16(), (torch.randn(E, 2 * I, H, device=DEV, generator=g) * 0.1).bfloat16()
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    want, gu = torch.zeros(rows, 2 * I, device=DEV).bfloat16(), torch.zeros(rows, 2 * I, device=DEV).bfloat16()
    act, only = torch.zeros(rows, I, device=DEV).bfloat16(), torch.zeros(rows, I, device=DEV).bfloat16()
    C.grouped_gemm_rows(x, w, want, tg, nt, False, False, 0, st)
    C.gated_gemm(x, w, act, gu, tg, nt, st)
    C.gated_gemm(x, w, only, None, tg, nt, st)
    assert st.item() == 0
    assert torch.equal(gu, want) and torch.equal(act, C.swiglu_fwd(want)) and torch.equal(only, act)


def test_extremes():
    from miles_b200.ops import _ext

    C = _ext.load(required=True)
    x, w = torch.zeros(4, 64, device=DEV).bfloat16(), torch.zeros(16, 64, device=DEV).bfloat16()
    x[0, 0], x[1, 0], x[2, 0], x[3, 0] = 1.0, -1.0, float("inf"), float("nan")
    w[:8, 0], w[8:, 0] = 300.0, 2.0  # gates of 300 and -300: silu of the latter is -0
    gu, act = torch.empty(4, 16, device=DEV).bfloat16(), torch.empty(4, 8, device=DEV).bfloat16()
    C.gated_gemm(x, w, act, gu, None, None, None)
    assert torch.equal(act.view(torch.int16), C.swiglu_fwd(gu).view(torch.int16))
    assert (act[0] == 600).all() and (act[1] == 0).all() and (act[2] == float("inf")).all() and act[3].isnan().all()  # silu(inf) = inf
