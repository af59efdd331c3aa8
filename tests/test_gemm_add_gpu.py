"""Weight gradients that add to what is there: the sums of the plain product, added in fp32 and rounded once, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _c():
    from miles_b200.ops import _ext

    return _ext.load(required=True), torch.zeros(1, dtype=torch.int32, device="cuda")


def _bf(*s):
    return torch.randn(*s, device="cuda", generator=torch.Generator(device="cuda").manual_seed(sum(s))).bfloat16()


def _old(shape, dtype):
    return torch.randn(shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(7)).mul_(30).to(dtype)


# a lone row, rows that end inside a warp's, one piece of columns, several tiles a CTA; contractions that end inside a block of 64, of
# one block, and too long for the small variants; pairs; columns that end inside a piece
@pytest.mark.parametrize("M, N, K, bn, pair", [(8, 64, 8, 0, 0), (152, 192, 200, 128, 1), (1000, 128, 60, 128, 1), (4104, 4096, 72, 128, 1),
                                               (72, 320, 64, 256, 1), (5000, 2048, 333, 256, 1), (3000, 2048, 790, 256, 1), (3000, 2048, 810, 256, 1), (3000, 2048, 1100, 256, 1),
                                               (1000, 1088, 640, 256, 2), (6016, 2048, 100, 256, 2), (200, 200, 96, 0, 0)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_adds_to_what_is_there(M, N, K, bn, pair, dtype):
    C, st = _c()
    a, b = _bf(K, M), _bf(K, N)
    product = torch.empty(M, N, device="cuda")
    C.gemm(a, b, product, True, True, False, bn, st, pair=pair)
    wide = _old((M, N + 64), dtype)  # (a row pitch of its own; the columns beside stay as they are)
    want = wide.clone()
    want[:, :N] = (want[:, :N].float() + product).to(dtype)
    C.gemm(a, b, wide[:, :N], True, True, True, bn, st, pair=pair)
    assert torch.equal(wide, want) and int(st.item()) == 0


# groups without rows, of one block, of several; capacities per group on each side of the lines between the variants
@pytest.mark.parametrize("rows", [[64, 0, 192, 0, 0, 64, 128, 0], [0, 448, 512, 640, 0, 512, 576, 640], [1024, 64, 1984, 960, 0, 1088, 2048, 1024],
                                  [0] * 8])
@pytest.mark.parametrize("M, N", [(256, 512), (200, 128), (1536, 2048)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_groups_add_to_theirs(rows, M, N, dtype):
    C, st = _c()
    off = torch.tensor([0] + rows).cumsum(0).int().cuda()
    total = max(int(off[-1]), 64)
    a, b = _bf(total, M), _bf(total, N)
    grads = _old((8, M, N), dtype)
    want = grads.clone()
    for g in range(8):
        lo, hi = int(off[g]), int(off[g + 1])
        if hi > lo:
            product = torch.empty(M, N, device="cuda")
            C.gemm(a[lo:hi], b[lo:hi], product, True, True, False, 0, st, pair=1)
            want[g] = (want[g].float() + product).to(dtype)
    C.grouped_gemm_contr(a, b, grads, off, True, 0, st)
    assert torch.equal(grads, want) and int(st.item()) == 0
