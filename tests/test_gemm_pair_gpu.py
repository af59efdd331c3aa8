"""GEMM tiles of two CTAs against those of one: the same sums in the same order, so the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


# one tile and its edges: rows that leave the second CTA empty or with one row, columns and contractions with remainders (also one
# that ends before the second CTA's half), contractions longer and shorter than the ring, more tiles than pairs of SMs
@pytest.mark.parametrize("M, N, K", [(256, 256, 64), (129, 256, 384), (128, 512, 512), (257, 264, 72), (300, 136, 1000), (777, 2048, 2048),
                                     (5000, 1032, 328), (2048, 4096, 128)])
@pytest.mark.parametrize("a_mn, b_mn", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("fp32, acc", [(False, False), (True, False), (False, True), (True, True)])
def test_dense_pairs(M, N, K, a_mn, b_mn, fp32, acc):
    from miles_b200.ops import _ext

    C = _ext.load(required=True)
    if (a_mn and M % 8) or (b_mn and N % 8) or (not (a_mn and b_mn) and K % 8):
        pytest.skip("rows of an operand are whole 16-byte pieces")
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g).bfloat16()  # noqa: E731
    a, b = rnd(*((K, M) if a_mn else (M, K))), rnd(*((K, N) if b_mn else (N, K)))
    c0 = torch.randn(M, N, device=DEV, generator=g).to(torch.float32 if fp32 else torch.bfloat16)
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    c1, c2 = c0.clone(), c0.clone()
    C.gemm(a, b, c1, a_mn, b_mn, acc, 256, st, pair=1)
    C.gemm(a, b, c2, a_mn, b_mn, acc, 256, st, pair=2)
    assert st.item() == 0
    assert torch.equal(c1, c2)
    af, bf = (a.t() if a_mn else a).float(), (b.t() if b_mn else b).float()
    want = af @ bf.t() + (c0.float() if acc else 0)
    assert ((c2.float() - want).norm() / want.norm()).item() < 5e-3
