"""The staged GEMM epilogue where it branches: adding to and setting fp32 and bf16 outputs, widths that end inside a chunk of
columns, rows that end inside a warp's 32, more tiles than CTAs, groups without rows between groups with some."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ext():
    from miles_b200.ops import _ext

    return _ext.load(required=True)


def _close(got, want, size, k):
    # fp32 sums of k products in any order, one addition, one rounding to the output's type
    bound = size * (k ** 0.5 + 1) * 2 ** -22 + want.abs() * (2 ** -8 if got.dtype == torch.bfloat16 else 2 ** -22)
    assert ((got.double() - want).abs() <= bound).all()


@pytest.mark.parametrize("block_n", [64, 128, 256])
@pytest.mark.parametrize("M,N,K", [(129, 64, 64), (333, 328, 200), (200, 2104, 64), (2500, 2056, 72)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("add", [False, True])
def test_dense_outputs(ext, block_n, M, N, K, dtype, add):
    g = torch.Generator(DEV).manual_seed(M + N + block_n)
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    a, b = torch.randn(M, K, generator=g, device=DEV).bfloat16(), torch.randn(N, K, generator=g, device=DEV).bfloat16()
    old = torch.randn(M, N + 16, generator=g, device=DEV).to(dtype)
    out = old.clone()
    ext.gemm(a, b, out[:, :N], False, False, add, block_n, st)
    want, size = a.double() @ b.double().t(), a.double().abs() @ b.double().abs().t()
    if add:
        want, size = want + old[:, :N].double(), size + old[:, :N].double().abs()
    _close(out[:, :N], want, size, K)
    assert torch.equal(out[:, N:], old[:, N:]) and st.item() == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("M,N", [(128, 64), (200, 328), (1536, 512)])
@pytest.mark.parametrize("add", [False, True])
def test_grouped_weight_gradients(ext, dtype, M, N, add):
    g = torch.Generator(DEV).manual_seed(M + N)
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    rows = [0, 64, 0, 0, 192, 64, 0] * 6
    off = torch.tensor([0] + rows).cumsum(0).to(torch.int32).to(DEV)
    a, b = (torch.randn(sum(rows), n, generator=g, device=DEV).bfloat16() for n in (M, N))
    old = torch.randn(len(rows), M, N, generator=g, device=DEV).to(dtype)
    out = old.clone()
    ext.grouped_gemm_contr(a, b, out, off, add, 0, st)
    for e, n in enumerate(rows):
        x, y = a[off[e]:off[e] + n].double(), b[off[e]:off[e] + n].double()
        want, size = x.t() @ y, x.abs().t() @ y.abs()
        if add:
            want, size = want + old[e].double(), size + old[e].double().abs()
        _close(out[e], want, size, max(n, 1))
    assert st.item() == 0
