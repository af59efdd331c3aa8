"""The split product of few rows where its tiles, splits and rings change: one row, the edges of every token tile, an output
narrower than a tile, contractions shorter than the ring or not a multiple of a block, or cut so that the last CTA of the
cluster gets none of it (33 and 42 blocks over eight), strided rows, fp32 and residual."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ext():
    from miles_b200.ops import _ext

    return _ext.load(required=True)


def _check(got, x, w, res=None):
    want = x.double() @ w.double().t()
    size = x.double().abs() @ w.double().abs().t()
    if res is not None:
        want = want + res.double()
    # products summed in fp32 in any order, then one rounding to the output's type
    bound = size * x.shape[1] ** 0.5 * 2 ** -24 * 4 + (want.abs() * 2 ** -8 if got.dtype == torch.bfloat16 else want.abs() * 2 ** -23)
    assert ((got.double() - want).abs() <= bound).all()


@pytest.mark.parametrize("T", [1, 9, 16, 17, 32, 33, 64, 65, 93, 128])
@pytest.mark.parametrize("N,K", [(8, 64), (128, 2048), (130, 72), (2048, 4096), (5120, 2048), (2560, 1000), (12296, 520), (57000, 64), (2048, 2112), (130, 2632)])
def test_product_of_few_rows(ext, T, N, K):
    g = torch.Generator(DEV).manual_seed(T * N + K)
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    x = torch.randn(T, K + 8, generator=g, device=DEV).bfloat16()[:, :K]  # rows longer than the contraction
    w = torch.randn(N, K, generator=g, device=DEV).bfloat16()
    for dtype in (torch.bfloat16, torch.float32):
        out = torch.full((T, N + 5), 7.0, device=DEV, dtype=dtype)
        ext.gemm(x, w, out[:, :N], False, False, False, 0, st)
        _check(out[:, :N], x, w)
        assert (out[:, N:] == 7).all()
    if T <= 64 and K % 32 == 0 and N % 16 == 0:
        res = torch.randn(T, N, generator=g, device=DEV).bfloat16()
        out = torch.empty(T, N, device=DEV, dtype=torch.bfloat16)
        ext.small_gemv(x.contiguous(), None, 0.0, w, res, out, st)
        _check(out, x, w, res)
    assert st.item() == 0


def test_repeated_products_are_bitwise_equal(ext):
    g = torch.Generator(DEV).manual_seed(0)
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    x, w = torch.randn(23, 9728, generator=g, device=DEV).bfloat16(), torch.randn(2560, 9728, generator=g, device=DEV).bfloat16()
    outs = [torch.empty(23, 2560, device=DEV, dtype=torch.bfloat16) for _ in range(4)]
    for o in outs:
        ext.gemm(x, w, o, False, False, False, 0, st)
    assert all(torch.equal(o, outs[0]) for o in outs)


@pytest.mark.parametrize("T", [33, 64, 65, 128])
@pytest.mark.parametrize("N,K", [(130, 2632), (2048, 2048), (2560, 9728)])
def test_whole_contractions_do_not_depend_on_the_rows(ext, T, N, K):
    g = torch.Generator(DEV).manual_seed(T + N)
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    x, w = torch.randn(300, K, generator=g, device=DEV).bfloat16(), torch.randn(N, K, generator=g, device=DEV).bfloat16()
    for dtype in (torch.bfloat16, torch.float32):
        few, many = (torch.empty(n, N, device=DEV, dtype=dtype) for n in (T, 300))
        ext.gemm(x[:T], w, few, False, False, False, 0, st, whole_k=True)
        ext.gemm(x, w, many, False, False, False, 0, st)
        assert torch.equal(few, many[:T])
        _check(few, x[:T], w)
    assert st.item() == 0


@pytest.mark.parametrize("name", ["qwen3-smoke", "qwen3-smoke-moe", "glm4-smoke"])
@pytest.mark.parametrize("tokens", [49, 70, 128])
def test_logprobs_of_a_sample_do_not_depend_on_its_pack(name, tokens):
    from miles_b200.models import ParamStore, build_model, get_config

    cfg = get_config(name)
    model = build_model(cfg, ParamStore(cfg, torch.device(DEV), torch.bfloat16, init_std=0.05, seed=3), "b200")
    g = torch.Generator().manual_seed(tokens)
    lens = [tokens, 200]
    ids = torch.randint(0, cfg.vocab_size, (sum(lens),), generator=g).to(DEV, torch.int32)
    pos = torch.cat([torch.arange(n) for n in lens]).to(DEV, torch.int32)
    rows = torch.arange(tokens - 1, device=DEV)
    cu = torch.tensor([0, tokens, sum(lens)], dtype=torch.int32, device=DEV)
    alone = model.forward_logprobs(ids[:tokens], pos[:tokens], cu[:2], rows, ids[1:tokens], 1.0)
    packed = model.forward_logprobs(ids, pos, cu, torch.cat([rows, torch.arange(tokens, tokens + 199, device=DEV)]),
                                    torch.cat([ids[1:tokens], ids[tokens + 1:]]), 1.0)
    model.check_status()
    assert all(torch.equal(a, b[:tokens - 1]) for a, b in zip(alone, packed))


def test_a_launch_that_the_runtime_refuses_is_raised(ext):
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    x, none = torch.zeros(2, 64, dtype=torch.bfloat16, device=DEV), torch.zeros(0, 64, dtype=torch.bfloat16, device=DEV)
    with pytest.raises(RuntimeError, match="small_gemv"):  # no rows of weights: an empty grid
        ext.small_gemv(x, None, 0.0, none, None, torch.zeros(2, 0, dtype=torch.bfloat16, device=DEV), st)
    w = torch.zeros(4, 128, 64, dtype=torch.bfloat16, device=DEV)
    i32 = torch.zeros(64, dtype=torch.int32, device=DEV)
    with pytest.raises(RuntimeError, match="moe_small_up"):  # no expert: the same
        ext.moe_small_up(x, x[0].clone(), 1e-6, w, i32, i32, i32, 0, 2, torch.zeros(4, 128, dtype=torch.bfloat16, device=DEV), st)
    with pytest.raises(RuntimeError, match="moe_small_down"):
        ext.moe_small_down(torch.zeros(4, 128, dtype=torch.bfloat16, device=DEV), w, i32, i32, i32, 0, torch.zeros(4, 128, dtype=torch.bfloat16, device=DEV), st)
    assert torch.ones(3, device=DEV).sum().item() == 3  # and is not found again by the next call
