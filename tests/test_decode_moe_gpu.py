"""Decode experts of at most eight rows with SwiGLU, the combination and the routing folded in, against plain fp32 and the unfused kernels."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _plan(C, ids, w, E):
    """The plan that router_decode would write, from ids and weights [T, K]."""
    T, K = ids.shape
    plan = torch.full((C.moe_decode_plan_size(E),), -7, dtype=torch.int32)
    used = sorted(set(ids.flatten().tolist()))
    plan[0] = len(used)
    for i, e in enumerate(used):
        rec = plan[4 + 20 * i:24 + 20 * i]
        rec[0], rec[4:12] = e, -1
        for t, k in (ids == e).nonzero().tolist():
            rec[4 + t], rec[12 + t] = t * K + k, w[t, k].view(torch.int32)
    return plan.cuda()


def _same_plan(a, b, T):
    n = int(a[0])
    ra, rb = (p[4:4 + 20 * n].view(n, 20) for p in (a, b))
    live = ra[:, 4:12] >= 0
    return int(b[0]) == n and torch.equal(ra[:, 0], rb[:, 0]) and torch.equal(ra[:, 4:12], rb[:, 4:12]) and torch.equal(ra[:, 12:][live], rb[:, 12:][live])


# every number of k slices in a stage (1 to 4 and parts of a second one), down widths that leave warps without one, one and two CTAs
# per tile, few and all experts, one expert per token, more choices than lanes in a half-warp
@pytest.mark.parametrize("T, E, K, H, I", [(1, 128, 8, 2048, 768), (8, 128, 8, 2048, 768), (3, 16, 2, 512, 96), (8, 16, 16, 1024, 256),
                                           (5, 32, 4, 4096, 1024), (2, 16, 2, 2560, 2112), (7, 48, 1, 256, 32), (4, 128, 8, 1792, 1408),
                                           (8, 112, 32, 768, 512), (6, 32, 4, 1280, 800), (8, 16, 4, 2816, 2048), (8, 48, 32, 1024, 2112)])
def test_fused_decode_experts(T, E, K, H, I):
    from miles_b200.ops import _ext

    C = _ext.load(required=True)
    assert C.moe_decode_fits(E, K, H, I)
    g = torch.Generator(device=DEV).manual_seed(T + E + I)
    rnd = lambda *s, std=1.0: (torch.randn(*s, device=DEV, generator=g) * std).bfloat16()  # noqa: E731
    x, nw, Wr, W1, W2 = rnd(T, H), 1 + rnd(H, std=0.1), rnd(E, H, std=0.06), rnd(E, 2 * I, H, std=0.03), rnd(E, H, I, std=0.03)
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    i32 = dict(dtype=torch.int32, device=DEV)
    ids, w, plan = torch.empty(T, K, **i32), torch.empty(T, K, device=DEV), torch.empty(C.moe_decode_plan_size(E), **i32)
    C.router_decode(x, nw, 1e-6, Wr, True, ids, w, plan)
    # the unfused kernels: the same choices and weights, bit for bit
    lg = torch.empty(T, E, device=DEV)
    ids2, w2 = torch.empty(T, K, **i32), torch.empty(T, K, device=DEV)
    active, pc, pl = torch.empty(1 + E, **i32), torch.empty(E, **i32), torch.empty(8 * E, **i32)
    C.small_gemv(x, nw, 1e-6, Wr, None, lg, st)
    C.router_small(lg, K, True, ids2, w2, active, pc, pl)
    assert torch.equal(ids, ids2) and torch.equal(w, w2)
    assert _same_plan(plan, _plan(C, ids.cpu(), w.cpu(), E), T)

    gu, act = torch.empty(T * K, 2 * I, device=DEV).bfloat16(), torch.empty(T * K, I, device=DEV).bfloat16()
    C.moe_small_up(x, nw, 1e-6, W1, active, pc, pl, min(E, T * K), K, gu, st)
    C.moe_decode_up(x, nw, 1e-6, W1, plan, act, st)
    # against 64 bits no further off than the two products, each rounded, and the activation of the rounded ones
    xn = x.double() * torch.rsqrt(x.double().square().mean(-1, keepdim=True) + 1e-6) * nw.double()
    flat = ids.flatten().long()
    p = torch.einsum("ph,pnh->pn", xn.repeat_interleave(K, 0), W1[flat].double())
    want = torch.nn.functional.silu(p[:, :I]) * p[:, I:]
    err, err2 = ((o.double() - want).norm() / want.norm() for o in (act, C.swiglu_fwd(gu)))
    assert err <= 1.02 * err2 and err < 6e-3
    y = torch.empty(T, H, device=DEV).bfloat16()
    C.moe_decode_down(act, W2, plan, x, y, st)
    yp = torch.einsum("pi,phi->ph", act.double(), W2[ids.flatten().long()].double()).view(T, K, H)
    want = x.double() + (w.double()[..., None] * yp).sum(1)
    # fp32 sums of I * K terms (2^-24 of their size each), every pair rounded to bf16 and the sum once more: half a unit in the last of eight
    # bits is at most 2^-8 of a value (and 2^-8 of the pairs' share of the sum)
    pairs = (w.double()[..., None] * yp).abs().sum(1)
    assert ((y.double() - want).abs() <= 2 ** -8 * (want.abs() + 1.01 * pairs) + 1e-4 * want.abs().mean()).all()
    # the unfused kernels, bit for bit
    yp2 = torch.empty(T * K, H, device=DEV).bfloat16()
    C.moe_small_down(gu, W2, active, pc, pl, min(E, T * K), yp2, st)
    y2 = C.moe_combine(yp2, torch.arange(T * K, **i32), w, T, K, x)
    assert torch.equal(act, C.swiglu_fwd(gu)) and torch.equal(y, y2)
    # and every row what it is alone: neither the others' experts nor its place among the rows shows
    for t in range(T):
        one, i1, w1 = torch.empty(1, H, device=DEV).bfloat16(), torch.empty(1, K, **i32), torch.empty(1, K, device=DEV)
        a1 = torch.empty(K, I, device=DEV).bfloat16()
        C.router_decode(x[t:t + 1], nw, 1e-6, Wr, True, i1, w1, plan)
        C.moe_decode_up(x[t:t + 1], nw, 1e-6, W1, plan, a1, st)
        C.moe_decode_down(a1, W2, plan, x[t:t + 1], one, st)
        assert torch.equal(i1[0], ids[t]) and torch.equal(w1[0], w[t]) and torch.equal(one[0], y[t])
    assert st.item() == 0


def test_router_ties_and_values_that_cannot_be_chosen():
    from miles_b200.ops import _ext

    C = _ext.load(required=True)
    T, E, K, H = 5, 32, 4, 256
    Wr = torch.zeros(E, H, device=DEV).bfloat16()
    Wr[torch.arange(E), torch.arange(E)] = 1.0  # logit e of a token is its value e, normalised
    x = torch.zeros(T, H, device=DEV).bfloat16()
    x[0, :E] = 1.0                                            # all equal: the lowest ids
    x[1, [3, 9, 17, 30]] = torch.tensor([1.0, 2.0, 2.0, -4.0], device=DEV).bfloat16()
    x[2, :E] = -torch.arange(1, E + 1, device=DEV).bfloat16()
    x[3, 5], x[3, 0] = -0.0, 1.0                              # zeros of both signs tie
    x[4, 31] = 1.0
    i32 = dict(dtype=torch.int32, device=DEV)
    out = []
    for new in (True, False):
        ids, w, plan = torch.empty(T, K, **i32), torch.empty(T, K, device=DEV), torch.empty(C.moe_decode_plan_size(E), **i32)
        if new:
            C.router_decode(x, torch.ones(H, device=DEV).bfloat16(), 1e-6, Wr, False, ids, w, plan)
        else:
            lg = torch.empty(T, E, device=DEV)
            C.small_gemv(x, torch.ones(H, device=DEV).bfloat16(), 1e-6, Wr, None, lg, None)
            C.router_small(lg, K, False, ids, w, torch.empty(1 + E, **i32), torch.empty(E, **i32), torch.empty(8 * E, **i32))
        out.append((ids, w))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    assert out[0][0][0].tolist() == [0, 1, 2, 3] and out[0][0][1].tolist()[:3] == [9, 17, 3]


def test_infinite_weights_stay_with_their_tokens():
    from miles_b200.ops import _ext

    C = _ext.load(required=True)
    T, E, K, H, I = 3, 16, 1, 256, 256
    act = torch.ones(T * K, I, device=DEV).bfloat16()
    W2 = torch.ones(E, H, I, device=DEV).bfloat16()
    W2[5] = float("inf")
    ids = torch.tensor([[2], [5], [2]])
    plan = _plan(C, ids, torch.full((T, K), 0.5), E)
    x = torch.zeros(T, H, device=DEV).bfloat16()
    y = torch.empty_like(x)
    C.moe_decode_down(act, W2, plan, x, y, torch.zeros(1, dtype=torch.int32, device=DEV))
    for t in range(T):
        assert (y[t] == (float("inf") if t == 1 else I / 2)).all()


def test_what_does_not_fit_is_refused():
    from miles_b200.ops import _ext

    C = _ext.load(required=True)
    for E, K, H, I in [(8, 2, 2048, 768), (144, 8, 2048, 768), (128, 8, 2080, 768), (128, 8, 8192, 768), (128, 8, 2048, 2144), (128, 8, 2048, 784)]:
        assert not C.moe_decode_fits(E, K, H, I)
