"""Packed keys / values behind a cached prefix: against indexing, for rows of odd numbers of vectors, strided new rows,
sequences without a prefix, and slots outside the cache, which are reported and read as zeros."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("heads", [1, 4, 8, 9])
@pytest.mark.parametrize("prefix,new", [([5], [1]), ([0, 64, 130], [3, 1, 70]), ([1500] * 7, [9] * 7)])
def test_gather_equals_indexing(heads, prefix, new):
    from miles_b200.models.torch_impl import PrefixInfo
    from miles_b200.ops import _ext

    ext = _ext.load(required=True)
    g = torch.Generator().manual_seed(heads + len(prefix))
    slots = torch.randperm(sum(prefix) + 40, generator=g)[:sum(prefix)]
    info = PrefixInfo.build(prefix, new, slots, DEV)
    kc, vc = (torch.randn(sum(prefix) + 40, heads, 128, generator=g).bfloat16().to(DEV) for _ in range(2))
    qkv = torch.randn(sum(new), 3 * heads, 128, generator=g).bfloat16().to(DEV)
    k, v = qkv[:, heads:2 * heads].contiguous(), qkv[:, 2 * heads:]
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    want = info.full_kv(k, v, kc, vc)
    got = ext.gather_prefix_kv(k, v, kc, vc, info.pre_slots, info.pre_dst, info.new_dst, info.total, st)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]) and st.item() == 0
    bad = info.pre_slots.clone()
    bad[0], bad[-1] = kc.shape[0], -1
    torch.full((4 * info.total * heads * 128,), float("nan"), dtype=torch.bfloat16, device=DEV)  # what freed memory may hold
    got = ext.gather_prefix_kv(k, v, kc, vc, bad, info.pre_dst, info.new_dst, info.total, st)
    for t, w in zip(got, want):
        w = w.clone()
        w[info.pre_dst[[0, -1]]] = 0
        assert torch.equal(t, w)
    assert st.item() == 9
