"""The persistent two-head attention kernel against the one that takes a (tile, head) pair per block: the same values bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# one row, one block and a row, ragged tails, more pairs than a round of SMs, groups of two to eight heads; cached prefixes
@pytest.mark.parametrize("lens, prefix, Hq, Hk", [([1] * 160, None, 2, 1), ([129, 1, 300, 128, 64], None, 32, 4), ([1300], None, 16, 8),
                                                  ([2048, 777], None, 32, 4), ([40, 64, 1, 17], [0, 448, 1024, 130], 48, 8),
                                                  ([37] * 31, [512 + 64 * i for i in range(31)], 32, 8)])
def test_pairs_match_single_heads(lens, prefix, Hq, Hk):
    from miles_b200.ops import _ext
    from miles_b200.ops.attention import build_tiles

    C = _ext.load(required=True)
    g = torch.Generator(device="cuda").manual_seed(len(lens) + Hq)
    T, Tkv = sum(lens), sum(lens) + sum(prefix or [0])
    q = (torch.randn(T, Hq, 128, device="cuda", generator=g) * 2).bfloat16()  # (a wide score range: maxima grow again and again)
    k, v = (torch.randn(Tkv, Hk, 128, device="cuda", generator=g).bfloat16() for _ in range(2))
    tiles = build_tiles(lens, prefix)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert tiles.shape[0] * Hq > sms
    out, lse = C.flash_attn_fwd(q, k, v, tiles.cuda(), 128 ** -0.5, status)
    per = sms // Hq  # as many tiles as the kernel with a block per head takes
    for some in tiles.split(per):
        o1, l1 = C.flash_attn_fwd(q, k, v, some.cuda(), 128 ** -0.5, status)
        for r0, n, _, _ in some.tolist():
            assert torch.equal(out[r0:r0 + n], o1[r0:r0 + n]) and torch.equal(lse[:, r0:r0 + n], l1[:, r0:r0 + n])
    assert status.item() == 0
