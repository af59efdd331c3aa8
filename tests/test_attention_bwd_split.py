"""The rule that deals a key block's heads out to CTAs in the attention backward: what it counts and what it may return."""
import pytest
import torch

from miles_b200.ops.attention import TileCache


@pytest.mark.parametrize("lens, Hq, Hk, split", [
    ([1], 32, 4, 4), ([389, 388], 32, 4, 4), ([2048], 32, 4, 4), ([4096], 32, 4, 2), ([200] * 9, 32, 4, 2), ([200] * 24, 32, 4, 1),
    ([1024] * 8, 32, 4, 1), ([2731] * 6, 32, 4, 1), ([777], 8, 8, 1), ([777], 24, 8, 1), ([777], 16, 8, 2)])
def test_split(lens, Hq, Hk, split):
    cu = torch.tensor([0] + lens).cumsum(0).int()
    cache = TileCache()
    assert cache.get_bwd_split(cu, Hq, Hk) == split
    blocks = [(c, n) for n in lens for c in range(0, n, 128)]
    tiles = [-(-(n - c) // 64) for c, n in blocks]
    assert cache._bwd_work == (len(blocks), max(tiles), sum(tiles)) and cache.get_bwd(cu).shape[0] == len(blocks)
    assert cache.get_bwd_split(torch.zeros(1, dtype=torch.int32), Hq, Hk) in (1, 2, 4)  # (a pack without sequences)


def test_operands_are_checked_before_the_first_launch():
    """From the source: maps, which check the alignment, come before the memset and the kernel that reads 16 bytes at a time."""
    from pathlib import Path

    import miles_b200

    text = (Path(miles_b200.__file__).resolve().parent / "csrc" / "attention_bwd.cu").read_text()
    body = text[text.index("int flash_attn_bwd("):]
    assert body.rindex("make_map(") < body.index("cudaMemsetAsync(") < body.index("<<<")
