"""Number of splits of the decode attention: its clusters are resident at once, and no sequence is cut finer than a cluster holds."""
import types

import pytest

from miles_b200.models.b200_impl import B200Qwen3


@pytest.mark.parametrize("heads", [1, 2, 4, 8, 32])
def test_clusters_fit(heads):
    model = types.SimpleNamespace(cfg=types.SimpleNamespace(num_kv_heads=heads))
    for rows in range(1, 300):
        s = B200Qwen3._decode_splits(model, rows, None)
        assert 1 <= s <= 16
        assert s == 1 or rows * heads * s <= (296 if s == 2 else 264)
        assert s >= 8 or rows * heads * (s + 1) > 264
