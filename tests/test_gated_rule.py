"""When the experts' gate-up product takes SwiGLU into its epilogue: by the pairs that are routed, not by the room their plan has."""
import pytest
import torch

from miles_b200.models.b200_impl import MoeCtx


def _plan(experts, max_rows, align=1, pairs=0):
    return MoeCtx(None, None, None, torch.zeros(experts + 1, dtype=torch.int32), None, None, None, None, max_rows, align, pairs)


@pytest.mark.parametrize("experts, tokens, top_k, want", [(128, 16, 8, False), (128, 767, 8, False), (128, 768, 8, True), (8, 191, 2, False), (8, 192, 2, True)])
def test_rows_per_expert(experts, tokens, top_k, want):
    n = tokens * top_k
    assert _plan(experts, n, pairs=n).gated() == want
    # an exchange between ranks has room for all that could come: it does not count
    assert _plan(experts, 16 * n, pairs=n).gated() == want
    # padded to whole tiles: always (the activation kernel would go through the padding)
    assert _plan(experts, n + experts * 63, 64, n).gated()
    assert _plan(experts, n).gated() == want
