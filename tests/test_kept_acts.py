"""Activations kept between the directions of a training pass: which ones, and that they change nothing."""
import pytest
import torch

from miles_b200.models.b200_impl import plan_kept


@pytest.mark.parametrize("room, want", [(0, (False, 5)), (4, (False, 5)), (9, (False, 4)), (10, (True, 5)), (14, (True, 5)), (15, (True, 4)),
                                        (30, (True, 3)), (34, (True, 3)), (35, (True, 2)), (-7, (False, 5))])
def test_plan_kept(room, want):
    # ten bytes of logits, layers 2, 3, 4 of 5, 15 and 5 bytes: the last layers first, none behind one that does not fit
    assert plan_kept(room, 10, [5, 15, 5], 2) == want


def test_plan_kept_without_head():
    assert plan_kept(100, 0, [5, 5], 0) == (False, 0)
    assert plan_kept(100, 0, [], 3) == (False, 3)


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["qwen3-smoke", "qwen3-smoke-moe", "glm4moe-smoke", "glm4-smoke", "qwen2moe-smoke"])
def test_kept_activations_change_nothing(name):
    from miles_b200.models import ParamStore, build_model, get_config
    from test_b200_model import _batch

    dev = torch.device("cuda")
    cfg = get_config(name)
    store = ParamStore(cfg, dev, torch.bfloat16, init_std=0.05, seed=7)
    store.allocate_grads(torch.float32)
    model = build_model(cfg, store, "b200")
    tokens, pos, cu, rows, tg = _batch(cfg, [200, 333, 75], dev)
    coef = torch.randn(rows.numel(), device=dev)
    T = tokens.numel()
    head = 6 * rows.numel() * cfg.vocab_size
    layers = [model._layer_act_bytes(i, T) for i in range(cfg.num_layers)]
    out = []
    for room in (0, head + layers[-1], 1 << 40):
        model.act_room = room
        assert model._plan_acts(T, rows.numel(), model.lm_chunk) == ((False, cfg.num_layers), (True, cfg.num_layers - 1), (True, 0))[len(out)]
        store.zero_grads()
        record = []
        model.forward_logprobs(tokens, pos, cu, rows, tg, 1.0, record=record)
        replay = torch.stack(record, 1) if record else None
        loss, _, lp, ent = model.forward_backward(tokens, pos, cu, rows, tg, 1.0, lambda lp, ent: ((lp * coef).sum() / 50 + 0.01 * ent.sum(), {}),
                                                  replay=replay)
        model.check_status()
        out.append((loss, lp, ent, {n: g.clone() for n, g in store.grads.items()}))
    for loss, lp, ent, grads in out[1:]:
        assert torch.equal(loss, out[0][0]) and torch.equal(lp, out[0][1]) and torch.equal(ent, out[0][2])
        for n, g in grads.items():  # (dQ and the head norms are summed with atomics, whose order differs from run to run)
            want = out[0][3][n]
            assert (g - want).norm() <= 1e-2 * want.norm() + 1e-12, n
