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


@pytest.mark.parametrize("name, tokens, free_gb", [("qwen3-8B", 2048, 150), ("qwen3-8B", 16384, 60), ("qwen3-8B", 98304, 150), ("qwen3-8B", 131072, 165),
                                                   ("qwen3-4B", 98304, 100), ("qwen3-30B-A3B", 16384, 30), ("qwen3-30B-A3B", 65536, 100)])
def test_what_is_kept_leaves_room_for_the_pass(monkeypatch, name, tokens, free_gb):
    """Activations are kept only beyond what the pass needs anyway: the inputs of all layers, a layer on its way back, a chunk of the head."""
    import types

    from miles_b200.models import get_config
    from miles_b200.models.b200_impl import B200Qwen3

    cfg = get_config(name)
    model = B200Qwen3.__new__(B200Qwen3)
    head = types.SimpleNamespace(shape=(cfg.vocab_size, cfg.hidden_size))
    model.__dict__.update(cfg=cfg, store=types.SimpleNamespace(layer_range=(0, cfg.num_layers), lm_head=lambda: head), ep=None, tp=None, cp_ctx=None,
                          act_room=None, dev="cuda", recompute_layers=0, recompute_logits=False)
    free, total, cached = int(free_gb * 1e9), int(192e9), int(5e9)
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda dev: (free - cached, total))
    monkeypatch.setattr(torch.cuda, "memory_reserved", lambda dev: total - free + cached)
    monkeypatch.setattr(torch.cuda, "memory_allocated", lambda dev: total - free)
    head_rows, chunk = tokens * 3 // 4, 2048
    keep_head, keep_from = model._plan_acts(tokens, head_rows, chunk)
    layer = model._layer_act_bytes(0, tokens)
    # written out again: inputs, hidden rows and gradients around them; recomputed activations and their gradients, or logits and dlogits
    need = 2 * tokens * cfg.hidden_size * (cfg.num_layers + 1) + 4 * head_rows * cfg.hidden_size
    work = max(2 * layer + 4 * tokens * cfg.num_q_heads * cfg.head_dim, 8 * chunk * cfg.vocab_size)
    kept = (4 * head_rows * cfg.vocab_size if keep_head else 0) + (cfg.num_layers - keep_from) * layer
    assert kept == 0 or kept + need + work + total // 28 <= free
    assert kept <= max(0, free - total // 7)
    if tokens <= 16384 and name == "qwen3-8B":  # (and room that is there is used)
        assert kept > 0
        assert keep_from == 0 or kept + layer > free - total // 7


# layers 3 .. 9 of 24, logits and activations that all fit: what the command line asks to recompute is recomputed
@pytest.mark.parametrize("flags, want", [([], (True, 3)), (["--recompute-granularity", "full"], (True, 10)),
                                         (["--recompute-granularity", "full", "--recompute-loss-function"], (False, 10)),
                                         (["--recompute-loss-function"], (False, 3)), (["--recompute-granularity", "selective"], (True, 3)),
                                         (["--recompute-granularity", "none"], (True, 3)),
                                         (["--recompute-granularity", "full", "--recompute-method", "uniform", "--recompute-num-layers", "2"], (True, 10)),
                                         (["--recompute-granularity", "full", "--recompute-method", "block", "--recompute-num-layers", "4"], (True, 7)),
                                         (["--recompute-granularity", "full", "--recompute-method", "block", "--recompute-num-layers", "40"], (True, 10))])
def test_recomputation_that_is_asked_for(flags, want):
    import types

    from miles_b200.models import get_config
    from miles_b200.models.b200_impl import B200Qwen3, recompute_policy
    from miles_b200.utils.arguments import parse_args

    args = parse_args(["--num-rollout", "1", "--rollout-batch-size", "2", "--n-samples-per-prompt", "2", "--model-preset", "qwen3-tiny"] + flags)
    cfg = get_config("qwen3-0.6B")
    model = B200Qwen3.__new__(B200Qwen3)
    head = types.SimpleNamespace(shape=(cfg.vocab_size, cfg.hidden_size))
    model.__dict__.update(cfg=cfg, store=types.SimpleNamespace(layer_range=(3, 10), lm_head=lambda: head), ep=None, tp=None, cp_ctx=None,
                          act_room=1 << 50, dev="cuda")
    model.recompute_layers, model.recompute_logits = recompute_policy(args)
    assert model._plan_acts(1000, 500, 2048) == want


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


@pytest.mark.gpu
@pytest.mark.parametrize("name, vocab", [("qwen3-smoke", 4096), ("qwen3-smoke", 32000), ("qwen3-smoke-moe", 32000)])
def test_head_in_chunks_does_not_depend_on_what_is_kept(name, vocab):
    """Several chunks, a short last one (of few rows, which the engine's products would split), logits by either way: scores, and all
    gradients that no atomic sum touches, are the same bit for bit whatever there was room for."""
    from miles_b200.models import ParamStore, build_model, get_config
    from test_b200_model import _batch

    dev = torch.device("cuda")
    cfg = get_config(name)
    cfg.vocab_size, cfg.tie_embeddings = vocab, False  # (an embedding's gradient is an atomic sum)
    store = ParamStore(cfg, dev, torch.bfloat16, init_std=0.05, seed=7)
    store.allocate_grads(torch.float32)
    model = build_model(cfg, store, "b200")
    tokens, pos, cu, rows, tg = _batch(cfg, [200, 333, 75], dev)
    rows, tg = rows[:64 * 6 + (9 if vocab == 32000 else 40)], tg[:64 * 6 + (9 if vocab == 32000 else 40)]
    coef = torch.randn(rows.numel(), device=dev)
    model.lm_chunk = 64
    record = []
    want = model.forward_logprobs(tokens, pos, cu, rows, tg, 1.0, record=record)
    replay = torch.stack(record, 1) if record else None
    last = f"layers.{cfg.num_layers - 1}."
    exact = ["lm_head.weight", "final_norm.weight"] + [n for n in store.grads if n.startswith(last) and ("mlp." in n or "moe.w" in n)]
    assert len(exact) >= 4
    out = []
    for room in (0, 4 * rows.numel() * vocab, 1 << 40):
        model.act_room = room
        assert model._plan_acts(tokens.numel(), rows.numel(), 64)[0] == (room > 0)
        store.zero_grads()
        loss, _, lp, ent = model.forward_backward(tokens, pos, cu, rows, tg, 1.0, lambda lp, ent: ((lp * coef).sum() / 50 + 0.01 * ent.sum(), {}),
                                                  replay=replay)
        model.check_status()
        assert torch.equal(lp, want[0]) and torch.equal(ent, want[1])
        out.append({n: store.grads[n].clone() for n in exact})
    for grads in out[1:]:
        for n, g in grads.items():
            assert g.abs().max() > 0 and torch.equal(g, out[0][n]), n


@pytest.mark.gpu
def test_scores_keep_to_the_chunks_bytes():
    """Scoring and differentiating hold what ``lm_chunk`` rows of fp32 logits take, and as much again for the logits' gradients."""
    from miles_b200.models import ParamStore, build_model, get_config

    dev = torch.device("cuda")
    cfg = get_config("qwen3-smoke")
    cfg.vocab_size, cfg.num_layers = 64000, 1
    store = ParamStore(cfg, dev, torch.bfloat16, init_std=0.05, seed=7)
    store.allocate_grads(torch.float32)
    model = build_model(cfg, store, "b200")
    n, model.lm_chunk, model.act_room = 8192, 128, 0
    h = torch.randn(n, cfg.hidden_size, device=dev).bfloat16()
    tokens, pos = torch.randint(0, cfg.vocab_size, (n,), device=dev).int(), torch.arange(n, device=dev).int()
    chunk = 4 * model.lm_chunk * cfg.vocab_size

    def peak(f):
        f()
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        f()
        return torch.cuda.max_memory_allocated() - before

    rows = 64 * n * 4 + 4 * n * 2 * cfg.hidden_size  # statistics, and the hidden rows with their gradients
    assert peak(lambda: model.logprobs_entropy(h, tokens, 1.0)) <= chunk + rows
    one = torch.tensor([0, 1], dtype=torch.int32, device=dev)  # (one token, whose row is scored again and again: the head is nearly all there is)
    assert peak(lambda: model.forward_backward(tokens[:1], pos[:1], one, torch.zeros(n, dtype=torch.int64, device=dev), tokens, 1.0,
                                               lambda lp, ent: (lp.sum(), {}))) <= 2 * chunk + rows + (1 << 20)


@pytest.mark.gpu
@pytest.mark.parametrize("where", ["layer", "head"])
def test_a_pass_that_runs_out_of_memory_keeps_nothing(monkeypatch, where):
    from miles_b200.models import ParamStore, build_model, get_config
    from test_b200_model import _batch

    dev = torch.device("cuda")
    cfg = get_config("qwen3-smoke")
    store = ParamStore(cfg, dev, torch.bfloat16, init_std=0.05, seed=7)
    store.allocate_grads(torch.float32)
    model = build_model(cfg, store, "b200")
    tokens, pos, cu, rows, tg = _batch(cfg, [200, 75], dev)
    run = lambda: model.forward_backward(tokens, pos, cu, rows, tg, 1.0, lambda lp, ent: (lp.sum(), {}))  # noqa: E731
    model.act_room = 0
    store.zero_grads()
    want = run()
    exact = ["final_norm.weight", "lm_head.weight", f"layers.{cfg.num_layers - 1}.mlp.down.weight"]
    grads = {n: store.grads[n].clone() for n in exact}
    model.act_room, calls = 1 << 40, []
    layer_acts, scores = model._layer_acts, model.logprobs_entropy

    def short_layer(i, *a, output=False, **kw):
        calls.append((i, output))
        if output and i == 1:
            raise torch.OutOfMemoryError("CUDA out of memory. Tried to allocate 1 GiB")
        return layer_acts(i, *a, output=output, **kw)

    def short_head(*a, keep_logits=None, **kw):
        calls.append(keep_logits is not None)
        if keep_logits is not None:
            keep_logits.append(None)
            raise RuntimeError("CUDA out of memory. Tried to allocate 1 GiB")
        return scores(*a, **kw)

    monkeypatch.setattr(model, *(("_layer_acts", short_layer) if where == "layer" else ("logprobs_entropy", short_head)))
    store.zero_grads()
    got = run()
    assert calls == ([(0, True), (1, True), (1, False), (0, False)] if where == "layer" else [True, False])
    assert torch.equal(got[0], want[0]) and torch.equal(got[2], want[2])
    assert all(torch.equal(store.grads[n], g) for n, g in grads.items())
