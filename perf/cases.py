"""The work of one GRPO step, case by case: what a user of this package has one GPU do, through its public entry points.

A step generates responses (``Engine.generate``, a decode step of the running rows at a time), brings prompts into the key / value cache
(``Engine.feed``), scores the packed samples (``forward_logprobs``), differentiates them (``forward_backward``) and updates the weights
(``FlatAdam.step``). The models are the layers of the headline benchmark's mixture of experts and of dense models beside it, in bf16, at full
width with their whole vocabularies and as many layers as let three sets of weights stand on one device: every layer is the same work, so
what holds for these holds for the full depth. Sizes are those of the headline benchmark (prompts of 1024 tokens, responses of 2048 in the
mean and 8192 at most, up to 64 running rows, packs of up to 16384 tokens here) and smaller ones down to single short sequences.
"""
from __future__ import annotations

import math
import zlib

import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

MODELS = {
    "qwen3-30B-A3B": dict(hidden=2048, heads=32, kv_heads=4, experts=128, top_k=8, ffn=768, vocab=151936, tied=False),
    "qwen3-4B": dict(hidden=2560, heads=32, kv_heads=8, experts=0, top_k=0, ffn=9728, vocab=151936, tied=True),
    "qwen3-8B": dict(hidden=4096, heads=32, kv_heads=8, experts=0, top_k=0, ffn=12288, vocab=151936, tied=False),
    "qwen3-0.6B": dict(hidden=1024, heads=16, kv_heads=8, experts=0, top_k=0, ffn=3072, vocab=151936, tied=True),
}
HEAD_DIM, THETA, EPS = 128, 1e6, 1e-6
ADAM = dict(lr=1e-6, beta1=0.9, beta2=0.98, eps=1e-8, weight_decay=0.1, clip_grad=1.0)
MOE = "qwen3-30B-A3B"


def listed():
    return [
        # the tail of a rollout: the last long response runs alone (latency of the launches)
        dict(name="decode-moe-1", kind="decode", model=MOE, layers=16, rows=1, context=3000, new=24),
        # a few long responses left; rows whose contexts differ
        dict(name="decode-moe-4", kind="decode", model=MOE, layers=16, rows=4, context=7900, new=24),
        # the middle of a rollout
        dict(name="decode-moe-16", kind="decode", model=MOE, layers=16, rows=16, context=1800, new=24),
        # its beginning: every row of the batch of 8 prompts x 8 samples runs
        dict(name="decode-moe-64", kind="decode", model=MOE, layers=16, rows=64, context=1500, new=24),
        # a dense model's rollout with an odd number of rows
        dict(name="decode-dense-23", kind="decode", model="qwen3-4B", layers=12, rows=23, context=2300, new=24),
        # the prompts of a step enter the cache
        dict(name="prefill-moe-8", kind="prefill", model=MOE, layers=8, sequences=8, tokens=8192),
        # one short question to a dense model (the smallest call)
        dict(name="prefill-dense-1", kind="prefill", model="qwen3-4B", layers=12, sequences=1, tokens=93),
        # scoring a pack of samples under the old policy
        dict(name="logprobs-moe", kind="logprobs", model=MOE, layers=8, sequences=6, tokens=16384),
        # forward and backward of a pack with the rollout's routing replayed
        dict(name="train-moe", kind="train", model=MOE, layers=4, sequences=6, tokens=16384),
        # the last, nearly empty pack of a step
        dict(name="train-moe-short", kind="train", model=MOE, layers=4, sequences=2, tokens=777),
        # a long response of a dense model
        dict(name="train-dense-long", kind="train", model="qwen3-8B", layers=3, sequences=1, tokens=9216),
        # the weight update: replicated and expert parameters
        dict(name="adam-moe", kind="adam", model=MOE, layers=1, state="bf16"),
    ]


def draw(rng):
    """One more case of the same ranges; sizes are drawn over their logarithm."""
    size = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    kind = rng.choice(["decode", "decode", "decode", "prefill", "logprobs", "train", "train", "adam"])
    model = rng.choice([MOE, MOE, "qwen3-4B"])
    if kind == "decode":
        rows = size(1, 64)
        return dict(kind=kind, model=model, layers=16 if model == MOE else 12, rows=rows, context=size(200, min(8192, 96000 // rows)), new=rng.randint(16, 24))
    if kind == "adam":
        return dict(kind=kind, model=rng.choice(["qwen3-0.6B", "qwen3-4B", MOE]), layers=1 if model == MOE else rng.randint(1, 8), state=rng.choice(["bf16", "fp32"]))
    tokens = size(64, 8192 if kind == "prefill" else 16384)
    sequences = rng.randint(1, max(1, min(8, tokens // 32)))
    model = rng.choice([MOE, MOE, "qwen3-4B", "qwen3-8B"]) if kind == "train" else model
    layers = {"prefill": 8, "logprobs": 8, "train": 4}[kind] if model == MOE else {"prefill": 12, "logprobs": 6, "train": 3}[kind]
    if model != MOE and kind == "train":
        tokens = min(tokens, 12288)
    return dict(kind=kind, model=model, layers=layers, sequences=sequences, tokens=tokens)


# ---------------------------------------------------------------------------------------------- inputs
def _gen(seed, key, device="cuda"):
    return torch.Generator(device=device).manual_seed((seed * 1000003 + zlib.crc32(key.encode())) & 0x7FFFFFFFFFFF)


def _shapes(case):
    m = MODELS[case["model"]]
    H, q, kv = m["hidden"], m["heads"] * HEAD_DIM, m["kv_heads"] * HEAD_DIM
    out = {"embed.weight": (m["vocab"], H)}
    for i in range(case["layers"]):
        p = f"layers.{i}."
        out.update({p + "ln1.weight": (H,), p + "attn.qkv.weight": (q + 2 * kv, H), p + "attn.q_norm.weight": (HEAD_DIM,), p + "attn.k_norm.weight": (HEAD_DIM,),
                    p + "attn.o.weight": (H, q), p + "ln2.weight": (H,)})
        if m["experts"]:
            out.update({p + "moe.router.weight": (m["experts"], H), p + "moe.w1": (m["experts"], 2 * m["ffn"], H), p + "moe.w2": (m["experts"], H, m["ffn"])})
        else:
            out.update({p + "mlp.gate_up.weight": (2 * m["ffn"], H), p + "mlp.down.weight": (H, m["ffn"])})
    out["final_norm.weight"] = (H,)
    if not m["tied"]:
        out["lm_head.weight"] = (m["vocab"], H)
    return out


def _weight(case, seed, name):
    """One weight in bf16. Norm weights lie around one, matrices have a standard deviation of 0.02 and the projections back into the residual
    stream 0.02 / sqrt(2 layers), as training programs begin; routers 0.06, so that a token's experts have clearly different weights, as
    in a trained model. For generation the head expects the token after the one at hand (the same token where head and embedding are tied): a
    trained model's next token is likewise mostly certain, and so a sampled response does not depend on the order of a sum."""
    shape = _shapes(case)[name]
    linked, tied = case["kind"] == "decode", MODELS[case["model"]]["tied"]
    if name == "lm_head.weight" and linked:
        return (_weight(case, seed, "embed.weight").roll(1, 0) * (0.04 / 0.4)).to(torch.bfloat16)
    std = 0.1 if len(shape) == 1 else 0.06 if name.endswith("router.weight") else 0.02
    if name.endswith(("attn.o.weight", "mlp.down.weight", "moe.w2")):
        std *= (2 * case["layers"]) ** -0.5
    if name == "embed.weight" and linked:
        std = 0.3 if tied else 0.4
    w = torch.randn(shape, generator=_gen(seed, name), device="cuda", dtype=torch.bfloat16).mul_(std)
    return w.add_(1.0) if len(shape) == 1 else w


def _model(case, seed):
    from miles_b200.models import ParamStore, build_model, get_config

    cfg = get_config(case["model"])
    cfg.num_layers = case["layers"]
    store = ParamStore(cfg, "cuda", torch.bfloat16, init=False)
    for name, p in store.params.items():
        p.copy_(_weight(case, seed, name))
    return cfg, store, build_model(cfg, store, "b200")


def _lengths(case):
    """Ragged lengths that add up to the pack's tokens (the same for every seed: results of one case have one shape)."""
    n, total = case["sequences"], case["tokens"]
    w = torch.rand(n, generator=_gen(n, f"lengths {total}", "cpu"), dtype=torch.float64) + 0.35
    lens = [max(2, int(x)) for x in (w / w.sum() * total).tolist()]
    lens[0] += total - sum(lens)
    return lens


def _tokens(case, seed, n, key="tokens"):
    return torch.randint(0, MODELS[case["model"]]["vocab"], (n,), generator=_gen(seed, key, "cpu"))


def _prompts(case, seed):
    """Contexts of the running rows: within a quarter of the case's, at least two tokens, pairwise different."""
    r = torch.rand(case["rows"], generator=_gen(case["rows"], "contexts", "cpu"))
    lens = [max(2, int(case["context"] * (1.0 - 0.25 * float(x)))) for x in r]
    return [_tokens(case, seed, n, f"prompt {i}").tolist() for i, n in enumerate(lens)]


def _pack(case, seed):
    """A pack of samples as the trainer stages it: the first quarter of each is prompt, the rest response. Routing ids are those a rollout
    would have recorded: every token's experts are distinct, and unevenly popular."""
    m = MODELS[case["model"]]
    lens = _lengths(case)
    T = sum(lens)
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    rows = torch.cat([torch.arange(a + max(1, n // 4) - 1, a + n - 1) for a, n in zip(cu, lens)])
    tokens = _tokens(case, seed, T)
    pack = dict(lens=lens, tokens=tokens.to("cuda", torch.int32), positions=torch.cat([torch.arange(n) for n in lens]).to("cuda", torch.int32),
                cu=torch.tensor(cu, dtype=torch.int32, device="cuda"), rows=rows.cuda(), targets=tokens[rows + 1].to("cuda", torch.int32),
                advantages=torch.randn(rows.numel(), generator=_gen(seed, "advantages"), device="cuda"), replay=None)
    if m["experts"]:
        lean = 0.5 * torch.randn(case["layers"], m["experts"], generator=_gen(seed, "popularity"), device="cuda")
        noise = torch.rand(T, case["layers"], m["experts"], generator=_gen(seed, "routing"), device="cuda").clamp_(1e-6, 1 - 1e-6)
        pack["replay"] = (lean - torch.log(-torch.log(noise))).topk(m["top_k"], -1).indices.to(torch.int32)
    return pack


def prepare(case, seed):
    kind, state = case["kind"], {"case": case}
    if kind == "adam":
        from miles_b200.trainer.optimizer import FlatAdam, OptimConfig

        _, store, _ = _model(case, seed)
        store.allocate_grads(torch.float32, torch.bfloat16)
        state.update(store=store, opt=FlatAdam(store, OptimConfig(state_dtype={"bf16": torch.bfloat16, "fp32": torch.float32}[case["state"]], **ADAM)))
        for name, g in store.grads.items():
            g.copy_(_gradient(case, seed, name, g.dtype))
        return state
    cfg, store, model = _model(case, seed)
    state.update(store=store, model=model)
    if kind in ("logprobs", "train"):
        state["pack"] = _pack(case, seed)
        if kind == "train":
            store.allocate_grads(torch.float32, torch.bfloat16)
        return state
    from miles_b200.engine import Engine, SamplingParams

    if kind == "prefill":
        lens = _lengths(case)
        state["prompts"] = [_tokens(case, seed, n, f"prompt {i}").tolist() for i, n in enumerate(lens)]
        state["engine"] = Engine(model, max_running=case["sequences"], num_pages=sum(n // 64 + 2 for n in lens) + 1, page_size=64, max_seq_len=max(lens) + 64)
        return state
    prompts = _prompts(case, seed)
    pages = 2 * sum((len(p) + case["new"]) // 64 + 2 for p in prompts) + 1  # (the cache may hold what no row uses any more)
    eng = Engine(model, max_running=case["rows"], num_pages=pages, page_size=64, max_seq_len=max(map(len, prompts)) + case["new"] + 64, prefix_cache=True)
    # the conversation so far is in the cache (the engine keeps what it has seen), and decode steps have run before
    eng.generate([p[:-1] for p in prompts], SamplingParams(temperature=1.0, max_new_tokens=3, ignore_eos=True, sampling_seed=seed))
    state.update(engine=eng, prompts=prompts, params=SamplingParams(temperature=1.0, max_new_tokens=case["new"], ignore_eos=True, sampling_seed=seed))
    return state


def _gradient(case, seed, name, dtype):
    shape = _shapes(case)[name]
    return (torch.randn(shape, generator=_gen(seed, "gradient " + name), device="cuda", dtype=torch.bfloat16) * 1e-5).to(dtype)


# ---------------------------------------------------------------------------------------------- one pass
def run(state):
    kind = state["case"]["kind"]
    if kind == "decode":
        # (the sampled tokens are nearly certain, so their log-probabilities are nearly zero: the newest logits stand for them)
        eng = state["engine"]
        done = eng.generate(state["prompts"], state["params"])
        return {"tokens": torch.tensor([r["output_ids"] for r in done]), "logits": eng.d_logits[:len(done)]}
    if kind == "prefill":
        eng = state["engine"]
        logits = eng.feed([(str(i), p, [len(p) - 1]) for i, p in enumerate(state["prompts"])])
        for i in range(len(logits)):
            eng.end_feed(str(i))
        return {"logits": logits}
    if kind == "adam":
        opt, store = state["opt"], state["store"]
        norm = opt.step()
        return {"norm": norm, "weights": dict(store.flat), "state": {g: {k: s[k] for k in ("m", "v", "lo")} for g, s in opt.state.items()}}
    k, model = state["pack"], state["model"]
    if kind == "logprobs":
        lp, ent = model.forward_logprobs(k["tokens"], k["positions"], k["cu"], k["rows"], k["targets"], 1.0, replay=k["replay"], max_seqlen=max(k["lens"]))
        return {"logprobs": lp, "entropy": ent}
    state["store"].zero_grads()
    adv = k["advantages"]
    loss, _, lp, ent = model.forward_backward(k["tokens"], k["positions"], k["cu"], k["rows"], k["targets"], 1.0, lambda lp, ent: (-(adv * lp).mean(), {}),
                                              replay=k["replay"], max_seqlen=max(k["lens"]))
    return {"loss": loss, "logprobs": lp, "entropy": ent, "gradients": dict(state["store"].grads)}


# ---------------------------------------------------------------------------------------------- what a pass cannot do without
def _sizes(case):
    m = MODELS[case["model"]]
    H, q, kv, I = m["hidden"], m["heads"] * HEAD_DIM, m["kv_heads"] * HEAD_DIM, m["ffn"]
    attn, router, expert = H * (2 * q + 2 * kv), m["experts"] * H, 3 * H * I
    used = attn + (router + m["top_k"] * expert if m["experts"] else expert)       # weights a token meets in a layer
    # weights that `n` tokens meet in a layer (in expectation)
    met = lambda n: attn + (router + m["experts"] * (1 - (1 - m["top_k"] / m["experts"]) ** n) * expert if m["experts"] else expert)  # noqa: E731
    return m, attn, used, met


def work(case):
    m, attn, used, met = _sizes(case)
    L, H, V, kv_row = case["layers"], m["hidden"], m["vocab"], 2 * m["kv_heads"] * HEAD_DIM * 2
    q_heads = m["heads"] * HEAD_DIM
    if case["kind"] == "adam":
        n, b = 0, 0
        for name, shape in _shapes(case).items():
            k = math.prod(shape)
            s = 2 if case["state"] == "bf16" else 4
            n, b = n + k, b + k * (2 * (2 + 2) + 4 * s + (2 if ".moe.w" in name else 4))  # weight, remainder, two moments in and out, gradient in
        return {"bytes": b, "flops": 12 * n}
    if case["kind"] == "decode":
        rows, ctx, new = case["rows"], 0.875 * case["context"] + case["new"] / 2, case["new"]
        # the newest position of each row comes with a pass over the weights as well
        bytes_ = new * (L * (met(rows) * 2 + rows * ctx * kv_row) + V * H * 2 + rows * V * 4)
        return {"bytes": bytes_, "flops": new * rows * (2 * L * used + 4 * L * ctx * q_heads + 2 * V * H)}
    lens = [case["tokens"] / case["sequences"]] * case["sequences"]
    T, pairs = case["tokens"], sum(n * (n + 1) / 2 for n in lens)
    body = T * 2 * L * used + 4 * L * pairs * q_heads
    weights = L * met(T) * 2 + V * H * 2 * (1 if m["tied"] else 2 if T > V / 8 else 1)
    if case["kind"] == "prefill":
        n = case["sequences"]
        return {"bytes": weights + L * T * kv_row + n * V * 4, "flops": body + n * 2 * V * H}
    rows = 0.75 * T
    if case["kind"] == "logprobs":
        return {"bytes": weights + rows * 8, "flops": body + rows * 2 * V * H}
    # backward: twice the forward's products and, for attention, two and a half times; the recomputation is this package's own choice
    grads = L * met(T) * (2 if m["experts"] else 4) + V * H * 4 * (1 if m["tied"] else 2)
    return {"bytes": 2 * weights + grads, "flops": 3 * T * 2 * L * used + 3.5 * 4 * L * pairs * q_heads + 3 * rows * 2 * V * H}


def tolerance(case):
    """Activations and gradients travel in bf16: outputs of the layers lie up to 0.028 (gradients of the router) from the 64-bit ones, two runs 0.0065 from each other (atomics), log-probs,
    whose logits stay in 32 bits, 0.0014. Sampled tokens and the 16-bit remainders of the weights are whole numbers."""
    return {"rel": {"logprobs": 0.005, "adam": 0.005}.get(case["kind"], 0.03), "differ": 0.01}


# ---------------------------------------------------------------------------------------------- the same in 64 bits
def _norm(x, w):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS) * w


def _rope(x, pos):
    half = HEAD_DIM // 2
    a = pos.double()[:, None] * THETA ** (-torch.arange(half, device=x.device, dtype=torch.float64) / half)
    cos, sin = a.cos()[:, None], a.sin()[:, None]
    return torch.cat([x[..., :half] * cos - x[..., half:] * sin, x[..., half:] * cos + x[..., :half] * sin], -1)


def _attend(q, k, v, lens):
    outs, at, group = [], 0, q.shape[1] // k.shape[1]
    for n in lens:
        qs, ks, vs = (t[at:at + n].transpose(0, 1) for t in (q, k, v))
        heads = []
        for h in range(k.shape[1]):
            for a in range(0, n, 2048):  # some query rows at a time: the scores of all of them would not fit
                s = torch.matmul(qs[h * group:(h + 1) * group, a:a + 2048], ks[h].t()) * HEAD_DIM ** -0.5
                rows = torch.arange(a, min(a + 2048, n), device=q.device)
                s = s.masked_fill(torch.arange(n, device=q.device)[None] > rows[:, None], -math.inf)
                heads.append(torch.matmul(torch.softmax(s, -1), vs[h]))
        per = len(range(0, n, 2048))
        outs.append(torch.cat([torch.cat(heads[h * per:(h + 1) * per], 1) for h in range(k.shape[1])], 0).transpose(0, 1))
        at += n
    return torch.cat(outs, 0)


def _layer(x, pos, lens, m, ids, ln1, qkv, qn, kn, o, ln2, *ff):
    T = x.shape[0]
    h = (_norm(x, ln1) @ qkv.t()).view(T, -1, HEAD_DIM)
    nq, nk = m["heads"], m["kv_heads"]
    q, k, v = _rope(_norm(h[:, :nq], qn), pos), _rope(_norm(h[:, nq:nq + nk], kn), pos), h[:, nq + nk:]
    x = x + _attend(q, k, v, lens).reshape(T, -1) @ o.t()
    h = _norm(x, ln2)
    if not m["experts"]:
        g, u = (h @ ff[0].t()).chunk(2, -1)
        return x + (F.silu(g) * u) @ ff[1].t()
    router, w1, w2 = ff
    probs = torch.softmax(h @ router.t(), -1)
    ids = probs.topk(m["top_k"], -1).indices if ids is None else ids.long()
    w = probs.gather(1, ids)
    w = w / w.sum(-1, keepdim=True)
    y = torch.zeros_like(x)
    for e in range(m["experts"]):
        t, slot = (ids == e).nonzero(as_tuple=True)
        if t.numel():
            g, u = (h[t] @ w1[e].to(h.dtype).t()).chunk(2, -1)
            y = y.index_add(0, t, ((F.silu(g) * u) @ w2[e].to(h.dtype).t()) * w[t, slot][:, None])
    return x + y


def _names(case, i):
    return [n for n in _shapes(case) if n.startswith(f"layers.{i}.")]


def _hidden(case, seed, tokens, lens, replay=None, params=None):
    """The final hidden states; ``params``: 64-bit leaves to differentiate by, else weights are made layer by layer."""
    m = MODELS[case["model"]]
    get = (lambda n: params[n]) if params is not None else (lambda n: _weight(case, seed, n) if ".moe.w" in n else _weight(case, seed, n).double())
    pos = torch.cat([torch.arange(n) for n in lens]).cuda()
    x = get("embed.weight")[tokens]
    for i in range(case["layers"]):
        args = (x, pos, lens, m, None if replay is None else replay[:, i], *[get(n) for n in _names(case, i)])
        x = checkpoint(_layer, *args, use_reentrant=False) if params is not None else _layer(*args)
    return _norm(x, get("final_norm.weight"))


def _head(case, seed):
    return _weight(case, seed, "embed.weight" if MODELS[case["model"]]["tied"] else "lm_head.weight").double()


def _scores(h, w, targets):
    ls = torch.log_softmax(h @ w.t(), -1)
    return ls.gather(1, targets.long()[:, None])[:, 0], -(ls.exp() * ls).sum(-1)


def exact(case, seed):
    m = MODELS[case["model"]]
    if case["kind"] == "adam":
        return _exact_adam(case, seed)
    if case["kind"] == "decode":
        with torch.no_grad():
            step = 0 if m["tied"] else 1
            seqs = [p + [(p[-1] + step * j) % m["vocab"] for j in range(1, case["new"])] for p in _prompts(case, seed)]
            lens = [len(s) for s in seqs]
            h = _hidden(case, seed, torch.tensor(sum(seqs, []), device="cuda"), lens)
            ends = torch.tensor(lens, device="cuda").cumsum(0) - 1
            return {"tokens": None, "logits": h[ends] @ _head(case, seed).t()}
    if case["kind"] == "prefill":
        with torch.no_grad():
            lens = _lengths(case)
            toks = torch.cat([_tokens(case, seed, n, f"prompt {i}") for i, n in enumerate(lens)]).cuda()
            h = _hidden(case, seed, toks, lens)[torch.tensor(lens, device="cuda").cumsum(0) - 1]
            return {"logits": list((h @ _head(case, seed).t()).split(1))}
    k = _pack(case, seed)
    toks = k["tokens"].long()
    if case["kind"] == "logprobs":
        with torch.no_grad():
            h, w = _hidden(case, seed, toks, k["lens"], k["replay"])[k["rows"]], _head(case, seed)
            got = [_scores(h[a:a + 2048], w, k["targets"][a:a + 2048]) for a in range(0, h.shape[0], 2048)]
            return {"logprobs": torch.cat([a for a, _ in got]), "entropy": torch.cat([b for _, b in got])}
    params = {n: _weight(case, seed, n).double().requires_grad_(True) for n in _shapes(case)}
    h = _hidden(case, seed, toks, k["lens"], k["replay"], params)[k["rows"]]
    w = params["embed.weight" if m["tied"] else "lm_head.weight"]
    got = [checkpoint(_scores, h[a:a + 1024], w, k["targets"][a:a + 1024], use_reentrant=False) for a in range(0, h.shape[0], 1024)]
    lp, ent = torch.cat([a for a, _ in got]), torch.cat([b for _, b in got])
    loss = -(k["advantages"].double() * lp).mean()
    loss.backward()
    return {"loss": loss.detach(), "logprobs": lp.detach(), "entropy": ent.detach(), "gradients": {n: p.grad for n, p in params.items()}}


def _exact_adam(case, seed):
    """The flat buffers hold each group's tensors one after another, each padded to 128 elements."""
    out = {"norm": None, "weights": {}, "state": {}}
    total = 0.0
    for group in ("dense", "expert"):
        names = [n for n in _shapes(case) if (".moe.w" in n) == (group == "expert")]
        if not names:
            continue
        parts = {"w": [], "m": [], "v": []}
        for n in names:
            g = _gradient(case, seed, n, torch.bfloat16).double().view(-1)
            w = _weight(case, seed, n).double().view(-1)
            total += float(g.square().sum())
            decay = ADAM["weight_decay"] if len(_shapes(case)[n]) > 1 else 0.0
            new = w - ADAM["lr"] * (g / (g.abs() + ADAM["eps"]) + decay * w)
            pad = -g.numel() % 128
            for key, t in (("w", new), ("m", (1 - ADAM["beta1"]) * g), ("v", (1 - ADAM["beta2"]) * g * g)):
                parts[key].append(F.pad(t, (0, pad)))
        out["weights"][group] = torch.cat(parts["w"])
        out["state"][group] = {"m": torch.cat(parts["m"]), "v": torch.cat(parts["v"]), "lo": None}
    out["norm"] = torch.tensor(math.sqrt(total), dtype=torch.float64)
    return out
