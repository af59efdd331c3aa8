"""Hand-scheduled sm_100a execution of the Qwen3 dense / MoE decoder (training and inference).

There is no autograd graph and no tracing compiler on this path: forward and backward of a decoder
layer are explicit sequences of kernel launches (tcgen05 GEMMs, fused norm / rope / swiglu / routing
kernels). The backward takes the activations of the last layers, and the logits, from where the forward
left them as far as the device has room, and recomputes the other layers from their inputs (the "full
recompute" policy of the reference recipe scripts/run_qwen3_30b_a3b.py:168-175, which runs where nothing
fits). Weight gradients are accumulated by the GEMM epilogue directly into the persistent flat gradient
buffer (the role of Megatron's ``main_grad`` + gradient-accumulation fusion).

The same object serves the rollout engine (prefill and paged-KV decode), so trainer and engine share
weights, kernels and rounding points — the basis for trainer/rollout log-prob parity. Reduction orders are the same in
passes of more than 128 rows; for fewer the engine has kernels that cut a sum over K into parts (``linear``).
"""
from __future__ import annotations

from dataclasses import dataclass
from typing import NamedTuple, Optional

import torch

from ..ops import _ext
from ..ops.attention import TileCache
from .config import ModelConfig
from .params import ParamStore
from .torch_impl import InferMeta


@dataclass
class MoeCtx:
    ids: torch.Tensor
    w: torch.Tensor
    probs: torch.Tensor
    offsets: torch.Tensor
    dest: torch.Tensor
    src: torch.Tensor
    tile_group: torch.Tensor
    num_tiles: torch.Tensor
    max_rows: int
    align: int = 1
    pairs: int = 0  # routed pairs to expect among max_rows (0: as many)

    def gated(self) -> bool:
        """Whether the gate-up product of these rows takes SwiGLU into its epilogue (csrc/gemm.cu). Experts of few rows stream their weights, which
        the plain product does faster, by more than the activation costs; where every expert's rows are padded to whole tiles the activation
        works through the padding, too, and nothing is lost. us, plain product and activation / gated, 128 experts of 768 x 2048: 16 tokens
        111 / 118, 200 153 / 159, 777 (49 pairs an expert) 159 / 162, 1500 171 / 168, 4000 255 / 226; 128 of 1536 x 4096: 200 tokens 513 / 517, 400
        (25 pairs) 525 / 523, 1000 548 / 534; padded to 64 rows, gate and up kept: 16 tokens 124 / 125, 200 171 / 170, 777 169 / 170, 1500
        183 / 178, 4000 267 / 249."""
        return self.align > 1 or (self.pairs or self.max_rows) >= 48 * (self.offsets.numel() - 1)


class LayerActs(NamedTuple):
    """What the backward of a layer needs of its forward."""
    qkv: tuple                    # h1, rstd1, qkv, q, k, q_rstd, k_rstd
    att: torch.Tensor
    lse: object
    ln2: tuple                    # h2, rstd2, x2
    post_attn: Optional[tuple]
    moe: Optional[tuple]
    mlp: Optional[tuple]          # gate | up, SwiGLU


def plan_kept(room: int, head_bytes: int, layer_bytes: list, first: int) -> tuple[bool, int]:
    """What fits into ``room`` bytes: (the logits, the first of the last layers whose activations are kept). The last ones,
    since they are the first to be given back. A mixture's layer of 16384 tokens is 2.4 GB and 3.2 ms of recomputation, 12288
    rows of 151936 logits are 7.5 GB and 6 ms, so the logits come first. Whole passes, all recomputed -> all kept: four layers
    and 16384 tokens of the mixture with its head 91.7 -> 70.5 ms, 777 tokens 12.3 -> 10.5, three layers of 4096 x 12288 with
    9216 tokens 89.8 -> 71.6."""
    head = 0 < head_bytes <= room
    room -= head_bytes if head else 0
    keep = first + len(layer_bytes)
    for b in reversed(layer_bytes):
        if b > room:
            break
        room -= b
        keep -= 1
    return head, keep


ALL_LAYERS = 1 << 30


def recompute_policy(args) -> tuple[int, bool]:
    """(how many of a stage's first layers are recomputed in the backward whatever there is room for, whether the logits are):
    ``--recompute-granularity full`` asks for all layers, or for --recompute-num-layers of them with ``--recompute-method block``;
    without it, and with ``none`` and ``selective``, those are recomputed whose activations do not fit. ``--recompute-loss-function`` asks
    for the logits."""
    layers = 0
    if getattr(args, "recompute_granularity", None) == "full":
        layers = int(args.recompute_num_layers or 0) if getattr(args, "recompute_method", None) == "block" else ALL_LAYERS
    return layers, bool(getattr(args, "recompute_loss_function", None))


def _out_of_memory(e: RuntimeError) -> bool:
    """What the allocator raises, be it called by PyTorch or by the extension."""
    return isinstance(e, torch.OutOfMemoryError) or "out of memory" in str(e)


class B200Qwen3:
    def __init__(self, cfg: ModelConfig, store: ParamStore, ep=None, tp=None):
        assert cfg.head_dim == 128, "the sm_100a attention/rope kernels are specialised for head_dim 128"
        self.cfg = store.cfg  # under tensor parallelism: this rank's view (local head counts, local FFN width)
        self.store = store
        self.ep = ep  # expert-parallel dispatcher (None = all experts local)
        self.tp = tp if (tp is not None and tp.n > 1) else None  # tensor-parallel exchange (None = not sharded)
        assert not (self.tp is not None and ep is not None), "tensor parallel attention with expert parallel MoE is not supported"
        self.C = _ext.load(required=True)
        self.dev = store.device
        self.status = torch.zeros(1, dtype=torch.int32, device=self.dev)
        self.launches = 0  # number of this library's kernels launched (reported by the benchmark)
        self._decode_scratch: Optional[torch.Tensor] = None
        self._tiles = TileCache()
        self.cp_ctx = None  # (sample lengths, cp size, cp rank, group, comm, layout) while a context-parallel micro-batch runs
        self._ident: Optional[torch.Tensor] = None
        self.small_decode = True  # weight-streaming kernels for decode steps of at most SMALL_T rows
        self.act_room: Optional[int] = None  # bytes of activations a training pass may keep (None: by what is free, see _room_for_acts)
        self.recompute_layers = 0     # of the stage's first layers no activations are kept, whatever there is room for (recompute_policy)
        self.recompute_logits = False
        self.lm_chunk = 2048      # rows of the LM head per pass (--log-probs-chunk-size)

    def attention(self, q, k, v, cu):
        """Causal attention over packed sequences: returns (out [T, Hq, 128], lse [Hq, T]).

        Under context parallelism (``cp_ctx`` set by the trainer: the rows are this rank's shard of every sequence)
        the sequence shard is traded for a head shard with one all-to-all per tensor, the kernel attends over whole
        sequences with ``Hq / cp`` query heads, and the output is traded back; what the backward needs in that layout
        travels in the second return value. NVSwitch gives the all-to-all full bandwidth between every pair, so this
        layout, not a ring of K/V blocks, is the one built for this path."""
        if self.cp_ctx is not None:
            return self._attention_cp(q, k, v)
        out, lse = self.C.flash_attn_fwd(q, k, v, self._tiles.get(cu), self.cfg.head_dim ** -0.5, self.status)
        self.launches += 1
        return out, lse

    def attention_backward(self, q, k, v, out, d_out, lse, cu):
        """dQ, dK, dV of :meth:`attention` from its output and log-sum-exp (tcgen05 kernel, csrc/attention_bwd.cu)."""
        if isinstance(lse, tuple):
            return self._attention_cp_backward(d_out, lse)
        dq, dk, dv = self.C.flash_attn_bwd(q, k, v, out, d_out.contiguous(), lse, self._tiles.get_bwd(cu),
                                           self.cfg.head_dim ** -0.5, self.status,
                                           self._tiles.get_bwd_split(cu, q.shape[1], k.shape[1]))
        self.launches += 3
        return dq, dk, dv

    def _cp_full_cu(self, lens):
        key = tuple(lens)
        if getattr(self, "_cp_cu_key", None) != key:
            self._cp_cu = torch.tensor([0] + list(torch.tensor(list(lens)).cumsum(0).tolist()), dtype=torch.int32, device=self.dev)
            self._cp_cu_key = key
        return self._cp_cu

    def _attention_cp(self, q, k, v):
        from ..parallel.context_parallel import heads_to_sequence, sequence_to_heads

        lens, cp, rank, group = self.cp_ctx[:4]
        layout = self.cp_ctx[5] if len(self.cp_ctx) > 5 else "zigzag"
        cfg = self.cfg
        assert cfg.num_kv_heads % cp == 0, (f"context parallelism on this path shards the {cfg.num_kv_heads} key / value heads "
                                            f"over the {cp} ranks (all-to-all layout)")
        qf, kf, vf = (heads_to_sequence(t.contiguous(), lens, cp, rank, group, layout).contiguous() for t in (q, k, v))
        cu = self._cp_full_cu(lens)
        out_f, lse_f = self.C.flash_attn_fwd(qf, kf, vf, self._tiles.get(cu), cfg.head_dim ** -0.5, self.status)
        self.launches += 1
        out = sequence_to_heads(out_f, lens, cp, rank, group, layout).contiguous()  # (a view when a rank holds one head)
        return out, (lse_f, qf, kf, vf, out_f, cu)

    def _attention_cp_backward(self, d_out, saved):
        from ..parallel.context_parallel import heads_to_sequence, sequence_to_heads

        lens, cp, rank, group = self.cp_ctx[:4]
        layout = self.cp_ctx[5] if len(self.cp_ctx) > 5 else "zigzag"
        lse_f, qf, kf, vf, out_f, cu = saved
        do_f = heads_to_sequence(d_out.contiguous(), lens, cp, rank, group, layout).contiguous()
        dqf, dkf, dvf = self.C.flash_attn_bwd(qf, kf, vf, out_f, do_f, lse_f, self._tiles.get_bwd(cu), self.cfg.head_dim ** -0.5,
                                              self.status, self._tiles.get_bwd_split(cu, qf.shape[1], kf.shape[1]))
        self.launches += 3
        return tuple(sequence_to_heads(t, lens, cp, rank, group, layout).contiguous() for t in (dqf, dkf, dvf))

    # ------------------------------------------------------------------ GEMM helpers
    def _gemm(self, a, b, out, a_mn=False, b_mn=False, acc=False):
        self.C.gemm(a, b, out, a_mn, b_mn, acc, 0, self.status)
        self.launches += 1
        return out

    # ------------------------------------------------------------------ block-scaled inference weights
    MX_SUFFIXES = ("attn.qkv.weight", "attn.o.weight", "mlp.gate_up.weight", "mlp.down.weight", "moe.w1", "moe.w2")

    def enable_block_scaled(self, kind: str) -> int:
        """Serve the projections and experts from MXFP8 / NVFP4 copies of the weights (`csrc/gemm_mx.cu`) whenever
        more than 32 rows are multiplied; the few-row decode kernels keep streaming the bf16 weights. Meant for a
        model object that only the rollout engine uses. Call again (or `refresh_block_scaled`) after a weight update.
        Returns the number of tensors quantised."""
        from ..ops.mx_gemm import quantize_operand

        step = 128 if kind == "mxfp8" else 256
        self.mx_kind, self.mx = kind, {}
        for name, w in self.store.params.items():
            if not name.endswith(self.MX_SUFFIXES):
                continue
            w2 = w.reshape(-1, w.shape[-1])
            if w2.shape[1] % step or w2.shape[0] % 128:
                continue
            self.mx[w.data_ptr()] = quantize_operand(w2, kind)
        return len(self.mx)

    def use_block_scaled(self, kind: str, operands: dict) -> None:
        """Serve from block-scaled copies that something else keeps up to date (``{parameter name: MxOperand}``, e.g.
        the buffers a peer-memory weight push quantises into)."""
        self.mx_kind, self.mx_external = kind, True
        self.mx = {self.store.params[n].data_ptr(): op for n, op in operands.items() if n in self.store.params}

    def refresh_block_scaled(self) -> None:
        if getattr(self, "mx_external", False):
            return
        if getattr(self, "mx", None):
            self.enable_block_scaled(self.mx_kind)

    def _mx_linear(self, x, wq, tile_group=None, num_tiles=None, n: int = 0, amax=None):
        from ..ops.mx_gemm import mx_linear, quantize_operand

        xq = quantize_operand(x, self.mx_kind, amax)
        self.launches += 3
        return mx_linear(xq, wq, self.status, tile_group, num_tiles, n)

    def linear(self, x, w, out_dtype=torch.bfloat16, serving=False):
        """``x @ w^T``. In passes that train or score, every sum over K of 33 rows and more runs in one order, so that a sample's
        log-probs do not depend on how much else is in its pack. (Gradients do, in their last bits: those of the weights add up the pack, dQ is
        summed by atomics, and who adds up the heads of dK and dV is chosen by the pack's lengths, ops/attention.py.) Passes of the
        engine (``serving``) may split the contraction of up to 128 rows over a cluster (csrc/gemm_skinny.cu)."""
        T, (N, K) = x.shape[0], w.shape
        mx = getattr(self, "mx", None)
        if mx and T > 32 and out_dtype == torch.bfloat16 and w.data_ptr() in mx:
            return self._mx_linear(x.contiguous(), mx[w.data_ptr()])
        out = torch.empty(x.shape[0], w.shape[0], dtype=out_dtype, device=x.device)
        if T <= 8 and self.small_decode and N % 16 == 0 and K % 32 == 0 and N * K * 2 < (48 << 20) and x.is_contiguous():
            # a few rows against a small weight matrix (decode projections): the blocks that start fastest
            self.C.small_gemv(x, None, 0.0, w, None, out, self.status)
            self.launches += 1
            return out
        split = self.small_decode and (serving or T <= 32)
        self.C.gemm(x, w, out, False, False, False, 0, self.status, whole_k=not split)
        self.launches += 1
        return out

    def _gated(self, x, w, keep: bool = False, serving: bool = False):
        """``(gate | up if kept, silu(gate) * up)`` for a gate-up weight [2I, K]: one launch where tiles of 128 such columns fill
        the device (csrc/gemm.cu), else the product and the activation. The same bits either way."""
        T, I = x.shape[0], w.shape[0] // 2
        mx = getattr(self, "mx", None)
        if T > 128 and I % 8 == 0 and -(-T // 128) * -(-I // 128) >= 148 and x.is_contiguous() and not (mx and w.data_ptr() in mx):
            gu = torch.empty(T, 2 * I, dtype=torch.bfloat16, device=x.device) if keep else None
            act = torch.empty(T, I, dtype=torch.bfloat16, device=x.device)
            self.C.gated_gemm(x, w, act, gu, None, None, self.status)
            self.launches += 1
            return gu, act
        gu = self.linear(x, w, serving=serving)
        self.launches += 1
        return gu if keep else None, self.C.swiglu_fwd(gu)

    def linear_dgrad(self, dy, w):
        dx = torch.empty(dy.shape[0], w.shape[1], dtype=torch.bfloat16, device=dy.device)
        return self._gemm(dy, w, dx, False, True)

    def linear_wgrad(self, dy, x, dw):
        """dw [N,K] += dy[M,N]^T . x[M,K]"""
        return self._gemm(dy, x, dw, True, True, True)

    def check_status(self) -> None:
        code = int(self.status.item())
        if code != 0:
            self.status.zero_()
            raise RuntimeError(f"a miles_b200 kernel reported error status {code} (bounded wait expired)")

    # ------------------------------------------------------------------ MoE block
    def _route(self, h2, router_w, replay_ids, bias=None, serving=False):
        cfg, C = self.cfg, self.C
        logits = self.linear(h2, router_w, torch.float32, serving)
        if cfg.router_score == "sigmoid":
            # GLM-4.5 / DeepSeek-V3 routing: a [T, E] problem, done with framework ops (ops/reference.py); what the
            # backward needs is the logits, kept in the place of the softmax probabilities
            from ..ops.reference import router_sigmoid_topk

            ids, w, _ = router_sigmoid_topk(logits, cfg.moe_top_k, cfg.norm_topk_prob, bias, cfg.routed_scaling_factor,
                                            cfg.n_group, cfg.topk_group, replay_ids)
            self.launches += 8
            return ids.contiguous(), w.contiguous(), logits
        rid = replay_ids.contiguous() if replay_ids is not None else None
        ids, w, probs = C.moe_router_topk(logits, rid, cfg.moe_top_k, cfg.norm_topk_prob, True)
        self.launches += 1
        return ids, w, probs

    def _permute_plan(self, ids, E_local, align: int = 1) -> MoeCtx:
        """Expert-sorted row layout. ``align`` pads every expert's rows: 64 when weight gradients will be taken
        (the wgrad contraction runs in 64-row blocks that must not straddle experts), 1 for inference."""
        T, K = ids.shape
        max_rows = max(T * K + E_local * (align - 1), 1)
        counts, offsets, dest, src, tg, nt = self.C.moe_build_permutation(ids, E_local, max_rows, align)
        self.launches += self.C.moe_permutation_launches(T, K, max_rows, E_local)
        return MoeCtx(ids, None, None, offsets, dest, src, tg, nt, max_rows, align, T * K)

    def _experts_fwd(self, xp, plan: MoeCtx, w1, w2, keep: bool, scatter=None):
        """``scatter = (row_ptrs, ctrl, flag_ptrs, rank)``: the second GEMM stores every output row at its own
        address (the expert-parallel return buffers of the ranks the tokens came from) and raises their flags."""
        C = self.C
        I2 = w1.shape[1]
        mx = getattr(self, "mx", None)
        if mx and not keep and scatter is None and w1.data_ptr() in mx and w2.data_ptr() in mx and plan.align == 128:
            # rows of xp past the live tiles are never written: the per-tensor scale of NVFP4 must not look at them
            gu = self._mx_linear(xp, mx[w1.data_ptr()], plan.tile_group, plan.num_tiles, I2, getattr(plan, "amax_in", None))
            act = C.swiglu_fwd(gu)
            yp = self._mx_linear(act, mx[w2.data_ptr()], plan.tile_group, plan.num_tiles, w2.shape[1])
            self.launches += 1
            return None, None, yp
        gated = plan.gated()
        gu = torch.empty(plan.max_rows, I2, dtype=torch.bfloat16, device=xp.device) if keep or not gated else None
        if gated:
            act = torch.empty(plan.max_rows, I2 // 2, dtype=torch.bfloat16, device=xp.device)
            C.gated_gemm(xp, w1, act, gu, plan.tile_group, plan.num_tiles, self.status)
        else:
            C.grouped_gemm_rows(xp, w1, gu, plan.tile_group, plan.num_tiles, False, False, 0, self.status)
            act = C.swiglu_fwd(gu)
            self.launches += 1
        yp = torch.empty(plan.max_rows if scatter is None else 1, w2.shape[1], dtype=torch.bfloat16, device=xp.device)
        if scatter is None:
            C.grouped_gemm_rows(act, w2, yp, plan.tile_group, plan.num_tiles, False, False, 0, self.status)
        else:
            C.grouped_gemm_rows(act, w2, yp.expand(plan.max_rows, -1), plan.tile_group, plan.num_tiles, False, False, 0,
                                self.status, scatter[0], scatter[1], scatter[2], scatter[3])
        self.launches += 2
        return (gu, act, yp) if keep else (None, None, yp)

    def moe_forward(self, i, h2, replay_ids=None, record=None, keep=False, residual=None, serving=False):
        cfg, P, C = self.cfg, self.store.params, self.C
        p = f"layers.{i}.moe."
        ids, w, probs = self._route(h2, P[p + "router.weight"], replay_ids, P.get(p + "router.bias"), serving)
        if record is not None:
            record.append(ids)
        if cfg.shared_expert_ffn and not (keep and residual is None):  # (the backward's recompute does not need the output)
            # the shared expert sees every token: its output joins the residual that the combine adds
            sh_gu = self.linear(h2, P[p + "shared.gate_up.weight"], serving=serving)
            sh_y = self.linear(C.swiglu_fwd(sh_gu), P[p + "shared.down.weight"], serving=serving)
            if cfg.shared_expert_gate:  # one sigmoid gate value per token (a [T, H] x [H] product: framework ops)
                g = torch.sigmoid(h2.float() @ P[p + "shared.gate.weight"].float().t())
                sh_y = (sh_y.float() * g).to(sh_y.dtype)
                self.launches += 3
            residual = sh_y.add_(residual) if residual is not None else sh_y
            self.launches += 3
        if self.ep is not None:
            return self.ep.moe_forward(self, i, h2, ids, w, probs, keep, residual)
        use_mx = bool(getattr(self, "mx", None)) and not keep and h2.shape[0] > 32
        plan = self._permute_plan(ids, cfg.num_experts, 64 if keep else (128 if use_mx else 1))
        plan.w, plan.probs = w, probs
        xp = C.moe_permute(h2, plan.src, plan.num_tiles, cfg.moe_top_k)
        if use_mx and self.mx_kind == "nvfp4":
            plan.amax_in = C.absmax(h2.contiguous())  # the permuted rows hold exactly these values
        gu, act, yp = self._experts_fwd(xp, plan, P[p + "w1"], P[p + "w2"], keep)
        y = C.moe_combine(yp, plan.dest, w, h2.shape[0], cfg.moe_top_k, residual)
        self.launches += 2
        saved = (plan, xp, gu, act, yp) if keep else None
        return y, saved

    def moe_backward(self, i, h2, dy, saved):
        """Returns dh2 (gradient wrt the normalised MoE input); accumulates router / expert weight grads."""
        cfg, P, G, C = self.cfg, self.store.params, self.store.grads, self.C
        p = f"layers.{i}.moe."
        if self.ep is not None:
            dh2 = self.ep.moe_backward(self, i, h2, dy, saved)
            return self._shared_expert_bwd(i, h2, dy, dh2)
        plan, xp, gu, act, yp = saved
        w1, w2 = P[p + "w1"], P[p + "w2"]
        dyp, dw = C.moe_combine_bwd(dy, yp, plan.src, plan.num_tiles, plan.w)
        dxp = self._experts_bwd(dyp, xp, gu, act, plan, w1, w2, G[p + "w1"], G[p + "w2"])
        dh2 = C.moe_combine(dxp, plan.dest, None, h2.shape[0], cfg.moe_top_k)
        self.launches += 2
        dh2 = self._router_bwd(i, h2, dh2, plan.probs, plan.ids, plan.w, dw)
        return self._shared_expert_bwd(i, h2, dy, dh2)

    def _shared_expert_bwd(self, i, h2, dy, dh2):
        """The shared expert's part of the MoE backward (recomputed from ``h2``): weight gradients, and its input gradient
        added to ``dh2``."""
        cfg, P, G, C = self.cfg, self.store.params, self.store.grads, self.C
        if not cfg.shared_expert_ffn:
            return dh2
        p = f"layers.{i}.moe.shared."
        wgu, wd = P[p + "gate_up.weight"], P[p + "down.weight"]
        dyb = dy if dy.dtype == torch.bfloat16 else dy.to(torch.bfloat16)
        gu = self.linear(h2, wgu)
        act = C.swiglu_fwd(gu)
        if cfg.shared_expert_gate:
            # y = g * s with g = sigmoid(h2 . w_g), s the shared expert's output (recomputed): ds = g dy,
            # d(logit) = (dy . s) g (1 - g), which reaches w_g and h2
            wg = P[p + "gate.weight"]
            s = self.linear(act, wd).float()
            g = torch.sigmoid(h2.float() @ wg.float().t())
            dlogit = (dy.float() * s).sum(-1, keepdim=True) * g * (1.0 - g)
            G[p + "gate.weight"].add_((dlogit.t() @ h2.float()).to(G[p + "gate.weight"].dtype))
            dh2.add_((dlogit @ wg.float()).to(dh2.dtype))
            dyb = (dy.float() * g).to(torch.bfloat16)
            self.launches += 8
        self.linear_wgrad(dyb, act, G[p + "down.weight"])
        dgu = C.swiglu_bwd(self.linear_dgrad(dyb, wd), gu)
        self.linear_wgrad(dgu, h2, G[p + "gate_up.weight"])
        self._gemm(dgu, wgu, dh2, False, True, True)  # dh2 += dgu . W
        self.launches += 7
        return dh2

    def _experts_bwd(self, dyp, xp, gu, act, plan, w1, w2, gw1, gw2, scatter=None):
        C = self.C
        dact = torch.empty_like(act)
        C.grouped_gemm_rows(dyp, w2, dact, plan.tile_group, plan.num_tiles, True, False, 0, self.status)
        C.grouped_gemm_contr(dyp, act, gw2, plan.offsets, True, 0, self.status)
        dgu = C.swiglu_bwd(dact, gu)
        if scatter is None:
            dxp = torch.empty_like(xp)
            C.grouped_gemm_rows(dgu, w1, dxp, plan.tile_group, plan.num_tiles, True, False, 0, self.status)
        else:  # the input-gradient rows go straight back to the ranks that own the tokens
            dxp = torch.empty(1, xp.shape[1], dtype=xp.dtype, device=xp.device)
            C.grouped_gemm_rows(dgu, w1, dxp.expand(xp.shape[0], -1), plan.tile_group, plan.num_tiles, True, False, 0,
                                self.status, scatter[0], scatter[1], scatter[2], scatter[3])
        C.grouped_gemm_contr(dgu, xp, gw1, plan.offsets, True, 0, self.status)
        self.launches += 5
        return dxp

    def _router_bwd(self, i, h2, dh2, probs, ids, w, dw):
        cfg, P, G, C = self.cfg, self.store.params, self.store.grads, self.C
        p = f"layers.{i}.moe."
        if cfg.router_score == "sigmoid":
            # ``probs`` holds the router logits (see _route): differentiate the [T, E] routing function with autograd
            from ..ops.reference import router_sigmoid_topk

            with torch.enable_grad():
                lg = probs.detach().requires_grad_(True)
                _, w2, _ = router_sigmoid_topk(lg, cfg.moe_top_k, cfg.norm_topk_prob, None, cfg.routed_scaling_factor, 1, 1, ids)
                (dlogits,) = torch.autograd.grad(w2, lg, dw.to(w2.dtype))
            dlogits = dlogits.to(torch.bfloat16)
            self.launches += 10
        else:
            dlogits = C.moe_router_bwd(probs, ids, w, dw, cfg.norm_topk_prob).to(torch.bfloat16)
        self._gemm(dlogits, P[p + "router.weight"], dh2, False, True, True)
        self.linear_wgrad(dlogits, h2, G[p + "router.weight"])
        self.launches += 1
        return dh2

    # ------------------------------------------------------------------ layer forward / backward
    def _attn_qkv(self, i, x, positions, meta: Optional[InferMeta], kv_cache):
        cfg, P, C = self.cfg, self.store.params, self.C
        p = f"layers.{i}."
        h1, rstd1 = C.rmsnorm_fwd(x, None, P[p + "ln1.weight"], cfg.rms_eps)
        qkv = self.linear(h1, P[p + "attn.qkv.weight"], serving=meta is not None)
        if cfg.qkv_bias:
            qkv += P[p + "attn.qkv.bias"]
        kc = vc = slots = None
        if kv_cache is not None:
            kc, vc = kv_cache[i]
            slots = meta.slot_mapping
        write_k = meta is None or meta.is_prefill
        if cfg.rope_scaling or cfg.rotary_dim:
            q, k, qr, kr = C.qk_norm_rope_fwd_scaled(qkv, P.get(p + "attn.q_norm.weight"), P.get(p + "attn.k_norm.weight"),
                                                     positions, cfg.num_q_heads, cfg.num_kv_heads, cfg.rope_theta, cfg.rms_eps,
                                                     kc, vc, slots, write_k, self._rope_table(), cfg.rotary_dim or cfg.head_dim)
        else:
            q, k, qr, kr = C.qk_norm_rope_fwd(qkv, P.get(p + "attn.q_norm.weight"), P.get(p + "attn.k_norm.weight"), positions,
                                              cfg.num_q_heads, cfg.num_kv_heads, cfg.rope_theta, cfg.rms_eps, kc, vc, slots,
                                              write_k)
        self.launches += 2
        return h1, rstd1, qkv, q, k, qr, kr

    def _rope_table(self) -> Optional[torch.Tensor]:
        """The inverse frequencies of a model with scaled rotary embeddings (fp32, on the device); None without scaling
        (the kernels then compute theta^(-d / half) themselves)."""
        if not self.cfg.rope_scaling:
            return None
        t = getattr(self, "_inv_freq", None)
        if t is None:
            from ..ops.reference import rope_inv_freq

            t = self._inv_freq = rope_inv_freq(self.cfg.rotary_dim or self.cfg.head_dim, self.cfg.rope_theta, self.cfg.rope_scaling,
                                               self.dev).contiguous()
        return t

    def _v_view(self, qkv):
        cfg = self.cfg
        return qkv.view(qkv.shape[0], cfg.num_q_heads + 2 * cfg.num_kv_heads, cfg.head_dim)[:, cfg.num_q_heads + cfg.num_kv_heads:]

    def layer_forward(self, i, x, positions, cu, max_seqlen, meta: Optional[InferMeta] = None, kv_cache=None,
                      replay_ids=None, record=None):
        """Inference/no-grad forward of one layer: returns the layer output."""
        cfg, P, C = self.cfg, self.store.params, self.C
        p = f"layers.{i}."
        if (meta is not None and not meta.is_prefill and x.shape[0] <= self.SMALL_T and replay_ids is None
                and self.small_decode and self.tp is None and not cfg.post_norms):
            # the fused few-row MoE kernels serve plain softmax routers whose expert count fits their 16-column tiles
            plain_moe = cfg.router_score == "softmax" and not cfg.shared_expert_ffn and cfg.num_experts % 16 == 0
            if (self.ep is None and plain_moe) or not cfg.layer_is_moe(i):
                return self._layer_forward_small(i, x, positions, meta, kv_cache, record)
            # expert-parallel MoE: the attention half still takes the light kernels, the experts go through the exchange
            x2 = self._attn_small(i, x, positions, meta, kv_cache)
            if getattr(self.ep, "low_latency", False) and plain_moe:
                return self.ep.moe_decode(self, i, x2, None, record)
            h2, _ = C.rmsnorm_fwd(x2, None, P[p + "ln2.weight"], cfg.rms_eps)
            self.launches += 1
            y, _ = self.moe_forward(i, h2, replay_ids, record, keep=False, residual=x2, serving=True)
            return y
        serving = meta is not None
        h1, rstd1, qkv, q, k, _, _ = self._attn_qkv(i, x, positions, meta, kv_cache)
        scale = cfg.head_dim ** -0.5
        if meta is not None and not meta.is_prefill:
            att = torch.empty_like(q)
            B = q.shape[0]
            splits = self._decode_splits(B, meta)
            need = B * cfg.num_q_heads * splits * 130
            if self._decode_scratch is None or self._decode_scratch.numel() < need:
                self._decode_scratch = torch.empty(need, dtype=torch.float32, device=self.dev)
            kc, vc = kv_cache[i]
            C.paged_decode_attention(q, kc, vc, meta.block_table, meta.seq_lens, att, self._decode_scratch, meta.page_size,
                                     splits, scale)
            self.launches += 1
        elif meta is not None and getattr(meta, "prefix", None) is not None:
            # prefill behind a cached prefix: the keys / values of the cached tokens come from their pages, the tile
            # table gives every query tile its sequence's key range and the position of its first query
            kf, vf = self._full_kv(meta.prefix, k, self._v_view(qkv), *kv_cache[i])
            att, _ = self.C.flash_attn_fwd(q, kf, vf, meta.prefix.tiles, scale, self.status)
            self.launches += 2
        else:
            att, _ = self.attention(q, k, self._v_view(qkv), cu)
        h2, _, x2 = self._o_proj_ln2(i, att.view(att.shape[0], -1), x, serving)
        if cfg.layer_is_moe(i):
            if (meta is not None and not meta.is_prefill and replay_ids is None and getattr(self.ep, "low_latency", False)
                    and x.shape[0] <= self.ep.rows and cfg.router_score == "softmax" and not cfg.shared_expert_ffn):
                return self.ep.moe_decode(self, i, x2, h2, record)
            y, _ = self.moe_forward(i, h2, replay_ids, record, keep=False, residual=x2, serving=serving)
            return y
        _, act = self._gated(h2, P[p + "mlp.gate_up.weight"], serving=serving)
        if cfg.post_norms:
            y = self.linear(act, P[p + "mlp.down.weight"], serving=serving)
            yn, _ = C.rmsnorm_fwd(y, None, P[p + "post_mlp_ln.weight"], cfg.rms_eps)
            self.launches += 2
            return yn.add_(x2)
        return self._row_parallel(act, P[p + "mlp.down.weight"], x2, serving)

    def _full_kv(self, prefix, k, v, kc, vc):
        """``PrefixInfo.full_kv`` in one launch for caches of the activations' type."""
        if kc.dtype != torch.bfloat16 or vc.dtype != torch.bfloat16:
            return prefix.full_kv(k, v, kc, vc)
        return self.C.gather_prefix_kv(k, v, kc, vc, prefix.pre_slots, prefix.pre_dst, prefix.new_dst, prefix.total, self.status)

    def _row_parallel(self, a, w, residual, serving=False):
        """``residual + a @ w^T`` for a row-parallel weight: under tensor parallelism the GEMM epilogue pushes the
        partial sums to the peers and the slots are added in rank order (one fused GEMM + all-reduce)."""
        if self.tp is not None:
            self.launches += 3
            return self.tp.linear_allreduce(a, w, residual=residual, gemm_status=self.status)
        if (serving and residual is not None and self.SMALL_T < a.shape[0] <= 64 and self.small_decode and not getattr(self, "mx", None)
                and a.is_contiguous() and w.shape[0] % 16 == 0 and w.shape[1] % 32 == 0):
            y = torch.empty_like(residual)  # the residual joins the sums before they are rounded
            self.C.small_gemv(a, None, 0.0, w, residual, y, self.status)
            self.launches += 1
            return y
        y = self.linear(a, w, serving=serving)
        return y.add_(residual) if residual is not None else y

    def _o_proj_ln2(self, i, att2, x, serving=False):
        """Attention output projection, residual add and the second RMSNorm: returns (h2, rstd2, x2)."""
        cfg, P, C = self.cfg, self.store.params, self.C
        p = f"layers.{i}."
        self.launches += 1
        if self.tp is not None:
            assert not cfg.post_norms, "models with sandwich norms run without tensor parallelism"
            x2 = self._row_parallel(att2, P[p + "attn.o.weight"], x, serving)
            h2, rstd2 = C.rmsnorm_fwd(x2, None, P[p + "ln2.weight"], cfg.rms_eps)
            return h2, rstd2, x2
        o = self.linear(att2, P[p + "attn.o.weight"], serving=serving)
        if cfg.post_norms:
            # sandwich norm (GLM-4 dense): the attention output is normalised before it joins the residual stream; the
            # backward's recompute picks the un-normalised output and its statistics up from here
            on, rstd_pa = C.rmsnorm_fwd(o, None, P[p + "post_attn_ln.weight"], cfg.rms_eps)
            self._post_attn_saved = (o, rstd_pa)
            self.launches += 1
            return C.rmsnorm_fwd(on, x, P[p + "ln2.weight"], cfg.rms_eps)
        return C.rmsnorm_fwd(o, x, P[p + "ln2.weight"], cfg.rms_eps)

    def _col_parallel_dgrad(self, dy, w):
        """Input gradient of a column-parallel weight: partial over the tensor-parallel ranks, so all-reduced."""
        if self.tp is not None:
            self.launches += 3
            return self.tp.linear_allreduce(dy, w, b_mn=True, gemm_status=self.status)
        return self.linear_dgrad(dy, w)

    SMALL_T = 8  # decode steps with at most this many rows take the weight-streaming kernels

    def _attn_small(self, i, x, positions, meta: InferMeta, kv_cache):
        """Attention half of a decode layer for at most 8 rows: returns ``x + attention(x)`` (RMSNorm folded into the
        qkv projection, residual folded into the output projection)."""
        cfg, P, C = self.cfg, self.store.params, self.C
        p = f"layers.{i}."
        T, dev = x.shape[0], x.device
        wqkv = P[p + "attn.qkv.weight"]
        qkv = torch.empty(T, wqkv.shape[0], dtype=torch.bfloat16, device=dev)
        C.small_gemv(x, P[p + "ln1.weight"], cfg.rms_eps, wqkv, None, qkv, self.status)
        if cfg.qkv_bias:
            qkv += P[p + "attn.qkv.bias"]
        kc, vc = kv_cache[i]
        if cfg.rope_scaling or cfg.rotary_dim:
            q, _, _, _ = C.qk_norm_rope_fwd_scaled(qkv, P.get(p + "attn.q_norm.weight"), P.get(p + "attn.k_norm.weight"),
                                                   positions, cfg.num_q_heads, cfg.num_kv_heads, cfg.rope_theta, cfg.rms_eps,
                                                   kc, vc, meta.slot_mapping, False, self._rope_table(),
                                                   cfg.rotary_dim or cfg.head_dim)
        else:
            q, _, _, _ = C.qk_norm_rope_fwd(qkv, P.get(p + "attn.q_norm.weight"), P.get(p + "attn.k_norm.weight"), positions,
                                            cfg.num_q_heads, cfg.num_kv_heads, cfg.rope_theta, cfg.rms_eps, kc, vc,
                                            meta.slot_mapping, False)
        att = torch.empty_like(q)
        splits = self._decode_splits(T, meta)
        need = T * cfg.num_q_heads * splits * 130
        if self._decode_scratch is None or self._decode_scratch.numel() < need:
            self._decode_scratch = torch.empty(need, dtype=torch.float32, device=dev)
        C.paged_decode_attention(q, kc, vc, meta.block_table, meta.seq_lens, att, self._decode_scratch, meta.page_size,
                                 splits, cfg.head_dim ** -0.5)
        x2 = torch.empty_like(x)
        C.small_gemv(att.view(T, -1), None, cfg.rms_eps, P[p + "attn.o.weight"], x, x2, self.status)
        self.launches += 4
        return x2

    def _layer_forward_small(self, i, x, positions, meta: InferMeta, kv_cache, record=None):
        """Decode forward of one layer for at most 8 rows: few light launches instead of 14-15, the two RMSNorms folded into the
        projections that consume them, SwiGLU and the combination into the experts', no expert permutation (per-expert pair lists)."""
        cfg, P, C = self.cfg, self.store.params, self.C
        p = f"layers.{i}."
        T, dev = x.shape[0], x.device
        x2 = self._attn_small(i, x, positions, meta, kv_cache)
        ln2 = P[p + "ln2.weight"]
        if cfg.layer_is_moe(i):
            E, K = cfg.num_experts, cfg.moe_top_k
            w1, w2 = P[p + "moe.w1"], P[p + "moe.w2"]
            I = w2.shape[2]
            ids = torch.empty(T, K, dtype=torch.int32, device=dev)
            w = torch.empty(T, K, dtype=torch.float32, device=dev)
            if C.moe_decode_fits(E, K, x.shape[1], I):
                plan = torch.empty(C.moe_decode_plan_size(E), dtype=torch.int32, device=dev)
                C.router_decode(x2, ln2, cfg.rms_eps, P[p + "moe.router.weight"], cfg.norm_topk_prob, ids, w, plan)
                if record is not None:
                    record.append(ids)
                act = torch.empty(T * K, I, dtype=torch.bfloat16, device=dev)
                C.moe_decode_up(x2, ln2, cfg.rms_eps, w1, plan, act, self.status)
                y = torch.empty_like(x2)
                C.moe_decode_down(act, w2, plan, x2, y, self.status)
                self.launches += 3
                return y
            lists = torch.empty(1 + E + E + 8 * E, dtype=torch.int32, device=dev)
            active, pc, pl = lists[:1 + E], lists[1 + E:1 + 2 * E], lists[1 + 2 * E:]
            logits = torch.empty(T, E, dtype=torch.float32, device=dev)
            C.small_gemv(x2, ln2, cfg.rms_eps, P[p + "moe.router.weight"], None, logits, self.status)
            C.router_small(logits, K, cfg.norm_topk_prob, ids, w, active, pc, pl)
            if record is not None:
                record.append(ids)
            max_active = min(E, T * K)
            act = torch.empty(T * K, w1.shape[1], dtype=torch.bfloat16, device=dev)  # gate | up; SwiGLU happens in the consumer
            C.moe_small_up(x2, ln2, cfg.rms_eps, w1, active, pc, pl, max_active, K, act, self.status)
            yp = torch.empty(T * K, x.shape[1], dtype=torch.bfloat16, device=dev)
            C.moe_small_down(act, w2, active, pc, pl, max_active, yp, self.status)
            if self._ident is None or self._ident.numel() < T * K:
                self._ident = torch.arange(self.SMALL_T * K, dtype=torch.int32, device=dev)
            y = C.moe_combine(yp, self._ident[:T * K], w, T, K, x2)
            self.launches += 5
            return y
        wgu = P[p + "mlp.gate_up.weight"]
        gu = torch.empty(T, wgu.shape[0], dtype=torch.bfloat16, device=dev)
        if wgu.numel() >= 24 << 20:  # (the split kernel reads 100 MB in 20 us, the one that folds the norm in takes 32)
            h2, _ = C.rmsnorm_fwd(x2, None, ln2, cfg.rms_eps)
            C.small_gemv(h2, None, 0.0, wgu, None, gu, self.status)
            self.launches += 1
        else:
            C.small_gemv(x2, ln2, cfg.rms_eps, wgu, None, gu, self.status)
        y = torch.empty_like(x)
        C.small_gemv(C.swiglu_fwd(gu), None, cfg.rms_eps, P[p + "mlp.down.weight"], x2, y, self.status)
        self.launches += 3
        return y

    def _decode_splits(self, B: int, meta: InferMeta) -> int:
        # Two CTAs per SM, but the splits of a sequence are a cluster that has to be placed as a whole: pairs always fit, of
        # larger ones some wait for a second round beyond 264 CTAs (us, 4 heads: 9 rows 7 splits 16.4, 8 24.2; 12 rows 5 16.2, 6 24.5; 18 rows 3 19.9, 4 26.9;
        # 24 rows 2 25.6, 3 34.1; 8 heads: 5 rows 6 19.2, 7 29.0). Clusters beyond the portable size of 8 fit only while they fill
        # about two thirds of the places (4 rows, 4 heads: 12 splits 19.5, 16 29.0).
        ctas = max(B * self.cfg.num_kv_heads, 1)
        splits = max(1, 296 // ctas)
        if splits > 2:
            splits = max(2, 264 // ctas)
        return splits if splits <= 8 else min(16, max(8, 192 // ctas))

    def _layer_acts(self, i, x, positions, cu, replay_ids=None, output: bool = False):
        """Forward of layer i that keeps what its backward needs: (activations, layer output or None). The values are those
        of ``layer_forward``, bit for bit: the same kernels, with the experts' rows padded for the weight gradients."""
        cfg, P, C = self.cfg, self.store.params, self.C
        p = f"layers.{i}."
        qkv = self._attn_qkv(i, x, positions, None, None)
        att, lse = self.attention(qkv[3], qkv[4], self._v_view(qkv[2]), cu)
        ln2 = h2, _, x2 = self._o_proj_ln2(i, att.view(att.shape[0], -1), x)
        post_attn = getattr(self, "_post_attn_saved", None) if cfg.post_norms else None
        self._post_attn_saved = None
        is_moe = cfg.layer_is_moe(i)
        assert not (is_moe and cfg.post_norms), "sandwich norms are wired for dense MLP layers"
        if is_moe:
            y, saved = self.moe_forward(i, h2, replay_ids, None, keep=True, residual=x2 if output else None)
            return LayerActs(qkv, att, lse, ln2, post_attn, saved, None), y
        gu, act = self._gated(h2, P[p + "mlp.gate_up.weight"], keep=True)
        y = None
        if output and cfg.post_norms:
            y, _ = C.rmsnorm_fwd(self.linear(act, P[p + "mlp.down.weight"]), None, P[p + "post_mlp_ln.weight"], cfg.rms_eps)
            y = y.add_(x2)
            self.launches += 1
        elif output:
            y = self._row_parallel(act, P[p + "mlp.down.weight"], x2)
        return LayerActs(qkv, att, lse, ln2, post_attn, None, (gu, act)), y

    # ------------------------------------------------------------------ activations kept between the two directions
    def _layer_act_bytes(self, i: int, T: int) -> int:
        """Bytes of one layer's ``LayerActs`` over T tokens (matrices; the per-row statistics are a hundredth of them)."""
        cfg = self.cfg
        H, D = cfg.hidden_size, cfg.head_dim
        cols = 3 * H + (3 * cfg.num_q_heads + 3 * cfg.num_kv_heads) * D + (H if cfg.post_norms else 0)  # h1, h2, x2; qkv and q, k; att; post_attn
        if not cfg.layer_is_moe(i):
            return 2 * T * (cols + 3 * cfg.ffn_hidden_size)
        rows = T * cfg.moe_top_k + cfg.num_experts * 63
        return 2 * T * cols + 2 * rows * (2 * H + 3 * cfg.moe_ffn_hidden_size) + 4 * T * cfg.num_experts

    def _pass_bytes(self, T: int, head_rows: int, chunk: int) -> int:
        """Bytes that a training pass holds whatever it keeps: the layers' inputs, the rows that are scored and their gradients, and the larger of
        a chunk of the head (logits, and the gradients of GRAD_CHUNKS) and a layer on its way back (its activations recomputed, their
        gradients, dQ in fp32; the shared expert's, which nobody keeps)."""
        cfg = self.cfg
        lo, hi = self.store.layer_range
        H = cfg.hidden_size
        layer = max((self._layer_act_bytes(i, T) for i in range(lo, hi)), default=0)
        work = 2 * layer + 4 * T * cfg.num_q_heads * cfg.head_dim + 12 * T * cfg.shared_expert_ffn
        head = (4 + 2 * self.GRAD_CHUNKS) * min(head_rows, chunk) * self.store.lm_head().shape[0] if head_rows else 0
        return 2 * T * H * (hi - lo + 4) + 4 * head_rows * H + max(work, head)

    def _room_for_acts(self, needed: int = 0) -> int:
        """Bytes a training pass that needs ``needed`` anyway may hold on to: what the device and the allocator's cache have free beyond a seventh
        of the device, the share that every part of this package that sizes itself by free memory leaves to activations, or beyond
        what the pass needs and a fourth of that share (for pieces that do not fit together), whichever is more."""
        if self.act_room is not None:
            return self.act_room
        free, total = torch.cuda.mem_get_info(self.dev)
        return free + torch.cuda.memory_reserved(self.dev) - torch.cuda.memory_allocated(self.dev) - max(total // 7, needed + total // 28)

    def _plan_acts(self, T: int, head_rows: int, chunk: int = 0) -> tuple[bool, int]:
        """(whether the logits are kept, first layer whose activations are). Where a pass exchanges data with other ranks
        everything is recomputed: they have to take the same steps, and how much is free is each rank's own. So it is for a
        subclass with layers of its own."""
        lo, hi = self.store.layer_range
        cls = type(self)
        if (self.ep is not None or self.tp is not None or self.cp_ctx is not None or getattr(self.store, "begin_pass", None) is not None
                or any(getattr(cls, f) is not getattr(B200Qwen3, f) for f in ("layer_forward", "layer_backward", "forward_hidden", "layers_backward"))):
            return False, hi
        head = 4 * head_rows * self.store.lm_head().shape[0] if head_rows and not self.recompute_logits else 0
        first = min(lo + self.recompute_layers, hi)
        if first == hi and not head:
            return False, hi
        return plan_kept(self._room_for_acts(self._pass_bytes(T, head_rows, chunk)), head, [self._layer_act_bytes(i, T) for i in range(first, hi)], first)

    def _forward_keeping(self, keep_from: int, inputs: list, acts: dict, *args, **kw):
        """``forward_hidden`` that keeps the layers' inputs, and the activations of the layers from ``keep_from`` on. Where memory runs out for
        those after all (whoever shares the device may have taken some), it starts again and keeps none."""
        if keep_from < self.store.layer_range[1]:
            try:
                return self.forward_hidden(*args, save_inputs=inputs, save_acts=acts, keep_from=keep_from, **kw)
            except RuntimeError as e:
                if not _out_of_memory(e):
                    raise
            inputs.clear()
            acts.clear()
        return self.forward_hidden(*args, save_inputs=inputs, **kw)

    # ``chunk`` rows of fp32 logits are what --log-probs-chunk-size lets the head hold at a time. In the same bytes are
    #  - the bf16 gradients of twice as many rows, which therefore go through the head's gradient together, whether their logits were kept or
    #    are recomputed chunk by chunk (each pass over that gradient, 151936 x 2048 in fp32, reads and writes 2.5 GB);
    #  - what the fused product leaves of 32 times as many (16 bytes for 128 columns); more than 16384 rows gain nothing.
    GRAD_CHUNKS, SCORE_CHUNKS, SCORE_ROWS = 2, 32, 16384

    def layer_backward(self, i, x, dy, positions, cu, max_seqlen, replay_ids=None, acts: Optional[LayerActs] = None):
        """Back-propagate ``dy`` through layer i, from the activations its forward kept or else recomputed from its input
        ``x``; returns dx."""
        cfg, P, G, C = self.cfg, self.store.params, self.store.grads, self.C
        p = f"layers.{i}."
        if acts is None:
            acts, _ = self._layer_acts(i, x, positions, cu, replay_ids)
        h1, rstd1, qkv, q, k, qr, kr = acts.qkv
        v, att, lse = self._v_view(qkv), acts.att, acts.lse
        att2 = att.view(att.shape[0], -1)
        h2, rstd2, x2 = acts.ln2
        post_attn, saved = acts.post_attn, acts.moe
        is_moe = cfg.layer_is_moe(i)
        if not is_moe:
            gu, act = acts.mlp
        # ---- backward: MLP / MoE
        if is_moe:
            dh2 = self.moe_backward(i, h2, dy, saved)
            del saved
        else:
            dyy = dy
            if cfg.post_norms:  # through the norm on the MLP output (its input is recomputed)
                y = self.linear(act, P[p + "mlp.down.weight"])
                _, rstd_pm = C.rmsnorm_fwd(y, None, P[p + "post_mlp_ln.weight"], cfg.rms_eps)
                dyy = C.rmsnorm_bwd(dy, y, P[p + "post_mlp_ln.weight"], rstd_pm, None, G[p + "post_mlp_ln.weight"], True)
                self.launches += 3
            dact = self.linear_dgrad(dyy, P[p + "mlp.down.weight"])
            self.linear_wgrad(dyy, act, G[p + "mlp.down.weight"])
            dgu = C.swiglu_bwd(dact, gu)
            dh2 = self._col_parallel_dgrad(dgu, P[p + "mlp.gate_up.weight"])
            self.linear_wgrad(dgu, h2, G[p + "mlp.gate_up.weight"])
            self.launches += 1
        # ---- ln2 (residual gradient dy flows straight through x2)
        dx2 = C.rmsnorm_bwd(dh2, x2, P[p + "ln2.weight"], rstd2, dy, G[p + "ln2.weight"], True)
        self.launches += 2
        # ---- attention output projection
        do = dx2
        if cfg.post_norms:  # through the norm on the attention output
            o, rstd_pa = post_attn
            do = C.rmsnorm_bwd(dx2, o, P[p + "post_attn_ln.weight"], rstd_pa, None, G[p + "post_attn_ln.weight"], True)
            self.launches += 1
        datt = self.linear_dgrad(do, P[p + "attn.o.weight"])
        self.linear_wgrad(do, att2, G[p + "attn.o.weight"])
        dq, dk, dv = self.attention_backward(q, k, v, att, datt.view_as(att), lse, cu)
        if cfg.rope_scaling or cfg.rotary_dim:
            dqkv = C.qk_norm_rope_bwd_scaled(dq, dk, dv, qkv, P.get(p + "attn.q_norm.weight"),
                                             P.get(p + "attn.k_norm.weight"), positions, qr, kr, G.get(p + "attn.q_norm.weight"),
                                             G.get(p + "attn.k_norm.weight"), cfg.num_q_heads, cfg.num_kv_heads, cfg.rope_theta,
                                             self._rope_table(), cfg.rotary_dim or cfg.head_dim)
        else:
            dqkv = C.qk_norm_rope_bwd(dq, dk, dv, qkv, P.get(p + "attn.q_norm.weight"),
                                      P.get(p + "attn.k_norm.weight"), positions, qr, kr, G.get(p + "attn.q_norm.weight"),
                                      G.get(p + "attn.k_norm.weight"), cfg.num_q_heads, cfg.num_kv_heads, cfg.rope_theta)
        self.launches += 1
        if cfg.qkv_bias:
            G[p + "attn.qkv.bias"].add_(dqkv.float().sum(0).to(G[p + "attn.qkv.bias"].dtype))
        dh1 = self._col_parallel_dgrad(dqkv, P[p + "attn.qkv.weight"])
        self.linear_wgrad(dqkv, h1, G[p + "attn.qkv.weight"])
        dx = C.rmsnorm_bwd(dh1, x, P[p + "ln1.weight"], rstd1, dx2, G[p + "ln1.weight"], True)
        self.launches += 2
        return dx

    # ------------------------------------------------------------------ whole-model passes
    @torch.no_grad()
    def forward_hidden(self, tokens, positions, cu_seqlens, meta: Optional[InferMeta] = None, kv_cache=None,
                       replay: Optional[torch.Tensor] = None, record: Optional[list] = None, max_seqlen: int = 0,
                       save_inputs: Optional[list] = None, x_in: Optional[torch.Tensor] = None, save_acts: Optional[dict] = None,
                       keep_from: int = 0):
        """Runs this pipeline stage's layers (all of them without pipeline parallelism). The first stage embeds
        ``tokens``, later stages continue from ``x_in``; every stage but the last returns the raw hidden states that
        the next stage consumes, the last one applies the final norm. ``save_acts`` receives the activations of the layers
        from ``keep_from`` on, for ``layer_backward``."""
        cfg, P, C = self.cfg, self.store.params, self.C
        begin = getattr(self.store, "begin_pass", None)
        if begin is not None:
            begin()  # a sharded store materialises units per pass
        lo, hi = self.store.layer_range
        x = P["embed.weight"][tokens.long()] if self.store.is_first_stage else x_in
        if not max_seqlen and cu_seqlens is not None:
            max_seqlen = int((cu_seqlens[1:] - cu_seqlens[:-1]).max().item())
        moe_idx = sum(cfg.layer_is_moe(j) for j in range(lo))  # replay columns are indexed over the whole model
        for i in range(lo, hi):
            if save_inputs is not None:
                save_inputs.append(x)
            rid = None
            if cfg.layer_is_moe(i):
                if replay is not None:
                    rid = replay[:, moe_idx]
                moe_idx += 1
            if save_acts is not None and i >= keep_from:
                save_acts[i], x = self._layer_acts(i, x, positions, cu_seqlens, rid, output=True)
                continue
            x = self.layer_forward(i, x, positions, cu_seqlens, max_seqlen, meta, kv_cache, rid, record)
        if save_inputs is not None:
            save_inputs.append(x)
        if not self.store.is_last_stage:
            return x
        h, _ = C.rmsnorm_fwd(x, None, P["final_norm.weight"], cfg.rms_eps)
        self.launches += 1
        return h

    @torch.no_grad()
    def _trunk_backward(self, inputs, x_last, h, rows, dhr, tokens, positions, cu_seqlens, max_seqlen, replay, acts=None):
        """Back-propagate ``dhr`` (gradient wrt the final-normed hidden rows) through the norm, layers and embedding."""
        cfg, P, G, C = self.cfg, self.store.params, self.store.grads, self.C
        dh = torch.zeros_like(h)
        dh.index_add_(0, rows, dhr.to(h.dtype))
        _, rstd = C.rmsnorm_fwd(x_last, None, P["final_norm.weight"], cfg.rms_eps)
        dx = C.rmsnorm_bwd(dh, x_last, P["final_norm.weight"], rstd, None, G["final_norm.weight"], True)
        self.launches += 3
        del dh
        return self.layers_backward(inputs, dx, tokens, positions, cu_seqlens, max_seqlen, replay, **(dict(acts=acts) if acts else {}))

    @torch.no_grad()
    def layers_backward(self, inputs, dx, tokens, positions, cu_seqlens, max_seqlen, replay, acts: Optional[dict] = None):
        """Backward through this stage's layers: ``inputs[j]`` is the saved input of local layer ``j``, ``acts`` the activations
        of the layers that kept them (given back as they are used), ``dx`` the gradient of the stage's output. Returns the gradient of the stage's input (on the first stage it has been
        added into the embedding gradient) and keeps it in ``self.last_dx_in``."""
        cfg, G = self.cfg, self.store.grads
        lo, hi = self.store.layer_range
        moe_layers = [i for i in range(cfg.num_layers) if cfg.layer_is_moe(i)]
        for i in reversed(range(lo, hi)):
            rid = replay[:, moe_layers.index(i)] if (replay is not None and cfg.layer_is_moe(i)) else None
            kw = dict(acts=acts.pop(i)) if acts and i in acts else {}
            dx = self.layer_backward(i, inputs[i - lo], dx, positions, cu_seqlens, max_seqlen, rid, **kw)
            del kw
            inputs[i - lo] = None
        if self.store.is_first_stage:
            G["embed.weight"].index_add_(0, tokens.long(), dx.to(G["embed.weight"].dtype))
        self.last_dx_in = dx
        return dx

    def forward_backward_hidden(self, tokens, positions, cu_seqlens, row_index, head_fn, replay=None, max_seqlen: int = 0,
                                x_in: Optional[torch.Tensor] = None):
        """Generic head: ``head_fn(hidden_rows_fp32_leaf) -> (loss, metrics)`` (e.g. a value head); the trunk is
        back-propagated with the gradient autograd computes for the hidden rows."""
        assert self.store.grads, "allocate_grads() must be called before training"
        if not max_seqlen:
            max_seqlen = int((cu_seqlens[1:] - cu_seqlens[:-1]).max().item())
        inputs: list = []
        acts: dict = {}
        keep_from = self._plan_acts(positions.shape[0], 0)[1]
        h = self._forward_keeping(keep_from, inputs, acts, tokens, positions, cu_seqlens, replay=replay, max_seqlen=max_seqlen, x_in=x_in)
        x_last = inputs.pop()
        rows = row_index.long()
        leaf = h[rows].float().detach().requires_grad_(True)
        with torch.enable_grad():
            loss, metrics = head_fn(leaf)
            loss.backward()
        self._trunk_backward(inputs, x_last, h, rows, leaf.grad, tokens, positions, cu_seqlens, max_seqlen, replay, acts)
        return loss.detach(), metrics

    @torch.no_grad()
    def logits(self, hidden_rows, out_dtype=torch.float32, serving=True):
        return self.linear(hidden_rows.contiguous(), self.store.lm_head(), out_dtype, serving)

    # From this many rows of the head on the scores leave with its product (csrc/gemm.cu). The two ways add a row's exponentials in different
    # orders, so the vocabulary alone decides: how many rows a pass has, scores at a time or keeps must not show in a row's score. us for
    # logits and kernel / fused, 2048 columns: 32000 rows with 8 tokens 50 / 50, 33 52 / 46, 512 89 / 75, 8192 1125 / 751; 4096 rows
    # with one token 26 / 40, 129 32 / 40, 512 38 / 38, 8192 241 / 144; 151936 rows with one token 254 / 216.
    SCORE_VOCAB = 32000

    def _fused_scores(self, vocab: int) -> bool:
        return vocab >= self.SCORE_VOCAB and type(self).logits is B200Qwen3.logits

    def _logits_again(self, hidden_rows, w, whole_k: bool):
        """Logits for a backward that did not keep them: the values of the forward, which fused scores sum over whole rows of the head."""
        if not whole_k:
            return self.logits(hidden_rows, serving=False)
        out = torch.empty(hidden_rows.shape[0], w.shape[0], dtype=torch.float32, device=hidden_rows.device)
        self.C.gemm(hidden_rows, w, out, False, False, False, 0, self.status, whole_k=True)
        self.launches += 1
        return out

    @torch.no_grad()
    def logprobs_entropy(self, hidden_rows, targets, inv_temp: float, chunk: int = 0, keep_stats: bool = False, keep_logits: Optional[list] = None):
        C = self.C
        chunk = chunk or self.lm_chunk
        n, W = hidden_rows.shape[0], self.store.lm_head()
        tg = targets.to(torch.int32).contiguous()
        fused = self._fused_scores(W.shape[0])
        if fused and keep_logits is None:  # no logits at all
            chunk = max(chunk, min(self.SCORE_CHUNKS * chunk, self.SCORE_ROWS))
        out = []
        for a in range(0, n, chunk):
            b = min(a + chunk, n)
            if fused:
                lg = torch.empty(b - a, W.shape[0], dtype=torch.float32, device=self.dev) if keep_logits is not None else None
                out.append(C.score_rows(hidden_rows[a:b].contiguous(), W, tg[a:b], inv_temp, lg, self.status))
                self.launches += 2
            else:
                lg = self.logits(hidden_rows[a:b], serving=False)
                out.append(C.logprob_entropy_fwd(lg, tg[a:b], inv_temp))
                self.launches += 1
            if keep_logits is not None:
                keep_logits.append(lg)
        if not out:
            out.append([torch.empty(0, dtype=torch.float32, device=self.dev)] * 4)
        lp, ent, lse, px = out[0] if len(out) == 1 else (torch.cat(t) for t in zip(*out))
        return (lp, ent, lse, px) if keep_stats else (lp, ent)

    @torch.no_grad()
    def forward_logprobs(self, tokens, positions, cu_seqlens, row_index, targets, inv_temp, replay=None, record=None,
                         max_seqlen: int = 0, x_in: Optional[torch.Tensor] = None):
        h = self.forward_hidden(tokens, positions, cu_seqlens, replay=replay, record=record, max_seqlen=max_seqlen, x_in=x_in)
        return self.logprobs_entropy(h[row_index.long()], targets, inv_temp)

    def forward_backward(self, tokens, positions, cu_seqlens, row_index, targets, inv_temp, loss_fn, replay=None,
                         max_seqlen: int = 0, chunk: int = 0, x_in: Optional[torch.Tensor] = None):
        """One micro-batch: forward, ``loss_fn(logprobs, entropy) -> (loss, metrics)``, backward into the grad buffers.
        On the last pipeline stage ``x_in`` is the activation received from the previous stage and ``self.last_dx_in``
        afterwards holds the gradient to send back."""
        cfg, P, G, C = self.cfg, self.store.params, self.store.grads, self.C
        assert G, "allocate_grads() must be called before training"
        chunk = chunk or self.lm_chunk
        if not max_seqlen:
            max_seqlen = int((cu_seqlens[1:] - cu_seqlens[:-1]).max().item())
        inputs: list[torch.Tensor] = []
        acts: dict = {}
        keep_head, keep_from = self._plan_acts(positions.shape[0], row_index.shape[0], chunk)
        h = self._forward_keeping(keep_from, inputs, acts, tokens, positions, cu_seqlens, replay=replay, max_seqlen=max_seqlen, x_in=x_in)
        x_last = inputs.pop()  # input of the final norm
        rows = row_index.long()
        hr = h[rows].contiguous()
        tg = targets.to(torch.int32).contiguous()
        kept: Optional[list] = [] if keep_head else None
        stats = None
        if keep_head:
            try:
                stats = self.logprobs_entropy(hr, tg, inv_temp, chunk, keep_stats=True, keep_logits=kept)
            except RuntimeError as e:
                if not _out_of_memory(e):
                    raise
                kept.clear()
        if stats is None:
            kept = None
            stats = self.logprobs_entropy(hr, tg, inv_temp, chunk, keep_stats=True)
        lp, ent, lse, px = stats
        lp_leaf, ent_leaf = lp.detach().requires_grad_(True), ent.detach().requires_grad_(True)
        with torch.enable_grad():
            loss, metrics = loss_fn(lp_leaf, ent_leaf)
            grads = torch.autograd.grad(loss, (lp_leaf, ent_leaf), allow_unused=True)
        dlp = grads[0].float().contiguous() if grads[0] is not None else torch.zeros_like(lp)
        dent = grads[1].float().contiguous() if grads[1] is not None else None
        with torch.no_grad():
            # ---- LM head backward, chunked: the logits, kept or recomputed, become dlogits
            W = self.store.lm_head()
            gW = G["embed.weight"] if cfg.tie_embeddings else G["lm_head.weight"]
            dhr = torch.empty_like(hr)
            whole_k = self._fused_scores(W.shape[0])
            n, step = hr.shape[0], self.GRAD_CHUNKS * chunk
            for g0 in range(0, n, step):
                g1 = min(g0 + step, n)
                dl = torch.empty(g1 - g0, W.shape[0], dtype=torch.bfloat16, device=hr.device)
                for a in range(g0, g1, chunk):
                    b = min(a + chunk, g1)
                    lg = kept[a // chunk] if kept is not None else self._logits_again(hr[a:b], W, whole_k)
                    C.logprob_entropy_bwd(lg, tg[a:b], lse[a:b].contiguous(), px[a:b].contiguous(), dlp[a:b].contiguous(),
                                          dent[a:b].contiguous() if dent is not None else None, inv_temp, dl[a - g0:b - g0])
                    del lg
                    if kept is not None:
                        kept[a // chunk] = None
                    self.launches += 1
                self._gemm(dl, W, dhr[g0:g1], False, True)
                self.linear_wgrad(dl, hr[g0:g1], gW)
                del dl
            self._trunk_backward(inputs, x_last, h, rows, dhr, tokens, positions, cu_seqlens, max_seqlen, replay, acts)
        return loss.detach(), metrics, lp.detach(), ent.detach()
