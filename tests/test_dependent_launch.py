"""Kernels that are launched while their predecessor runs (csrc/pdl.cuh). From the sources: tensor memory is allocated before
dependents are let in; otherwise a dependent on the same SM may take it and keep it until this kernel ends. On the GPU: each reads what
the one before it on the stream wrote, be that an ordinary kernel, a dependent one, a memset or a node of a captured graph."""
import re
from pathlib import Path

import pytest
import torch

import miles_b200

CSRC = Path(miles_b200.__file__).resolve().parent / "csrc"
LET_IN = ("pdl_enter()", "pdl_let_dependents_in()")
ALLOC = re.compile(r"\btmem_alloc\w*\(")  # by one CTA, or by a pair


def _kernels(path):
    """(name, body) of every kernel of a file; bodies are found by their braces, comments are dropped."""
    text = re.sub(r"//[^\n]*", "", path.read_text())
    for m in re.finditer(r"__global__", text):
        brace = text.index("{", text.index(")", text.index("(", m.end())) if "__launch_bounds__" not in text[m.end():m.end() + 40]
                           else text.index("(", text.index(")", text.index("__launch_bounds__", m.end())) + 1))
        at, depth = brace, 0
        while True:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
            if depth == 0:
                break
        yield re.findall(r"(\w+)\s*\(", text[m.end():brace].replace("__launch_bounds__", ""))[-1], text[brace:at]


@pytest.mark.parametrize("path", sorted(CSRC.glob("*.cu")), ids=lambda p: p.name)
def test_tensor_memory_is_allocated_before_dependents_are_let_in(path):
    for name, body in _kernels(path):
        lets = [body.index(w) for w in LET_IN if w in body]
        allocs = [m.start() for m in ALLOC.finditer(body)]
        if lets and allocs:
            assert max(allocs) < min(lets), f"{path.name}: {name}"


def test_the_search_sees_the_kernels_it_is_about():
    both = {name: {body[m.start():m.end() - 1] for m in ALLOC.finditer(body)} for path in CSRC.glob("*.cu") for name, body in _kernels(path)
            if any(w in body for w in LET_IN)}
    assert {"fa_fwd_kernel", "fa_fwd_pair_kernel", "gemm_bf16_kernel", "gemm_skinny_kernel"} <= {name for name, allocs in both.items() if allocs}
    assert both["gemm_bf16_kernel"] == {"tmem_alloc", "tmem_alloc_pair"}


def _chain(ext, b, src, after):
    """Ordinary, dependent and memset steps by turns, each with the result of the one before; returns what they wrote."""
    b["x"].copy_(src); after()
    h, _ = ext.rmsnorm_fwd(b["x"], None, b["g"], 1e-6); after()
    b["sum"].zero_(); after()
    ext.gemm(h, b["w"], b["sum"], False, False, True, 0, b["st"]); after()
    act = ext.swiglu_fwd(b["sum"]); after()
    ext.gemm(act[:96], b["v"], b["few"], False, False, False, 0, b["st"]); after()
    b["few"].mul_(2); after()
    h2, _ = ext.rmsnorm_fwd(b["few"], None, b["g"], 1e-6); after()
    ext.small_gemv(h2[:5], None, 0.0, b["v2"], None, b["logits"], b["st"]); after()
    ext.router_small(b["logits"], 8, True, b["ids"], b["weights"], b["active"], b["count"], b["lists"]); after()
    b["x"].zero_(); after()
    return h, b["sum"], act, b["few"], h2, b["logits"], b["ids"], b["weights"], b["count"]


@pytest.mark.gpu
@pytest.mark.parametrize("graph", [False, True])
def test_each_step_reads_what_the_one_before_wrote(graph):
    from miles_b200.ops import _ext

    ext = _ext.load(required=True)
    g = torch.Generator("cuda").manual_seed(1)
    bf = dict(dtype=torch.bfloat16, device="cuda")
    T, H, E = 2048, 2048, 128
    b = dict(x=torch.empty(T, H, **bf), g=torch.randn(H, generator=g, device="cuda").bfloat16(), st=torch.zeros(1, dtype=torch.int32, device="cuda"),
             w=torch.randn(2 * H, H, generator=g, device="cuda").bfloat16(), v=torch.randn(H, H, generator=g, device="cuda").bfloat16(),
             v2=torch.randn(E, H, generator=g, device="cuda").bfloat16(), sum=torch.empty(T, 2 * H, **bf), few=torch.empty(96, H, **bf),
             logits=torch.empty(5, E, device="cuda"), weights=torch.empty(5, 8, device="cuda"))
    b.update({k: torch.empty(n, dtype=torch.int32, device="cuda") for k, n in (("ids", (5, 8)), ("active", 1 + E), ("count", E), ("lists", 8 * E))})
    srcs = [torch.randn(T, H, generator=g, device="cuda").bfloat16() for _ in range(6)]
    want = [[t.clone() for t in _chain(ext, b, s, torch.cuda.synchronize)] for s in srcs]
    assert not torch.equal(want[0][-2], want[1][-2])
    if graph:
        still = srcs[0].clone()
        _chain(ext, b, still, lambda: None)
        torch.cuda.synchronize()
        cg = torch.cuda.CUDAGraph()
        with torch.cuda.graph(cg):
            out = _chain(ext, b, still, lambda: None)
        got = []
        for s in srcs * 4:
            still.copy_(s)
            cg.replay()
            got.append([t.clone() for t in out])
        del cg
    else:
        got = [[t.clone() for t in _chain(ext, b, s, lambda: None)] for s in srcs * 4]
    assert b["st"].item() == 0
    for i, outs in enumerate(got):
        assert all(torch.equal(a, w) for a, w in zip(outs, want[i % len(srcs)])), i
