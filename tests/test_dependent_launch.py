"""Order inside kernels that are launched while their predecessor runs (csrc/pdl.cuh), read from the sources: tensor memory is
allocated before dependents are let in. Otherwise a dependent on the same SM may take it and keep it until this kernel ends."""
import re
from pathlib import Path

import pytest

import miles_b200

CSRC = Path(miles_b200.__file__).resolve().parent / "csrc"
LET_IN = ("pdl_enter()", "pdl_let_dependents_in()")


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
        if lets and "tmem_alloc(" in body:
            assert body.rindex("tmem_alloc(") < min(lets), f"{path.name}: {name}"


def test_the_search_sees_the_kernels_it_is_about():
    both = {name for path in CSRC.glob("*.cu") for name, body in _kernels(path) if "tmem_alloc(" in body and any(w in body for w in LET_IN)}
    assert {"fa_fwd_kernel", "gemm_bf16_kernel", "gemm_skinny_kernel"} <= both
