"""A launch that the runtime refuses is reported once: whoever raises it takes it off the runtime, where the next call would find it again."""
from pathlib import Path

import pytest

import miles_b200

CSRC = Path(miles_b200.__file__).resolve().parent / "csrc"


@pytest.mark.parametrize("name", ["attention_bwd.cu", "attention_fwd.cu", "decode_moe.cu", "decode_stream.cu", "gemm.cu", "gemm_mx.cu", "gemm_skinny.cu"])
def test_refused_launches_are_taken_off_the_runtime(name):
    lines = (CSRC / name).read_text().splitlines()
    said = [i for i, line in enumerate(lines) if "launch failed" in line]
    assert said
    for i in said:
        assert any("cudaGetLastError()" in line for line in lines[i - 2:i]), f"{name}:{i + 1}"
