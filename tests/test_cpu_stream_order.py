"""Order of the factorization's copies. Its buffers come from a stream-ordered pool and are used on the
handle's non-blocking stream, which does not follow the legacy stream: a synchronous copy or set
there would run beside the allocation it writes to and the kernels that read it. Such a race shows on
no run that can be relied on, so the sources are read instead."""

from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "polysolve_b200" / "csrc"


def _code(text: str) -> str:
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


def _factorize_body() -> str:
    text = _code((CSRC / "mas_capi.cpp").read_text())
    start = text.index("void factorize(int n_")
    return text[start:text.index("void require_factorized", start)]


@pytest.mark.parametrize("name", ["mas_bsr.cu", "mas_build.cu", "factorize"])
def test_factorization_copies_follow_the_stream(name):
    text = _factorize_body() if name == "factorize" else _code((CSRC / name).read_text())
    assert re.findall(r"\bcudaMem(?:cpy|set)(?:2D|3D)?\s*\(", text) == []
    # Every launch names its stream (the fourth launch argument).
    for launch in re.findall(r"<<<(.*?)>>>", text, flags=re.S):
        assert re.search(r",\s*(s|stream)\s*$", launch), launch
