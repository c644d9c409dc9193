"""Orders of memory accesses that no run shows to be wrong reliably, so the sources are read instead.

The factorization's copies: its buffers come from a stream-ordered pool and are used on the
handle's non-blocking stream, which does not follow the legacy stream: a synchronous copy or set
there would run beside the allocation it writes to and the kernels that read it.

The MAS apply that starts beside the coarse sums: it has not waited for the kernel before them itself, so
what that kernel and earlier ones wrote is read past L1."""

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


@pytest.mark.parametrize("form", ["mas_apply_warps", "mas_apply_rows"])
def test_early_apply_reads_past_l1(form):
    text = _code((CSRC / "mas_apply.cu").read_text())
    start = text.index(f"bool {form}(")
    body = text[start:text.index("return true;", start)]
    assert "solve_done(st)" in body and "st->done" not in body
    assert re.findall(r"bool solve_done\(.*?stop = __ldcg\(&st->done\);", text, flags=re.S)
    assert "__ldcg(in + " in body
    assert re.findall(r"\bin\[", body) == []
