"""A kernel that may start before the one ahead of it on the stream has ended
(craw_launch_early) reads what that one writes by ordinary loads: the
read-only path (__ldg, ld.global.nc, a const __restrict__ pointer) promises
that nothing writes the data while the kernel lives. The sources of those
kernels are read for it: each read-only load that is left must name a buffer
that was complete before the chain's first plain launch."""
import re
from pathlib import Path

import pytest

KERNELS = Path(__file__).resolve().parent.parent / "libcraw_gb300" / "csrc" / "kernels"

# File: what a read-only load there may read (the caller's mosaic; in the
# highlights' chain the mosaic its first, plain launch waits for).
EARLY = {
    "develop_walk.cuh": None,
    "chroma.cu": None,
    "awb.cu": None,
    "noise.cu": r"\bp\b",                     # plane_quad: the mosaic's row
    "denoise_history.cuh": r"io\.src|\b(src|lvl|var)\b",
    "highlight.cu": r"io\.src|\brow\b",
}


def code(name):
    text = (KERNELS / name).read_text()
    return re.sub(r"/\*.*?\*/|//[^\n]*", " ", text, flags=re.S)


@pytest.mark.parametrize("name", list(EARLY))
def test_read_only_loads(name):
    text, ok = code(name), EARLY[name]
    assert "ld.global.nc" not in text
    assert not re.search(r"\bconst\s+\w+\s*\*\s*__restrict__", text)
    for m in re.finditer(r"__ldg\(", text):
        depth, end = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[end], 0)
            end += 1
        arg = text[m.end():end - 1]
        assert ok and re.search(ok, arg), f"{name}: __ldg({arg})"
