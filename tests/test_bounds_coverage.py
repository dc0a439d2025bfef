"""What the documents say of the bounds-checked build: the loads and stores of
global memory in these functions go through craw_in_bounds. Each names the
accesses, in order, that a check has to stand before (since the access before
it, or the function's start)."""
import re
from pathlib import Path

import pytest

KERNELS = Path(__file__).resolve().parent.parent / "libcraw_gb300" / "csrc" / "kernels"

# (file, the function's head, its accesses)
CASES = [
    ("develop_walk.cuh", r"uint2 load\(const char \*row\) const", ["walk_ld4("]),
    ("develop_walk.cuh", r"void store\(char \*d, const void \*base", ["reinterpret_cast<float4 *>(p + i) ="]),
    ("develop_walk.cuh", r"void store\(char \*at, size_t pitch, int f, int r", ["p[0] = make_float2"]),
    ("develop_walk.cuh", r"void quarter\(int r, bool last", ["craw_store_rgba"]),
    ("develop_walk.cuh", r"void quarter\(int y, bool last", ["craw_store_rgba"]),
    ("develop_walk.cuh", r"void ring_walk\(", ["walk_ld("]),
    ("develop_walk.cuh", r"void rcd_walk\(", ["walk_ld("]),
    ("denoise_history.cuh", r"void temporal_walk\(",
     ["__ldg", "reinterpret_cast<float2 *>(at) =", "reinterpret_cast<float2 *>(lr)[qx + j] ="]),
    ("denoise_history.cuh", r"void history_tile\(",
     ["*reinterpret_cast<const float4 *>(", "__ldg", "reinterpret_cast<uint4 *>(dr) ="]),
    ("chroma.cu", r"ChromaTexel texel\(", ["craw_load_rgb"]),
    ("chroma.cu", r"void fetch\(int y, int ylim\)", ["cp.async.cg"]),
    ("highlight.cu", r"k_hl_level0\(", ["__ldg", "reinterpret_cast<float4 *>(io.levels)"]),
    ("highlight.cu", r"k_hl_fill\(", ["__ldg", "reinterpret_cast<__half2 *>((char *)io.dst"]),
]


def body(text, head):
    start = re.search(head, text).start()
    at = text.index("{", text.index(")", start))
    depth, end = 1, at + 1
    while depth:
        depth += {"{": 1, "}": -1}.get(text[end], 0)
        end += 1
    return text[at:end]


@pytest.mark.parametrize("file,head,accesses", CASES)
def test_checked(file, head, accesses):
    text = body(re.sub(r"/\*.*?\*/", " ", (KERNELS / file).read_text(), flags=re.S), head)
    at = 0
    for a in accesses:
        nxt = text.index(a, at)
        assert "craw_in_bounds(" in text[at:nxt], f"{file}: {a}"
        at = nxt + len(a)
