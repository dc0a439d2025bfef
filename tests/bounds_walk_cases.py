"""Frames developed through whichever build of libcraw.so this process loaded
(CRAW_LIBRARY), as bounds_cases.py, over the kernels of the walking warps and
of the denoise with a history (packed 2x8: the averaged planes, their tiles by
TMA and by plain loads): every output layout, the kept intermediate, FP16
storage, chroma and highlights, at the smallest frames and at sizes whose
strips, segments and tiles end short. `python bounds_walk_cases.py OUT.npz`
writes each case's output and the kernel error bits of its pipeline."""
from __future__ import annotations

import sys
from pathlib import Path

import numpy as np

sys.path.insert(0, str(Path(__file__).resolve().parent))
sys.path.insert(0, str(Path(__file__).resolve().parent.parent))

import libcraw_gb300 as L  # noqa: E402
from libcraw_gb300 import workloads as W  # noqa: E402
from gpu_util import develop  # noqa: E402

AWB, KEEP = L.FLAG_AWB_HISTOGRAM, L.FLAG_KEEP_INTERMEDIATE
NLM, TMP, CHR, HL = (L.FLAG_DENOISE, L.FLAG_TEMPORAL_DENOISE, L.FLAG_CHROMA_DENOISE,
                     L.FLAG_HIGHLIGHT_RECONSTRUCTION)
SIZES = [(8, 8), (10, 14), (122, 34), (126, 18), (242, 70), (1030, 262)]

# (name, w, h, debayer, pipeline flags, frames)
CASES = [(f"{n}_{w}x{h}", w, h, d, f, 1) for w, h in SIZES
         for n, d, f in (("bilinear", L.DEBAYER_BILINEAR, AWB), ("mhc", L.DEBAYER_MHC, AWB),
                         ("mhc_keep", L.DEBAYER_MHC, AWB | KEEP), ("mhc_plain", L.DEBAYER_MHC, 0),
                         ("rcd", L.DEBAYER_RCD, AWB), ("hl", L.DEBAYER_BILINEAR, HL))]
CASES += [(f"history_{w}x{h}", w, h, L.DEBAYER_BILINEAR, NLM | TMP | AWB, 3) for w, h in
          [(12, 12), (62, 34), (66, 30), (130, 62), (518, 262)]]
CASES += [(f"chroma_{w}x{h}", w, h, L.DEBAYER_MHC, NLM | CHR | AWB, 1) for w, h in [(20, 20), (122, 34), (518, 262)]]


def run_cases() -> dict[str, np.ndarray]:
    out: dict[str, np.ndarray] = {}
    prof = W.make_profile()
    L.debug_force_denoise_shape(L.DN_SHAPES.index("2x8 f32x2"))
    with L.Context(0) as ctx:
        for name, w, h, deb, flags, nfr in CASES:
            fp = L.frame_params(prof, noise_override=W.noise_model(4.0, 40.0), denoise_strength=1.0,
                                denoise_temporal_strength=0.8, denoise_chroma_strength=0.5,
                                flags=L.FRAME_HIGHLIGHT_RECONSTRUCTION if flags & HL else 0)
            for fmt, storage, tma in ((L.FORMAT_RGBA32F, L.STORAGE_FP32, True), (L.FORMAT_RGB32F, L.STORAGE_FP32, False),
                                      (L.FORMAT_RGBA16F, L.STORAGE_FP16, True)):
                L.debug_denoise_tma(tma)
                pp = L.pipeline_params(w, h, debayer=deb, out_space=L.CS_BT709, out_format=fmt, flags=flags,
                                       storage=storage)
                key = f"{name}/{fmt}"
                with L.Pipeline(ctx, pp) as pipe:
                    for f in range(nfr):
                        m = (W.highlight_frame(w, h, 55 + f) if flags & HL else
                             W.synth_frame(w, h, 17 * w + h + f, noise_a_dn=4.0, noise_b_dn=40.0))
                        out[f"{key}/{f}"] = develop(pipe, m, fp, fmt)
                    out[f"{key}/errors"] = np.array([pipe.kernel_errors()], np.uint32)
    L.debug_denoise_tma(True)
    L.debug_force_denoise_shape(-1)
    return out


if __name__ == "__main__":
    np.savez(sys.argv[1], **run_cases())
