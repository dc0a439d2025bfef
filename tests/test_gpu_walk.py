"""GPU: the walking warps of the develop stage (a quad column a lane, a
segment of rows a warp) where their dispatch branches: the RCD's interior
against its 64x16 tiles, bit for bit (the two evaluate the same formulas
with the same roundings), for every output layout, an output whose rows are
16-byte but not 32-byte aligned, the chroma path's block means (through the
whole chroma denoise), and the gamut compression on saturated colours; the
bilinear and MHC frames against the batch's per-pixel tiles, bit for bit, at
the widths where a lane or an AWB block hangs over the edge, their histogram
against the CPU builder, and their chroma path against the oracle."""
import numpy as np
import pytest
import torch

import libcraw_gb300 as L
from libcraw_gb300 import workloads as W
from gpu_util import alloc_rgba, develop, download_image, upload_mosaic
from oracle import Oracle, max_rel

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = L.Context(0)
    yield c
    L.debug_rcd_strips(1)
    c.close()


def by_tiles_and_walk(ctx, pp, run):
    out = []
    for mode in (0, 2):
        L.debug_rcd_strips(mode)
        with L.Pipeline(ctx, pp) as pipe:
            out.append((run(pipe), pipe.awb_histogram()))
            assert pipe.kernel_errors() == 0
    L.debug_rcd_strips(1)
    (a, ha), (b, hb) = out
    assert np.array_equal(a.view(np.uint8), b.view(np.uint8))
    assert np.array_equal(ha.count, hb.count) and np.array_equal(ha.weight, hb.weight) and \
        np.array_equal(ha.weight_bright, hb.weight_bright)
    return a


# Interiors of one 24-quad strip and a part, of a few segments, and of one
# segment's least height; sizes that leave 64-pixel tiles at the edges.
SIZES = [(198, 50), (330, 118), (1038, 302)]


@pytest.mark.parametrize("w,h", SIZES)
@pytest.mark.parametrize("fmt", [L.FORMAT_RGBA32F, L.FORMAT_RGB32F, L.FORMAT_RGBA16F])
@pytest.mark.parametrize("space", [L.CS_ACES_AP1, L.CS_BT2020])
def test_rcd_output_layouts(ctx, w, h, fmt, space):
    m = W.synth_frame(w, h, 3 * w + h, rects=48, noise_a_dn=4.0, noise_b_dn=40.0)
    pp = L.pipeline_params(w, h, debayer=L.DEBAYER_RCD, out_space=space, out_format=fmt,
                           flags=L.FLAG_AWB_HISTOGRAM)
    fp = L.frame_params(W.make_profile(), flags=L.FRAME_CLAMP_NEGATIVE if h == 118 else 0)
    by_tiles_and_walk(ctx, pp, lambda pipe: develop(pipe, m, fp, fmt))


@pytest.mark.parametrize("w,h", SIZES)
@pytest.mark.parametrize("storage", [L.STORAGE_FP32, L.STORAGE_FP16])
def test_rcd_chroma_path(ctx, w, h, storage):
    m = W.synth_frame(w, h, 5 * w + h, rects=48, noise_a_dn=4.0, noise_b_dn=40.0)
    pp = L.pipeline_params(w, h, debayer=L.DEBAYER_RCD, out_space=L.CS_P3D65, out_format=L.FORMAT_RGBA32F,
                           flags=L.FLAG_AWB_HISTOGRAM | L.FLAG_CHROMA_DENOISE, storage=storage)
    fp = L.frame_params(W.make_profile(), denoise_chroma_strength=0.7)
    by_tiles_and_walk(ctx, pp, lambda pipe: develop(pipe, m, fp))


def test_rcd_output_16_byte_aligned(ctx):
    w, h = 330, 118
    m = W.synth_frame(w, h, 9, rects=48, noise_a_dn=4.0, noise_b_dn=40.0)
    _, src = upload_mosaic(m)
    pp = L.pipeline_params(w, h, debayer=L.DEBAYER_RCD, out_space=L.CS_BT709, out_format=L.FORMAT_RGBA32F,
                           flags=L.FLAG_AWB_HISTOGRAM)
    fp = L.frame_params(W.make_profile())

    def run(pipe):
        # Rows of w + 1 pixels: their starts are 16 bytes off a 32-byte
        # boundary on every other row, and so is the image's.
        buf = torch.full((h * (w + 1) * 4 + 4,), float("nan"), device="cuda")
        dst = L.Image(buf.data_ptr() + 16, (w + 1) * 16, L.FORMAT_RGBA32F, w, h)
        pipe.record(torch.cuda.current_stream().cuda_stream, src, dst, fp)
        torch.cuda.synchronize()
        assert torch.isnan(buf[:4]).all()
        img = buf[4:].view(h, w + 1, 4)
        assert torch.isnan(img[:, w]).all()
        return img[:, :w].cpu().numpy()

    a = by_tiles_and_walk(ctx, pp, run)
    with L.Pipeline(ctx, pp) as pipe:
        assert np.array_equal(develop(pipe, m, fp).view(np.uint8), np.ascontiguousarray(a).view(np.uint8))


def test_gamut_compression_against_float64(ctx):
    """The compression on strongly saturated flat colours, against its
    definition in float64 on the camera RGB the frame itself gives in AP1
    without it. Bound: the distance's reciprocal, two roots and products on
    float values, 16 roundings and two MUFU powers of 2 ulp an exponent
    unit, within 4e-6 of the peak channel."""
    w, h = 330, 118
    m = W.synth_frame(w, h, 77, rects=64, noise_a_dn=2.0, noise_b_dn=16.0)
    prof = W.make_profile()
    out = {}
    pp = L.pipeline_params(w, h, debayer=L.DEBAYER_RCD, out_space=L.CS_ACES_AP1, out_format=L.FORMAT_RGBA32F)
    with L.Pipeline(ctx, pp) as pipe:
        for f in (0, L.FRAME_NO_GAMUT_COMPRESSION):
            out[f] = develop(pipe, m, L.frame_params(prof, flags=f))[..., :3].astype(np.float64)
    x = out[L.FRAME_NO_GAMUT_COMPRESSION]
    ach = x.max(-1, keepdims=True)
    d = (ach - x) / np.abs(ach)
    lim, thr, p = np.array([1.147, 1.264, 1.312]), np.array([0.815, 0.803, 0.880]), 1.2
    scl = (lim - thr) / (((1 - thr) / (lim - thr)) ** -p - 1) ** (1 / p)
    nd = np.maximum(d - thr, 0.0) / scl
    want = np.where(d < thr, x, ach - (thr + scl * nd / (1 + nd ** p) ** (1 / p)) * np.abs(ach))
    assert (d >= thr).mean() > 0.001, "the scene has no saturated colours"
    assert (np.abs(out[0] - want) <= 4e-6 * np.abs(ach)).all()


# The smallest frame; widths of every remainder by 8 (and by the strips of
# 120 columns: one short, whole, one over); heights of every remainder by 8.
LINEAR = [(8, 8), (10, 12), (118, 18), (120, 24), (122, 38), (244, 62), (366, 50), (1030, 20)]


@pytest.mark.parametrize("w,h", LINEAR)
@pytest.mark.parametrize("deb", [L.DEBAYER_BILINEAR, L.DEBAYER_MHC])
@pytest.mark.parametrize("fmt", [L.FORMAT_RGBA32F, L.FORMAT_RGB32F, L.FORMAT_RGBA16F])
def test_linear_frames_equal_tiles(ctx, w, h, deb, fmt):
    m = W.synth_frame(w, h, 11 * w + h, rects=12, noise_a_dn=4.0, noise_b_dn=40.0)
    fp = L.frame_params(W.make_profile())
    space = L.CS_ACES_AP1 if w % 4 else L.CS_BT2020
    if min(w, h) >= 12:                       # a batch takes frames from 12 pixels a side
        _, src = upload_mosaic(m)
        out, dst = alloc_rgba(w, h, fmt)
        with L.Batch(ctx, L.batch_params(w, h, max_frames=1, debayer=deb, out_space=space, out_format=fmt,
                                         direct_pixels=L.BATCH_ALL_PERSISTENT)) as b:
            b.record(torch.cuda.current_stream().cuda_stream, [src], [dst], [fp])
            torch.cuda.synchronize()
        want = out.float().cpu().numpy()
    pp = L.pipeline_params(w, h, debayer=deb, out_space=space, out_format=fmt, flags=L.FLAG_AWB_HISTOGRAM)
    with L.Pipeline(ctx, pp) as pipe:
        got = develop(pipe, m, fp, fmt)
        hist = pipe.awb_histogram()
        assert pipe.kernel_errors() == 0
    if min(w, h) >= 12:
        assert np.array_equal(got.view(np.uint8), want.view(np.uint8))
    # The same frame with its intermediate kept (another epilogue).
    pp = L.pipeline_params(w, h, debayer=deb, out_space=space, out_format=fmt,
                           flags=L.FLAG_AWB_HISTOGRAM | L.FLAG_KEEP_INTERMEDIATE)
    with L.Pipeline(ctx, pp) as pipe:
        kept = develop(pipe, m, fp, fmt)
        rgb = download_image(pipe.intermediate()[0], "rgba32f")
        hist2 = pipe.awb_histogram()
    assert np.array_equal(got.view(np.uint8), kept.view(np.uint8))
    cnt, wgt, brt = L.awb_histogram_from_rgb(rgb, W.WB)
    for x in (hist, hist2):
        assert np.array_equal(x.count, cnt) and np.array_equal(x.weight, wgt) and \
            np.array_equal(x.weight_bright, brt)


@pytest.mark.parametrize("w,h", [(20, 20), (118, 22), (122, 26), (244, 62)])
@pytest.mark.parametrize("deb", [L.DEBAYER_BILINEAR, L.DEBAYER_MHC])
def test_linear_chroma_vs_oracle(ctx, w, h, deb):
    """The bound is the stage's own (the float oracle within 2e-4)."""
    m = W.synth_frame(w, h, 13 * w + h, rects=12, noise_a_dn=4.0, noise_b_dn=40.0)
    pp = L.pipeline_params(w, h, debayer=deb, out_space=L.CS_BT709, out_format=L.FORMAT_RGBA32F,
                           flags=L.FLAG_CHROMA_DENOISE)
    fp = L.frame_params(W.make_profile(), denoise_chroma_strength=0.8)
    with L.Pipeline(ctx, pp) as pipe:
        got = develop(pipe, m, fp)
        assert pipe.kernel_errors() == 0
    assert max_rel(got, Oracle().process(m, pp, fp, "f32")) <= 2e-4
