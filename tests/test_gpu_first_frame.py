"""GPU: a pipeline's creation loads its develop kernels, and a batch's the batch
kernels, so that the first recording of a process does not wait for them (some
hundred microseconds)."""
import subprocess
import sys
from pathlib import Path

import pytest

import libcraw_gb300 as L

pytestmark = pytest.mark.gpu

HERE = Path(__file__).resolve().parent
SCRIPT = """
import sys, time
sys.path[:0] = [%r, %r]
import torch
import libcraw_gb300 as L
from libcraw_gb300 import workloads as W
from gpu_util import alloc_rgba, upload_mosaic
w, h = 1280, 720
_, src = upload_mosaic(W.synth_frame(w, h, 3))
out, dst = alloc_rgba(w, h)
fp = L.frame_params(W.make_profile())
with L.Context(0) as ctx, L.Pipeline(ctx, L.pipeline_params(w, h, debayer=int(sys.argv[1]), out_space=L.CS_BT709,
                                                            out_format=L.FORMAT_RGBA32F)) as pipe:
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    t = time.perf_counter()
    pipe.record(s.cuda_stream, src, dst, fp)
    print(time.perf_counter() - t)
    torch.cuda.synchronize()
""" % (str(HERE), str(HERE.parent))


# Recording it takes 40 to 80 us; with the kernels yet to load 250 and more
# (730 while the three debayers' kernels were one module). The quickest of a few
# processes, since other work on the host can hold any one up.
@pytest.mark.parametrize("debayer", [L.DEBAYER_BILINEAR, L.DEBAYER_MHC, L.DEBAYER_RCD])
def test_first_record_does_not_load(debayer):
    took = []
    while len(took) < 4 and min(took, default=1.0) > 200e-6:
        r = subprocess.run([sys.executable, "-c", SCRIPT, str(debayer)], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, r.stderr[-2000:]
        took.append(float(r.stdout))
    assert min(took) < 200e-6, took


BATCH = """
import sys, time
sys.path[:0] = [%r, %r]
import torch
import libcraw_gb300 as L
from libcraw_gb300 import workloads as W
from gpu_util import alloc_rgba, upload_mosaic
w, h = 640, 360
src = [upload_mosaic(W.synth_frame(w, h, i, noise_a_dn=4.0, noise_b_dn=40.0)) for i in range(4)]
dst = [alloc_rgba(w, h) for _ in src]
fp = [L.frame_params(W.make_profile(), denoise_strength=1.0, noise_override=W.noise_model(4.0, 40.0)) for _ in src]
with L.Context(0) as ctx, L.Batch(ctx, L.batch_params(w, h, max_frames=4, debayer=int(sys.argv[1]),
                                                     out_space=L.CS_BT709, out_format=L.FORMAT_RGBA32F,
                                                     flags=L.FLAG_DENOISE)) as b:
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    t = time.perf_counter()
    b.record(s.cuda_stream, [i for _, i in src], [i for _, i in dst], fp)
    print(time.perf_counter() - t)
    torch.cuda.synchronize()
""" % (str(HERE), str(HERE.parent))


# Its graph's capture among it, a batch's first recording takes 200 us; with the
# kernels yet to load 800.
@pytest.mark.parametrize("debayer", [L.DEBAYER_MHC, L.DEBAYER_RCD])
def test_first_batch_does_not_load(debayer):
    took = []
    while len(took) < 4 and min(took, default=1.0) > 450e-6:
        r = subprocess.run([sys.executable, "-c", BATCH, str(debayer)], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, r.stderr[-2000:]
        took.append(float(r.stdout))
    assert min(took) < 450e-6, took
