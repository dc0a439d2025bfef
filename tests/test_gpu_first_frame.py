"""GPU: a pipeline's creation loads its develop kernels, so that the first frame
a process records does not wait for them (some hundred microseconds)."""
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
