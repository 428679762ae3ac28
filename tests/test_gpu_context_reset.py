"""Every path runs again, to the same bits, in a CUDA context that follows a
device reset and in a second context on the device: what is kept for the life of
the process may not stand for what a context holds. In a child process, whose
own contexts these are."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = r"""
import ctypes, os, sys
import numpy as np
import life_simulation_b200 as lb
from life_simulation_b200 import workloads as wl

lb.load_library()
rt = ctypes.CDLL("libcudart.so.12")

def modules():
    yield "ffma", {"radius": 32, "growthMode": 0}, 300, 200
    yield "ffma", {"radius": 13, "growthMode": 0}, 1024, 600
    yield "tensor", {"radius": 32, "growthMode": 0}, 300, 200
    for w, h in ((1024, 512), (810, 486), (60, 60), (1024, 4096)):  # catalogue, wide, runtime plan, tensor-core columns
        p = wl.fft3_params(w, h)
        if h == 4096:
            p["fftPrecision"] = "fp16x3"
        yield "", dict(p, radius=12, fftAnySize=True), w, h

def run():
    out = []
    for engine, p, w, h in modules():
        os.environ["LENIA_DIRECT_ENGINE"] = engine
        m = lb.LeniaModule(p, w, h)
        m.reset(3)
        m.upload(np.random.default_rng(w).random((h, w), np.float32))
        m.encode(0, 2)
        f = m.field()
        if h != 4096:  # (its engine is timed at setup)
            out.append(f)
        m.close()
    for persistent in ("0", "1"):
        os.environ["LENIA_BATCH_PERSISTENT"] = persistent
        ws = [lb.make_world(width=512, height=512, radius=r, mu=0.2, sigma=0.06, dt=0.1, seed=r) for r in (6, 30)]
        b = lb.LeniaBatch(ws)
        for i in range(2):
            b.upload(i, np.random.default_rng(i).random((512, 512), np.float32))
        b.step(3)
        out += [b.field(i) for i in range(2)]
        b.close()
    return out

first = run()
if sys.argv[1] == "reset":
    assert rt.cudaDeviceReset() == 0
    second = run()
else:
    cu = ctypes.CDLL("libcuda.so.1")
    ctx = ctypes.c_void_p()
    assert cu.cuCtxCreate_v2(ctypes.byref(ctx), 0, 0) == 0
    second = run()
    assert cu.cuCtxDestroy_v2(ctx) == 0
for a, b in zip(first, second):
    np.testing.assert_array_equal(a, b)
print("same", len(second))
"""


@pytest.mark.parametrize("how", ["reset", "second context"])
def test_paths_run_in_another_context(how):
    r = subprocess.run([sys.executable, "-c", CHILD, how.split()[0]], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same 10" in r.stdout, r.stderr[-2000:]
