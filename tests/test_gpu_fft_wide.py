"""The compile-time-plan spectral passes of the lengths outside the catalogue:
odd and unpadded half rows, two to four passes, the ends of their ranges, and
lengths that still take the runtime plan, against the FP64 oracle."""
import numpy as np
import pytest
import torch

import life_simulation_b200 as lb
from life_simulation_b200 import workloads as wl
from oracle.lenia_oracle import OracleLenia

pytestmark = pytest.mark.gpu

SIZES = [
    (1280, 720), (810, 486),   # a video format; an odd half row (405), rows 8 bytes off 16
    (64, 72), (90, 75),        # the smallest column lengths; half rows 32 and 45
    (100, 81), (162, 125),     # half rows 50 and 81: one and seven padding columns
    (1250, 625), (2560, 96),   # four passes of 5; a half row of 1280
    (4050, 96), (4000, 64),    # half rows near the end of the range; a catalogue column length
    (128, 2160), (96, 4050),   # column lengths above 2048
    (512, 360), (300, 1080),   # one length of the catalogue, the other not
    (96, 3000), (60, 60),      # outside: the runtime plan
]


def params(w, h):
    p = wl.fft3_params(w, h)
    p.update(radius=min(12, min(w, h) // 4), growthMode=1, noiseAmount=0.05, muJitter=0.1, injectAmount=0.2)
    return p


@pytest.mark.parametrize("w,h", SIZES)
def test_steps_against_fp64_oracle(w, h):
    init = wl.patches(w, h, 6, min(w, h) // 3, seed=w)
    m, o = lb.LeniaModule(params(w, h), w, h), OracleLenia(params(w, h), w, h, "f64")
    assert not m.warning and m.tuning() == (0, 0)
    m.reset(5)
    o.reset(5)
    m.upload(init)
    o.set_initial_field(init)
    for f in range(2):  # the spectral path's bound per step
        m.encode(f, 1)
        assert np.abs(m.field() - o.encode(f, 1)).max() <= (f + 1) * 1e-5
    m.close()


@pytest.mark.parametrize("w,h", [(810, 486), (640, 360), (90, 75)])
def test_fused_colour_layer_equals_step_then_render(w, h):
    out = []
    for fused in (True, False):
        m = lb.LeniaModule(params(w, h), w, h)
        m.reset(5)
        m.upload(wl.patches(w, h, 6, min(w, h) // 3, seed=w))
        rgba = torch.zeros((h, w, 4), dtype=torch.float16, device="cuda")
        torch.cuda.synchronize()
        fp = m.frame_params(0)
        if fused:
            m.step_render(fp, 2, rgba.data_ptr(), w, h)
        else:
            m.step(fp, 2)
            m.render_device(rgba.data_ptr(), w, h)
        m.sync()
        out.append((m.field(), rgba.cpu().numpy()))
        m.close()
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])
