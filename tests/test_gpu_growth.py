"""The growth epilogue's noise and blob injection on every path's kernels, at
the blob counts where their code changes (the centres kept per CTA, and
those past them hashed per pixel), against the FP32 restatement of the
reference."""
import numpy as np
import pytest

import life_simulation_b200 as lb
from oracle.lenia_oracle import OracleLenia

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,conv", [(90, 70, "direct"), (331, 257, "direct"), (256, 128, "fft"), (90, 75, "fft")])
@pytest.mark.parametrize("count", [1, 32, 33, 40])
def test_noise_and_blobs(w, h, conv, count):
    # Growth switched off (dt = 0): a frame adds only the hashed noise and
    # blends in the hashed blobs. A blob's share rounds three times, its
    # exponent's rounding weighs x e^-x, and its centre's distance is exact to
    # 2^-24 of the field against a radius of 1/20 of it: 4e-7 a blob in all.
    p = {"convMode": conv, "fftAnySize": True, "radius": 4, "dt": 0.0, "noiseAmount": 0.5, "injectAmount": 0.8,
         "injectCount": count, "growthMode": 0}
    init = np.random.default_rng(w).random((h, w)).astype(np.float32)
    m, o = lb.LeniaModule(p, w, h), OracleLenia(p, w, h, "ref32" if conv == "direct" else "f64")
    m.reset(9)
    o.reset(9)
    m.upload(init)
    o.set_initial_field(init)
    for f in (0, 13):  # another injection cycle every 12 frames
        m.encode(f, 1)
        assert np.abs(m.field() - o.encode(f, 1)).max() <= 4e-7 * (count + 1), f
    m.close()
