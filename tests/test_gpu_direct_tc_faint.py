"""Faint fields on the direct path: the byte form's 32-bit values, and the
growth centres near zero that it leaves to the FP32 kernels, against FP64."""
import numpy as np
import pytest

import life_simulation_b200 as lb
from oracle.lenia_oracle import OracleLenia

pytestmark = pytest.mark.gpu

HALF_STEP = 8388.5 * 2.0**-23  # 1e-3, halfway between two multiples of 2^-23: off by 2^-24 in 24 bits


@pytest.mark.parametrize("field", ["flat", "random", "spots"])
@pytest.mark.parametrize("mu", [0.02, 0.002])
def test_faint_fields_against_fp64(monkeypatch, field, mu):
    w, h = 131, 150
    # Growth centre and width of one size with the field, growth mode 1.
    p = {"radius": 5, "growthMode": 1, "growthMu": mu, "growthSigma": mu, "kernelCore": "gaussShell"}
    rng = np.random.default_rng(3)
    a = np.full((h, w), HALF_STEP, np.float32)
    if field == "random":
        a = (rng.random((h, w)) * 2e-3).astype(np.float32)
    elif field == "spots":  # bright pixels beside the flat ground
        a[rng.random((h, w)) < 0.002] = 0.9
    monkeypatch.setenv("LENIA_DIRECT_ENGINE", "tensor")
    m, o = lb.LeniaModule(p, w, h), OracleLenia(p, w, h, "f64")
    m.reset(3)
    o.reset(3)
    m.upload(a)
    o.set_initial_field(a)
    m.encode(0, 1)
    err = np.abs(m.field() - o.encode(0, 1)).max()
    m.sync()
    m.close()
    # The growth's slope is dt * 0.607 / sigma = 0.0607 / mu. At mu = 0.02 a sum is
    # off by 2^-32 and U - mu rounds at 2^-25 of at most 0.16 (a spot's share); at
    # mu = 0.002 the FP32 sum rounds once for each of 80 taps of U = 1e-3 (0.16 at a
    # spot, but there the bell is zero). The exponential's argument, the exponential and
    # A' round at 4 * 2^-24 of dt and 2^-24 of A' (0.9 beside a spot).
    du = 2.0**-32 + 2.0**-25 * 0.16 if mu == 0.02 else 80 * 2.0**-24 * 1.5e-3
    assert err <= 0.0607 / mu * du + 0.1 * 4 * 2.0**-24 + 2.0**-24
