"""The direct step's byte form on the tensor cores (LENIA_DIRECT_ENGINE=tensor)
at the sizes where its tiles, chunks and row pairs change, against the FP64
oracle and, for values it cannot hold, against the FP32 kernels."""
import numpy as np
import pytest

import life_simulation_b200 as lb
from life_simulation_b200 import workloads as wl
from oracle.lenia_oracle import OracleLenia

pytestmark = pytest.mark.gpu

# Sums are exact to the fields' 2^-24 and one rounding of U <= 1 (1.2e-7 in
# all); the growth's slope dt * 1.22 / sigma is 8.1 at sigma = 0.015, and its
# exponential and A' round at 2e-7 more.
TOL = 1.2e-7 * 8.1 + 2e-7


def engine(monkeypatch, name, params, w, h):
    monkeypatch.setenv("LENIA_DIRECT_ENGINE", name)
    m = lb.LeniaModule(params, w, h)
    monkeypatch.delenv("LENIA_DIRECT_ENGINE")
    m.reset(3)
    return m


@pytest.mark.parametrize("w,h", [(32, 128), (33, 129), (31, 127), (160, 256), (90, 40), (300, 391)])
@pytest.mark.parametrize("radius,core", [(5, "gaussShell"), (16, "exp"), (17, "gaussShell"), (32, "exp")])
def test_tiles_and_chunks(monkeypatch, w, h, radius, core):
    p = {"radius": radius, "kernelCore": core, "growthMode": 0, "growthSigma": 0.015}
    # Potentials around mu, where the growth is steepest.
    init = (np.random.default_rng(w + radius).random((h, w)) * 0.31).astype(np.float32)
    m, o = engine(monkeypatch, "tensor", p, w, h), OracleLenia(p, w, h, "f64")
    o.reset(3)
    m.upload(init)
    o.set_initial_field(init)
    m.encode(0, 1)
    assert np.abs(m.field() - o.encode(0, 1)).max() <= TOL
    m.sync()
    m.close()


@pytest.mark.parametrize("count", [1, 2, 3, 4])
def test_kernel_counts_with_every_option(monkeypatch, count):
    w, h = 200, 150
    p = wl.fft3_params(w, h, conv="directMulti")
    p["kernels"] = (p["kernels"] + [{"radiusScale": 0.5, "mu": 0.2, "sigma": 0.03, "weight": 0.4, "betas": [1.0, 0.6]}])[:count]
    p.update(radius=20, noiseAmount=0.1, muJitter=0.3, injectAmount=0.3, injectCount=5, growthMode=1)
    init = wl.patches(w, h, 8, 40, seed=9)
    out = []
    for eng in ("ffma", "tensor"):
        m = engine(monkeypatch, eng, p, w, h)
        m.upload(init)
        m.encode(0, 2)
        out.append(m.field())
        m.close()
    # Two steps of two roundings each (the FP32 form's sums round per tap).
    assert np.abs(out[0] - out[1]).max() <= 1e-5


@pytest.mark.parametrize("value", [2.5, -0.5, -0.0, np.inf, np.nan])
def test_values_without_a_byte_form(monkeypatch, value):
    # Tiles that see such a value run the FP32 loop in the FP32 kernels' tap
    # order; the others the byte form.
    w, h = 256, 300
    p = {"radius": 9, "growthMode": 0, "growthSigma": 0.015}
    init = (np.random.default_rng(5).random((h, w)) * 0.31).astype(np.float32)
    init[200, 70] = value
    out = []
    for eng in ("ffma", "tensor"):
        m = engine(monkeypatch, eng, p, w, h)
        m.upload(init)
        m.encode(0, 1)
        out.append(m.field())
        m.close()
    assert np.isfinite(out[1]).all()
    assert np.abs(out[0] - out[1]).max() <= 2 * TOL + 1e-6


def test_large_fields_take_it_and_repeat_their_bits():
    # A size rule: the same configuration sums the same way every time.
    p = {"radius": 13, "growthMode": 0}
    init = wl.patches(1000, 700, 12, 96, seed=8)
    out = []
    for _ in range(2):
        m = lb.LeniaModule(p, 1000, 700)
        m.reset(3)
        m.upload(init)
        m.encode(0, 5)
        out.append(m.field())
        m.close()
    np.testing.assert_array_equal(out[0], out[1])
