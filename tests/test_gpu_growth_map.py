"""The growth map's arithmetic: the full-range exponential on the paths that
have it, on both direct engines."""
import numpy as np
import pytest

import life_simulation_b200 as lb

pytestmark = pytest.mark.gpu


def module(monkeypatch, engine, params, w, h):
    monkeypatch.setenv("LENIA_DIRECT_ENGINE", engine)
    m = lb.LeniaModule(params, w, h)
    monkeypatch.delenv("LENIA_DIRECT_ENGINE")
    m.reset(3)
    return m


@pytest.mark.parametrize("engine,conv", [("ffma", "direct"), ("tensor", "direct"), ("ffma", "directMulti"),
                                         ("tensor", "directMulti")])
def test_far_tail_of_the_bell(monkeypatch, engine, conv):
    """13.5 widths from mu the bell is subnormal; a time step of 1e37 shows it at
    a pixel that is zero in a flat field (its own weight is zero)."""
    w, h, flat, mu, sigma, dt = 131, 70, np.float32(0.31), np.float32(0.15), np.float32(0.0118), np.float32(1e37)
    p = {"convMode": conv, "radius": 5, "kernelCore": "gaussShell", "growthMode": 1, "growthMu": float(mu),
         "growthSigma": float(sigma), "dt": float(dt)}
    m = module(monkeypatch, engine, p, w, h)
    a = np.full((h, w), flat, np.float32)
    a[20, 20] = 0.0
    m.upload(a)
    m.encode(0, 1)
    got = m.field()[20, 20]
    m.close()
    t = (np.float64(flat) - mu) / sigma
    expected = np.float64(dt) * np.exp(-0.5 * t * t)
    # U rounds at 2^-24 of 0.31 and 80 taps: t * dU / sigma of the bell, and the
    # bell at 2^-149.
    assert 1e-3 < expected < 0.5
    assert abs(got - expected) <= expected * (t / float(sigma) * 0.31 * 80 * 2.0**-24 + 1e-5) + float(dt) * 2.0**-149


@pytest.mark.parametrize("weight", [0.42, 0.77, 41.0])
@pytest.mark.parametrize("w,h,conv,engine", [(96, 64, "directMulti", "ffma"), (131, 150, "directMulti", "tensor"),
                                             (256, 128, "fft", ""), (512, 72, "fft", ""), (90, 75, "fft", ""),
                                             (60, 60, "fft", "")])
def test_the_weights_sum_divides(monkeypatch, w, h, conv, engine, weight):
    """A kernel so wide that its bell is one everywhere: the target is h / h, which
    a division gives as exactly one and a product with 1 / h does not."""
    assert np.float32(weight) * (np.float32(1.0) / np.float32(weight)) != np.float32(1.0)
    p = {"convMode": conv, "fftAnySize": True, "radius": 9, "growthMode": 1, "dt": 1.0,
         "kernels": [{"radiusScale": 1.0, "mu": 0.2, "sigma": 1e6, "weight": weight, "betas": [1.0]}]}
    m = module(monkeypatch, engine, p, w, h)
    assert not m.warning
    m.upload(np.zeros((h, w), np.float32))
    m.encode(0, 1)
    np.testing.assert_array_equal(m.field(), np.float32(1.0))
    m.close()
