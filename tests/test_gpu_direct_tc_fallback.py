"""Tiles of the byte form whose values it cannot hold: their FP32 sums at the
tiles' and rows' edges with every option, and -0, which it can hold."""
import numpy as np
import pytest

import life_simulation_b200 as lb
from life_simulation_b200 import workloads as wl

pytestmark = pytest.mark.gpu


def stepped(monkeypatch, engine, p, a):
    monkeypatch.setenv("LENIA_DIRECT_ENGINE", engine)
    m = lb.LeniaModule(p, a.shape[1], a.shape[0])
    monkeypatch.delenv("LENIA_DIRECT_ENGINE")
    assert m.info()["tc_engine"] == (4 if engine == "tensor" else 0)
    m.reset(3)
    m.upload(a)
    m.encode(0, 1)
    out = m.field()
    m.sync()
    m.close()
    return out


@pytest.mark.parametrize("w,h", [(31, 127), (33, 129), (160, 256), (5, 300), (301, 17), (2, 3)])
@pytest.mark.parametrize("radius,count", [(5, 1), (32, 2)])
def test_out_of_range_everywhere(monkeypatch, w, h, radius, count):
    p = wl.fft3_params(w, h, conv="directMulti")
    p["kernels"] = p["kernels"][:count]
    p.update(radius=radius, noiseAmount=0.1, muJitter=0.3, injectAmount=0.3, injectCount=5, growthMode=count - 1)
    a = (np.random.default_rng(w).random((h, w)) - 0.4).astype(np.float32)
    # The same taps, in another order where a small field splits its rows: 3200 of
    # them at 2^-24 of sums up to 0.2, a tenth of it left as they partly cancel, times
    # the growth's slope dt * 1.22 / 0.0118.
    np.testing.assert_allclose(stepped(monkeypatch, "tensor", p, a), stepped(monkeypatch, "ffma", p, a), rtol=0,
                               atol=3200 * 2.0**-24 * 0.2 * 10.4 * 0.1)


@pytest.mark.parametrize("radius", [9, 32])
def test_negative_zero_is_zero(monkeypatch, radius):
    # Potentials around mu, where the growth shows a sum's last places.
    a = np.random.default_rng(5).random((200, 163), np.float32) * np.float32(0.4)
    p = {"radius": radius, "growthMode": 0, "growthSigma": 0.015}
    a[a < 0.2] = 0.0
    zero = stepped(monkeypatch, "tensor", p, a)
    a[a == 0.0] = -0.0
    np.testing.assert_array_equal(stepped(monkeypatch, "tensor", p, a), zero)
