"""The byte form's integer sums on dense fields: every product reaches its
level, the same in every run, whatever the products of other bytes do."""
import numpy as np
import pytest

import life_simulation_b200 as lb
from oracle.lenia_oracle import OracleLenia

pytestmark = pytest.mark.gpu

RINGS = [{"radiusScale": 1.0, "mu": 0.16, "sigma": 0.015, "weight": 0.5, "betas": [1.0]},
         {"radiusScale": 0.9, "mu": 0.15, "sigma": 0.02, "weight": 0.3, "betas": [0.5, 1.0]},
         {"radiusScale": 0.6, "mu": 0.17, "sigma": 0.03, "weight": 0.2, "betas": [1.0, 0.667, 0.333]},
         {"radiusScale": 0.3, "mu": 0.14, "sigma": 0.015, "weight": 0.4, "betas": [1.0, 0.6]}]


@pytest.mark.parametrize("kernels,radius", [(1, 32), (4, 32), (4, 16)])
def test_dense_sums_repeat_and_match_fp64(monkeypatch, kernels, radius):
    w, h = 420, 300  # 42 tiles, some past the field's edges
    p = {"convMode": "directMulti", "radius": radius, "growthMode": 0, "kernels": RINGS[:kernels]}
    a = (np.random.default_rng(radius).random((h, w)) * 0.31).astype(np.float32)
    monkeypatch.setenv("LENIA_DIRECT_ENGINE", "tensor")
    m, o = lb.LeniaModule(p, w, h), OracleLenia(p, w, h, "f64")
    monkeypatch.delenv("LENIA_DIRECT_ENGINE")
    m.reset(3)
    o.reset(3)
    o.set_initial_field(a)
    exact = o.encode(0, 1)
    first = None
    for _ in range(20):
        m.upload(a)
        m.encode(0, 1)
        f = m.field()
        first = f if first is None else first
        np.testing.assert_array_equal(f, first)
    m.sync()
    m.close()
    # U <= 1 rounds at 1.2e-7 in all (its values at 2^-24, its combination three
    # times at 2^-25 of at most 0.35), the growth's slope is dt * 1.22 / sigma = 8.1
    # at most over weights that sum to 1.4, and its exponential and A' round at 2e-7.
    assert np.abs(first - exact).max() <= 1.2e-7 * 8.1 * 1.4 + 2e-7


@pytest.mark.parametrize("w,h", [(256, 200), (199, 131)])
@pytest.mark.parametrize("mode", [0, 1])
def test_every_option_against_fp64(monkeypatch, w, h, mode):
    """Noise, mu jitter and blobs on the byte form's epilogue, rows aligned and not."""
    p = {"convMode": "directMulti", "radius": 14, "growthMode": mode, "kernels": RINGS[:3], "noiseAmount": 0.1,
         "muJitter": 0.3, "injectAmount": 0.3, "injectCount": 5}
    a = (np.random.default_rng(w).random((h, w)) * 0.31).astype(np.float32)
    monkeypatch.setenv("LENIA_DIRECT_ENGINE", "tensor")
    for f in (0, 13):  # another injection cycle every 12 frames
        m, o = lb.LeniaModule(p, w, h), OracleLenia(p, w, h, "f64")
        assert m.info()["tc_engine"] == 4
        m.reset(9)
        o.reset(9)
        m.upload(a)
        o.set_initial_field(a)
        m.encode(f, 1)
        # The sums' and the growth's rounding as above, and 4e-7 a blob and one more
        # for the noise.
        assert np.abs(m.field() - o.encode(f, 1)).max() <= 1.2e-7 * 8.1 + 2e-7 + 4e-7 * 6, f
        m.sync()
        m.close()
