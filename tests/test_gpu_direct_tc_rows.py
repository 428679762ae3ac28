"""The byte form of the direct step on rows that start anywhere in 16 bytes:
the same field rolled by a column, or on a torus tiled twice, is the same
integer sums, and so the same bits, whichever way a tile is staged."""
import numpy as np
import pytest

import life_simulation_b200 as lb

pytestmark = pytest.mark.gpu


def stepped(monkeypatch, a, radius):
    monkeypatch.setenv("LENIA_DIRECT_ENGINE", "tensor")
    m = lb.LeniaModule({"radius": radius, "growthMode": 0, "growthSigma": 0.02}, a.shape[1], a.shape[0])
    monkeypatch.delenv("LENIA_DIRECT_ENGINE")
    m.reset(3)
    m.upload(np.ascontiguousarray(a))
    m.encode(0, 2)
    out = m.field()
    m.sync()
    m.close()
    return out


@pytest.mark.parametrize("w,h", [(129, 130), (130, 129), (131, 257), (199, 150), (163, 3)])
@pytest.mark.parametrize("radius", [4, 16, 17, 32])
def test_rolled_and_tiled_fields(monkeypatch, w, h, radius):
    a = (np.random.default_rng(w + radius).random((h, w)) * 0.31).astype(np.float32)
    out = stepped(monkeypatch, a, radius)
    for by in (1, 2, 3, 33):
        np.testing.assert_array_equal(stepped(monkeypatch, np.roll(a, by, 1), radius), np.roll(out, by, 1))
    np.testing.assert_array_equal(stepped(monkeypatch, np.tile(a, (1, 4)), radius), np.tile(out, (1, 4)))
