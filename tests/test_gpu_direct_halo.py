"""The direct kernels' halo staging around the torus: fields narrower than a
warp, a tile or its halo, where a tile's columns and rows wrap several times."""
import numpy as np
import pytest

import life_simulation_b200 as lb
from oracle.lenia_oracle import OracleLenia

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (2, 3), (31, 33), (32, 17), (33, 8), (76, 9), (65, 64)]


@pytest.mark.parametrize("w,h", SIZES)
@pytest.mark.parametrize("radius", [3, 16, 32])
def test_a_tiled_world_repeats_the_small_one(w, h, radius):
    """A periodic field on a larger torus is the same computation, tap by tap
    in the same order, with other tile edges: the same bits."""
    nx, ny = -(-160 // w), -(-144 // h)
    a = (np.random.default_rng(w + radius).random((h, w)) * 0.31).astype(np.float32)
    common = dict(radius=radius, mu=0.15, sigma=0.03, dt=0.1, seed=5)
    b = lb.LeniaBatch([lb.make_world(width=w, height=h, **common),
                       lb.make_world(width=w * nx, height=h * ny, **common)], lb.BATCH_DIRECT)
    b.upload(0, a)
    b.upload(1, np.tile(a, (ny, nx)))
    b.step(2)
    np.testing.assert_array_equal(np.tile(b.field(0), (ny, nx)), b.field(1))
    b.close()


@pytest.mark.parametrize("w,h", SIZES)
def test_small_fields_against_fp64_oracle(monkeypatch, w, h):
    p = {"radius": 5, "growthMode": 0, "growthSigma": 0.015}
    monkeypatch.setenv("LENIA_DIRECT_ENGINE", "ffma")
    m, o = lb.LeniaModule(p, w, h), OracleLenia(p, w, h, "f64")
    a = (np.random.default_rng(w).random((h, w)) * 0.31).astype(np.float32)
    m.reset(3)
    o.reset(3)
    m.upload(a)
    o.set_initial_field(a)
    m.encode(0, 1)
    # 81 taps, each rounded once, times the growth's slope dt * 1.22 / sigma.
    assert np.abs(m.field() - o.encode(0, 1)).max() <= 81 * 2.0**-24 * 8.1 + 2e-7
    m.close()


@pytest.mark.parametrize("few", [1, 40])
def test_batch_tiles_of_four_and_eight_outputs_agree(few):
    """`few` worlds of 64 tiles each, below and above the launch's line of tiles
    per SM: the same world in either batch is the same bits."""
    a = np.random.default_rng(7).random((256, 128), np.float32)
    out = []
    for n in (1, few):
        b = lb.LeniaBatch([lb.make_world(width=128, height=256, radius=9, mu=0.15, sigma=0.03, dt=0.1, seed=5)] * n,
                          lb.BATCH_DIRECT)
        for i in range(n):
            b.upload(i, a)
        b.step(3)
        out += [b.field(i) for i in range(n)]
        b.close()
    for f in out[1:]:
        np.testing.assert_array_equal(f, out[0])
