"""Policy AUTO of a batch: the paths are a rule on sizes and taps, the same for
every batch of the same worlds, and each world is what its path gives alone."""
import numpy as np
import pytest

import life_simulation_b200 as lb

pytestmark = pytest.mark.gpu

SIZES = [(128, 128), (256, 256), (384, 216), (512, 512), (90, 70)]


def worlds(n, seed):
    rng = np.random.default_rng(seed)
    return [lb.make_world(width=SIZES[i % 5][0], height=SIZES[i % 5][1], radius=int(rng.integers(3, 33)), mu=0.2,
                          sigma=0.06, dt=0.1, growth_mode=1, seed=i) for i in range(n)]


def stepped(ws, policy):
    b = lb.LeniaBatch(ws, policy)
    for i, w in enumerate(ws):
        b.upload(i, np.random.default_rng(w.seed).random((w.height, w.width), np.float32))
    b.step(2)
    out = [b.field(i) for i in range(len(ws))], [b.path(i) for i in range(len(ws))]
    b.close()
    return out


@pytest.mark.parametrize("n", [1, 4, 10, 45])
def test_auto_paths_are_the_same_each_time_and_change_no_bits(n):
    ws = worlds(n, n)
    fields, paths = stepped(ws, lb.BATCH_AUTO)
    again, paths_again = stepped(ws, lb.BATCH_AUTO)
    assert paths == paths_again
    for i in range(n):
        np.testing.assert_array_equal(fields[i], again[i])
    for path, policy in ((0, lb.BATCH_DIRECT), (1, lb.BATCH_FFT)):
        ids = [i for i in range(n) if paths[i] == path]
        for i, f in zip(ids, stepped([ws[i] for i in ids], policy)[0] if ids else []):
            np.testing.assert_array_equal(fields[i], f)


def test_auto_keeps_few_taps_direct_and_many_spectral():
    one = lambda r: stepped([lb.make_world(width=512, height=512, radius=r, mu=0.2, sigma=0.06, dt=0.1)], 0)[1]  # noqa: E731
    assert one(3) == [0] and one(32) == [1]
