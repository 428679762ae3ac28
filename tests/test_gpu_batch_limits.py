"""A persistent batch steps on after batches of smaller worlds were made: their
launches' shared-memory needs are their own."""
import numpy as np
import pytest

import life_simulation_b200 as lb

pytestmark = pytest.mark.gpu


def worlds(size, radius, n):
    return [lb.make_world(width=size[0], height=size[1], radius=radius, mu=0.2, sigma=0.06, dt=0.1, seed=i) for i in range(n)]


def test_a_smaller_batch_lowers_no_other_batchs_limit(monkeypatch):
    monkeypatch.setenv("LENIA_BATCH_PERSISTENT", "1")
    a = np.random.default_rng(1).random((2, 512, 512), np.float32)

    def stepped(smaller_in_between):
        # Direct tiles of the largest radius need the most, spectral items the least.
        big = lb.LeniaBatch(worlds((512, 512), 32, 1) + worlds((512, 512), 4, 1), lb.BATCH_DIRECT)
        assert big.launch_form() == 1
        for i in range(2):
            big.upload(i, a[i])
        big.step(2)
        if smaller_in_between:
            small = lb.LeniaBatch(worlds((128, 64), 8, 2), lb.BATCH_FFT)
            assert small.launch_form() == 1
            small.step(2)
            small.close()
        big.step(3)  # a count not captured before
        out = [big.field(i) for i in range(2)]
        big.close()
        return out

    for x, y in zip(stepped(False), stepped(True)):
        np.testing.assert_array_equal(x, y)
