"""The adjoint row pass keeps three sums per kernel and thread: gradients for
every number of kernels, both growth modes, against the FP64 oracle (the
bounds of test_gpu_adjoint.py)."""
import numpy as np
import pytest

import life_simulation_b200 as lb
from oracle import lenia_adjoint_oracle as O
from test_gpu_adjoint import fields, oracle_params, oracle_vector, run_engine

pytestmark = pytest.mark.gpu

KERNELS = [{"mu": 0.15, "sigma": 0.03, "weight": 0.5, "betas": [1.0]},
           {"mu": 0.25, "sigma": 0.05, "weight": 0.3, "betas": [0.5, 1.0]},
           {"mu": 0.2, "sigma": 0.04, "weight": 0.4, "betas": [1.0, 0.6]},
           {"mu": 0.3, "sigma": 0.06, "weight": 0.2, "betas": [1.0]}]


@pytest.mark.parametrize("count", [1, 2, 3, 4])
@pytest.mark.parametrize("mode", [0, 1])
def test_gradients_for_each_number_of_kernels(count, mode):
    w, h, batch, steps, radius = 128, 64, 2, 4, 9
    kernels = KERNELS[:count]
    eng = lb.LeniaAdjoint(w, h, batch, kernels, radius, steps, checkpoint_every=2, dt=0.1, growth_mode=mode)
    a0 = fields(batch, h, w, seed=4)
    target = fields(batch, h, w, seed=5) * 0.5
    _, ga0, gp = run_engine(eng, a0, target)
    p = oracle_params(kernels, radius, 0.1, mode, lb.CORE_EXP)
    _, g = O.loss_and_grads(a0.astype(np.float64), target.astype(np.float64), p, steps)
    assert np.abs(ga0 - g.field).max() <= 2e-3 * np.abs(g.field).max()
    ref = oracle_vector(g, p)
    for i, v in enumerate(ref):
        assert abs(gp[i] - v) <= 2e-3 * abs(v) + 1e-7 * np.abs(ref).max(), (i, gp[i], v)
    eng.close()
