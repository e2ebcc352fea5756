"""The warm-start network's tile kernels at row counts around a tile, a slice and one block per SM."""
import os
import sys

import numpy as np
import pytest
from test_surrogate_gpu import BLOCKS, GAMMA, _features, _norm, _random_params, _states

from euler3d_b200 import api

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import mlp_oracle as mo  # noqa: E402

pytestmark = pytest.mark.gpu


# 64-row tiles; 64 slices of whole tiles: 4,096 rows are one tile each, 4,097 make the slices two tiles
@pytest.mark.parametrize("n", [1, 15, 63, 64, 65, 129, 4096, 4097, 9473])
def test_rows(n):
    rng = np.random.default_rng(n)
    f = _features(rng, max(n, 64))
    norm = _norm(f, _states(f))
    f, p = f[:n], _random_params(rng)
    s = _states(f)
    m = api.Surrogate(seed=1, gamma=GAMMA)
    m.set_params(p, norm)
    loss, g = m.gradient(f, s)
    x, t = mo.prepare(f, s, norm, GAMMA, bf=True)
    loss_ref, g_ref = mo.loss_and_grad(p.astype(np.float64), x, t, bf=True)
    # BF16 rounding (2^-9) of activations and of the gradient at three layers, some of it resolved the other way
    # where the FP32 and FP64 sums straddle a tie: at most a few units of 2^-9, as one row shows it undiluted
    assert abs(loss - loss_ref) <= 8e-3 * loss_ref
    for name, (a, b) in BLOCKS.items():
        assert np.linalg.norm(g[a:b] - g_ref[a:b]) <= 2e-2 * np.linalg.norm(g_ref[a:b]), name
    w_ref = mo.predict(p.astype(np.float64), f, norm, GAMMA, bf=True)
    assert np.max(np.abs(m.predict(f) - w_ref) / norm[16:21]) < 2e-2
    m.close()
