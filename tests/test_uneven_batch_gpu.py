"""A batch of one mesh of several norm chunks beside many of one chunk: norms, and memory no larger than its parts'."""
import numpy as np
import pytest

from euler3d_b200 import api
from euler3d_b200 import meshgen as mg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("big_first", [True, False])
def test_uneven_batch(big_first, tmp_path, monkeypatch):
    monkeypatch.setenv("E3D_BATCH_FORM", "per-pass")
    # 24,576 cells (24 chunks of 1,024), 20 meshes of 750 cells (less than a chunk)
    sizes = [16] + [5] * 20 if big_first else [5] * 20 + [16]
    deck = mg.Deck(topology="", mach=0.5, flux="ausm", order=1)
    path = {n: mg.write_case(str(tmp_path / str(n)), n, deck=deck) for n in set(sizes)}
    cases = [api.Case(path[n]) for n in sizes]
    parts = {}
    for n in set(sizes):
        s = api.Solver(cases[sizes.index(n)], precision="fp64")
        parts[n] = s.device_bytes()
        s.close()
    batch = api.Batch(cases, precision="fp64")
    # what only a batch has: a few numbers a ghost cell (12 n^2) or wall face
    assert batch.device_bytes() <= sum(parts[n] for n in sizes) + sum(16 * 12 * n * n for n in sizes)
    batch.solve_batch(3, -1e300, iters_per_launch=3)
    eps = np.finfo(np.float64).eps
    for c, n in enumerate(sizes):
        n_real = 6 * n**3
        r = batch.get(c, "conv_res") - batch.get(c, "diss_res")
        ref = np.sqrt((r.reshape(5, -1) ** 2).sum(axis=1)) / n_real
        # two summation orders of n positive terms, halved by the root; its rounding and the division's
        assert np.all(np.abs(batch.case_history(c)["rms"][-1] - ref) <= (0.5 * n_real + 2) * eps * ref), c
    batch.close()
