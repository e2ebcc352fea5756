"""A batch with so many wall faces that its ring of pending iterations is shorter than the longest."""
import numpy as np
import pytest

from euler3d_b200 import api
from euler3d_b200 import meshgen as mg

pytestmark = pytest.mark.gpu


def test_short_ring(tmp_path, monkeypatch):
    monkeypatch.setenv("E3D_BATCH_FORM", "per-pass")
    # 64 meshes of 29,478 cells (29 norm chunks) with 578 wall faces: 1.55 MB an iteration, ten of them in 16 MB
    n, count, iters = 17, 64, 23
    case = api.Case(mg.write_case(str(tmp_path), n, deck=mg.Deck(topology="", mach=0.5, flux="ausm", order=1)))
    s = api.Solver(case, precision="fp32")
    part = s.device_bytes()
    s.close()
    a, b = (api.Batch([case] * count, precision="fp32") for _ in range(2))
    # 32 iterations' slots of every mesh at most 16 MB together; a few numbers a ghost cell only a batch has
    ring = 32 * 40 * (29 + 2 * n * n)
    assert a.device_bytes() <= count * (part - ring + 16 * 12 * n * n) + 2**24
    a.solve_batch(iters, -1e300, iters_per_launch=iters)
    b.solve_batch(iters, -1e300, iters_per_launch=1)
    for c in (0, 31, 63):
        ha, hb = a.case_history(c), b.case_history(c)
        assert len(ha["iter"]) == iters
        for k in ha:
            assert np.array_equal(ha[k], hb[k]), (c, k)
    a.close()
    b.close()
