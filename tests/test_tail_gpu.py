"""End-of-iteration sums: the ring of pending iterations and its chunk edges."""
import numpy as np
import pytest

from euler3d_b200 import api
from euler3d_b200 import meshgen as mg

pytestmark = pytest.mark.gpu


# 750, 1,296 and 3,072 cells: below, above and exactly three 1,024-cell norm chunks; 2 blocks: halo copies in the tail
@pytest.mark.parametrize("n,blocks", [(5, 1), (6, 1), (8, 1), (6, 2)])
@pytest.mark.parametrize("iters", [1, 31, 32, 33, 65])
def test_ring_matches_single_iterations(n, blocks, iters, tmp_path):
    deck = mg.Deck(topology="", mach=0.6, aoa_deg=1.0, flux="roe", order=1)
    case = api.Case(mg.write_case(str(tmp_path), n, blocks, deck=deck))
    a, b = api.Solver(case), api.Solver(case)
    a.iterate(iters)
    for _ in range(iters):
        b.iterate(1)
    ha, hb = a.history(), b.history()
    for k in ha:
        assert np.array_equal(ha[k], hb[k]), k
    flow = a.flow_data()
    eps = np.finfo(np.float64).eps
    for blk in range(blocks):
        assert np.array_equal(a.get(blk, "prim"), b.get(blk, "prim"))
        r = a.get(blk, "conv_res") - a.get(blk, "diss_res")
        ref = (r.reshape(5, -1) ** 2).sum(axis=1)
        n_real = case.block_info(blk).n_real
        assert np.all(np.abs(flow[blk, :5] - ref) <= n_real * eps * ref)  # two summation orders of n positive terms
    a.close()
    b.close()
    case.close()


# the same ring inside one batch launch
@pytest.mark.parametrize("iters", [31, 32, 33, 70])
def test_batch_ring(iters, tmp_path, monkeypatch):
    monkeypatch.setenv("E3D_BATCH_FORM", "per-pass")
    cases = [api.Case(mg.write_case(str(tmp_path / str(n)), n, deck=mg.Deck(topology="", mach=0.5, flux="ausm")))
             for n in (5, 8)]
    a, b = (api.Batch(cases, precision="fp64") for _ in range(2))
    a.solve_batch(iters, -1e300, iters_per_launch=iters)
    b.solve_batch(iters, -1e300, iters_per_launch=1)
    for c in range(2):
        ha, hb = a.case_history(c), b.case_history(c)
        assert len(ha["iter"]) == iters
        for k in ha:
            assert np.array_equal(ha[k], hb[k]), (c, k)
    a.close()
    b.close()
