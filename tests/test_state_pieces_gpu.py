"""State arrays longer than the 2^22 values that come from the device at a time."""
import numpy as np
import pytest

from euler3d_b200 import api
from euler3d_b200 import meshgen as mg

pytestmark = pytest.mark.gpu


def test_arrays_of_several_pieces(tmp_path):
    case = api.Case(mg.write_case(str(tmp_path), 52, deck=mg.Deck(topology="", mach=0.5, order=1)))
    info = case.block_info(0)
    s = api.Solver(case)
    # rows of real cells and packed values of all cells: two pieces; gradients: four, the later ones from within a triple
    for name, size in (("diss_res", 5 * info.n_real), ("limiter", 5 * info.n_all), ("grad", 15 * info.n_all)):
        assert size > 2**22
        x = np.random.default_rng(size).standard_normal(size)
        s.set(0, name, x)
        assert np.array_equal(np.asarray(s.get(0, name)).ravel(), x), name
    s.close()
    case.close()
