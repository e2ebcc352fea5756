"""The reported device memory follows the buffers that are made on first use and kept."""
import pytest

from euler3d_b200 import api
from euler3d_b200 import meshgen as mg

pytestmark = pytest.mark.gpu


def test_kept_buffers_are_counted(tmp_path):
    n = 8
    case = api.Case(mg.write_case(str(tmp_path), n, deck=mg.Deck(topology="", mach=0.5)))
    info = case.block_info(0)
    s = api.Solver(case)
    at = s.device_bytes()
    s.get(0, "dt")  # one value a cell on its way, and the cells' places
    assert s.device_bytes() - at == 8 * info.n_real + 4 * info.n_real
    s.get(0, "prim")  # five values a cell, ghosts too
    assert s.device_bytes() - at == 8 * 5 * info.n_all + 4 * info.n_real
    s.get(0, "w0")  # fits
    assert s.device_bytes() - at == 8 * 5 * info.n_all + 4 * info.n_real
    at = s.device_bytes()
    walls, clusters = 2 * n * n, 2 * n * n // 64
    api.cell_features(s)  # FP32 centres; a box and a first face each cluster and one past the last; two offsets
    assert s.device_bytes() - at == 16 * walls + (32 + 4) * (clusters + 1) + 4 * 2
    s.close()
    case.close()
