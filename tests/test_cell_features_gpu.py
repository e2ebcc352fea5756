"""Nearest wall faces through clusters against all pairs, on meshes whose warps cross blocks and cases."""
import numpy as np
import pytest

from euler3d_b200 import api
from euler3d_b200 import meshgen as mg

pytestmark = pytest.mark.gpu


# wall faces: 2 n^2 = 18 (one partial cluster), 128 (two exact ones), 450; blocks of uneven warps; two cases in one batch
@pytest.mark.parametrize("sizes,blocks", [((3,), 1), ((8,), 1), ((15,), 3), ((3, 8), 1), ((15, 5), 1)])
def test_wall_distance(sizes, blocks, tmp_path):
    cases = [api.Case(mg.write_case(str(tmp_path / str(i)), n, blocks, deck=mg.Deck(topology="", mach=0.5 + 0.1 * i)))
             for i, n in enumerate(sizes)]
    s = api.Solver(cases[0], precision="fp32") if len(cases) == 1 else api.Batch(cases)
    got = api.cell_features(s)
    at = 0
    for i, case in enumerate(cases):
        wall = np.concatenate([case.get(b, "face_center").reshape(-1, 3)[case.get(b, "wall_faces")]
                               for b in range(case.n_blocks)]).astype(np.float32).astype(np.float64)
        for b in range(case.n_blocks):
            n = case.block_info(b).n_real
            x = case.get(b, "cell_center").reshape(-1, 3)[:n][case.cell_order(b, "none+boundary_last")].astype(np.float32)
            d = np.sqrt(((x.astype(np.float64)[:, None] - wall[None]) ** 2).sum(axis=2).min(axis=1))
            row = got[at:at + n]
            assert np.array_equal(row[:, :3], x)
            # FP32: rounded component differences, three products and sums, one square root
            assert np.all(np.abs(row[:, 3] - d) <= 4 * np.finfo(np.float32).eps * d)
            assert np.all(row[:, 4] == np.float32(0.5 + 0.1 * i))
            at += n
    assert at == got.shape[0]
    s.close()
