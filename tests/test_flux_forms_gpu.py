"""The flux pass's two forms (one lane per slot, one thread per cell) on both sides of the size where they change."""
import os

import numpy as np
import pytest
from oracle_c import case_oracle

from euler3d_b200 import api
from euler3d_b200 import meshgen as mg

pytestmark = pytest.mark.gpu


# tetrahedra: 80,000 cells (AUSM) and 220,000 (Roe); hexahedra: half of these; last blocks partly filled
@pytest.mark.parametrize("mesh,n,nz,flux,order", [
    ("bump", 23, 1, "ausm", 2), ("bump", 24, 1, "ausm", 1), ("bump", 33, 1, "roe", 2), ("bump", 34, 1, "roe", 1),
    ("hex", 20, 100, "ausm", 2), ("hex", 20, 101, "ausm", 2), ("hex", 3, 1, "roe", 2),
])
def test_matches_oracle(mesh, n, nz, flux, order, tmp_path):
    deck = mg.Deck(topology="", mach=0.7, aoa_deg=2.0, flux=flux, order=order)
    path = mg.write_hex_case(str(tmp_path), n, nz, deck=deck) if mesh == "hex" else mg.write_case(str(tmp_path), n, deck=deck)
    case = api.Case(path)
    ref = case_oracle(case, os.path.join(str(tmp_path), deck.topology))
    s = api.Solver(case)
    ref.iterate(2)
    s.iterate(2)
    for k in ("prim", "conv_res", "diss_res"):  # FP64: the reference's operation order, bit for bit
        got = s.get(0, k).reshape(5, -1)
        assert np.array_equal(got, np.asarray(getattr(ref.blocks[0], k)).reshape(5, -1)[:, :got.shape[1]]), k
    s.close()
    case.close()
