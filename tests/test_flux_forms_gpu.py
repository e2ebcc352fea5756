"""Stage passes against the oracle at the sizes where their forms change and where their last blocks are partly filled."""
import os

import numpy as np
import pytest
from oracle_c import case_oracle

from euler3d_b200 import api
from euler3d_b200 import meshgen as mg

pytestmark = pytest.mark.gpu


# one lane per slot up to 60,000 (AUSM) and 180,000 (Roe) tetrahedra, 30,000 and 40,000 hexahedra; last blocks partly filled
@pytest.mark.parametrize("mesh,n,nz,flux,order", [
    ("bump", 21, 1, "ausm", 2), ("bump", 22, 1, "ausm", 1), ("bump", 31, 1, "roe", 2), ("bump", 32, 1, "roe", 1),
    ("hex", 20, 75, "ausm", 2), ("hex", 20, 76, "ausm", 2), ("hex", 20, 100, "roe", 1), ("hex", 20, 101, "roe", 2),
    ("hex", 3, 1, "roe", 2),
])
def test_matches_oracle(mesh, n, nz, flux, order, tmp_path):
    deck = mg.Deck(topology="", mach=0.7, aoa_deg=2.0, flux=flux, order=order)
    path = mg.write_hex_case(str(tmp_path), n, nz, deck=deck) if mesh == "hex" else mg.write_case(str(tmp_path), n, deck=deck)
    _check(path, deck, str(tmp_path))


# hexahedra, one lane per (cell, variable): 32 cells fill a block exactly, 99 leave the fourth with 3
@pytest.mark.parametrize("n,nz", [(4, 2), (3, 11)])
@pytest.mark.parametrize("gradient", ["greengauss", "leastsquares"])
@pytest.mark.parametrize("limiter", ["barthjespersen", "venkatakrishnan"])
def test_hex_reconstruction(n, nz, gradient, limiter, tmp_path):
    deck = mg.Deck(topology="", mach=0.7, aoa_deg=2.0, flux="ausm", order=2, gradient=gradient, limiter=limiter)
    _check(mg.write_hex_case(str(tmp_path), n, nz, deck=deck), deck, str(tmp_path))


def _check(path, deck, directory):
    case = api.Case(path)
    ref = case_oracle(case, os.path.join(directory, deck.topology))
    s = api.Solver(case)
    ref.iterate(2)
    s.iterate(2)
    for k in ("prim", "conv_res", "diss_res"):  # FP64: the reference's operation order, bit for bit
        got = s.get(0, k).reshape(5, -1)
        assert np.array_equal(got, np.asarray(getattr(ref.blocks[0], k)).reshape(5, -1)[:, :got.shape[1]]), k
    s.close()
    case.close()
