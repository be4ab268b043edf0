"""The cell passes of the searching solvers (k_hydro_plain, k_density_plain) at
the edges of their batches and tiles: single particles, cells of more than one
batch of 32, more candidates than a tile, particles at one place and boxes of
three cells an axis, against the FP64 oracle at the tolerances of the other
parity tests (counts exact; relative L2 1e-5)."""
import numpy as np
import pytest

from tests.test_lists_gpu import oracle_list_check
from tests.test_scan_gpu import build
from weaklycompressiblesph_b200 import _native as N
from weaklycompressiblesph_b200.sim import Solver

pytestmark = pytest.mark.gpu
KINDS = ["lone1", "lone2", "lone31", "lone33", "lone65", "lone300", "lone900", "dense", "twins", "box9", "box10"]


@pytest.mark.parametrize("density_pass", [0, 1, 2], ids=["none", "summation", "shepard"])
@pytest.mark.parametrize("kind", KINDS)
def test_cell_passes(kind, density_pass, native, oracle_lib):
    case = build(kind)
    with Solver(case.n, precision=N.PREC_FP32, autotune=False) as s:
        k = s.add(case, density_mode=N.DENSITY_CONTINUITY)
        st = s.read(k)
        pr = s.probe(k, density_pass=density_pass)
    r = oracle_list_check(oracle_lib, case, st, pr, density_pass)
    np.testing.assert_array_equal(pr["nbr"], r["cnt"])
    assert r["acc"] < 1e-5 and r["div_v"] < 1e-5 and r["dt"] < 1e-5, r
    assert r.get("dens", 0.0) < 1e-5, r
