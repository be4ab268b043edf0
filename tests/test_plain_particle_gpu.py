"""The thread-per-particle passes of the searching solvers (k_hydro_particle,
k_density_particle), which large solvers with few particles a cell take, against
the cell passes: the same terms in the same order, so the same bits.

The launch is chosen by the particles that fill a cell, the cell's volume over
m / rho0.  A case of any size gets the thread-per-particle passes when its
particle mass is made larger by a power of two; sums that carry the mass are
then larger by exactly that power, the others equal."""
import numpy as np
import pytest

from tests.helpers import rel_l2, small_dam
from tests.test_lists_gpu import oracle_list_check
from tests.test_scan_gpu import build
from weaklycompressiblesph_b200 import _native as N
from weaklycompressiblesph_b200 import cases
from weaklycompressiblesph_b200.sim import Solver

pytestmark = pytest.mark.gpu
KINDS = ["lone1", "lone2", "lone31", "lone33", "lone65", "lone300", "lone900", "dense", "twins", "box9", "box10"]
HEAVIER = 2.0 ** 24  # 900 particles and 2.7e-6 of them a cell: both rules ask for at least 19,000 a particle in a cell


@pytest.mark.parametrize("vsig", [0, 1], ids=["ref-cpu", "signal"])
@pytest.mark.parametrize("density_pass", [0, 1, 2], ids=["none", "summation", "shepard"])
@pytest.mark.parametrize("kind", KINDS)
def test_same_bits_as_the_cell_passes(kind, density_pass, vsig, native, oracle_lib):
    case = build(kind)
    case.phys.vsig_mode = vsig
    case.phys.beta = 0.3
    pr = []
    for factor in (1.0, HEAVIER):
        c = cases.Case(**{**case.__dict__, "mass": case.mass * factor})
        with Solver(c.n, precision=N.PREC_FP32) as s:
            k = s.add(c, density_mode=N.DENSITY_CONTINUITY)
            pr.append(s.probe(k, density_pass=density_pass))
            st = s.read(k)
    cell, part = pr
    if density_pass == 1:  # the density itself carries the mass, and what follows it is another state
        np.testing.assert_array_equal(part["dens"], cell["dens"] * np.float32(HEAVIER))
        return
    for f in ("dens", "dt", "nbr"):
        np.testing.assert_array_equal(part[f], cell[f])
    for f in ("acc", "div_v"):
        np.testing.assert_array_equal(part[f], cell[f] * np.float32(HEAVIER))
    r = oracle_list_check(oracle_lib, c, st, part, density_pass)
    np.testing.assert_array_equal(part["nbr"], r["cnt"])
    assert r["acc"] < 1e-5 and r["div_v"] < 1e-5 and r["dt"] < 1e-5, r


@pytest.mark.parametrize("mode", [N.DENSITY_SUMMATION, N.DENSITY_SHEPARD], ids=["summation", "shepard"])
def test_steps_with_few_particles_a_cell(mode, native):
    """54,508 particles, 1.7 a cell: steps, a removed particle among them (with the larger dt of the Shepard mode),
    against the tiled path."""
    case = small_dam(dx=0.02, seed=3, phys=cases.Physics(h_over_dx=0.6, density_mode=mode))
    top = int(np.argmax(np.where(case.type == N.HYDRO, case.pos[:, 2], -1.0)))
    case.vel[top] = [0.0, 0.0, 400.0]
    case.kill_hi = (case.kill_hi[0], case.kill_hi[1], 1.2)
    got = []
    for prec in (N.PREC_FP32, N.PREC_TILED):
        with Solver(case.n, precision=prec) as s:
            k = s.add(case)
            s.step(12)
            got.append((s.read(k), s.last_pairs(), s.status(k)["time"]))
    (a, pa, ta), (b, pb, tb) = got
    assert np.array_equal(a["alive"], b["alive"])
    assert mode == N.DENSITY_SUMMATION or a["alive"].sum() == case.n - 1
    assert pa == pb and abs(ta - tb) <= 1e-5 * tb
    assert rel_l2(a["pos"], b["pos"]) < 1e-6 and rel_l2(a["vel"], b["vel"]) < 1e-4 and rel_l2(a["dens"], b["dens"]) < 1e-6
