"""The list build's scan (k_list_scan) at the edges of its batches, tiles and
row buffers, through wcsph_sim_list_entries and the list pass: the number of
entries against a brute-force count in FP64 (pairs within 1e-6 of the list
radius may fall either way), and the neighbour counts and forces of the list
pass against the FP64 oracle at the tolerances of the other list tests (counts
exact; 1e-5 FP32, 1e-3 half2)."""
import numpy as np
import pytest

from tests.helpers import small_dam
from tests.test_lists_gpu import LIST_TOL, oracle_list_check
from weaklycompressiblesph_b200 import _native as N
from weaklycompressiblesph_b200 import cases
from weaklycompressiblesph_b200.sim import Solver

pytestmark = pytest.mark.gpu
SKIN = 0.3


def entries_bounds(case):
    """Ordered pairs (a particle at another's very place excluded) certainly
    and possibly within the list radius."""
    p = case.pos.astype(np.float32).astype(np.float64)
    R = (2.0 + SKIN) * case.h
    box = np.array(case.hi) - np.array(case.lo) if case.periodic else None
    lo = hi = 0
    for a in range(0, len(p), 500):
        d = p[a:a + 500, None] - p[None]
        if box is not None:
            d -= box * np.round(d / box)
        r = np.sqrt((d * d).sum(2))
        lo += int(((r > 0) & (r < R * (1 - 1e-6))).sum())
        hi += int(((r > 0) & (r < R * (1 + 1e-6))).sum())
    return lo, hi


def lone(n):
    """n particles in a small box: one cell, a few, none of them full."""
    rng = np.random.default_rng(n)
    phys = cases.Physics(g=0.0, density_mode=N.DENSITY_CONTINUITY)
    pos = rng.uniform(0.02, 0.06, size=(n, 3))
    return cases.Case(name=f"lone{n}", pos=pos, vel=rng.normal(0, 0.1, (n, 3)), dens=np.full(n, phys.rho0),
                      type=np.zeros(n, np.int32), dx=0.01, h=0.013, mass=1e-3, phys=phys, lo=(0.0, 0.0, 0.0),
                      hi=(0.09, 0.09, 0.09))


def build(kind):
    if kind.startswith("lone"):
        return lone(int(kind[4:]))
    if kind == "dense":  # 41 particles a cell (two batches), 800 staged candidates (two tiles), rows of 172
        return small_dam(dx=0.05, seed=3, phys=cases.Physics(h_over_dx=1.5))
    if kind == "rows":  # rows between one and two row buffers, cells of about 32
        return small_dam(dx=0.05, seed=4, phys=cases.Physics(h_over_dx=1.38))
    if kind == "twins":  # two particles at one place are not in each other's list
        c = small_dam(dx=0.08, seed=5)
        c.pos[7] = c.pos[11]
        return c
    # three cells an axis: every neighbour cell but one is reached through a face of the box
    c = cases.periodic_lattice(n_side=9 if kind == "box9" else 10, dx=0.01, seed=6,
                               phys=cases.Physics(g=0.0, density_mode=N.DENSITY_CONTINUITY))
    c.vel *= 0.02
    return c


@pytest.mark.parametrize("prec", [N.PREC_TILED, N.PREC_HALF2], ids=["tiled", "half2"])
@pytest.mark.parametrize("kind", ["lone1", "lone2", "lone31", "lone32", "lone33", "lone65", "dense", "rows", "twins",
                                  "box9", "box10"])
def test_scan_writes_every_entry(kind, prec, native, oracle_lib):
    case = build(kind)
    with Solver(case.n, precision=prec, list_interval=50, list_skin=SKIN, autotune=False) as s:
        k = s.add(case, density_mode=N.DENSITY_CONTINUITY)
        pr = s.probe(k, lists=True)  # builds
        st = s.read(k)
        n = s.list_entries()
        assert s.list_stats()["overflows"] == 0
    lo, hi = entries_bounds(case)
    assert lo <= n <= hi
    r = oracle_list_check(oracle_lib, case, st, pr, 0)
    np.testing.assert_array_equal(pr["nbr"], r["cnt"])
    assert r["acc"] < LIST_TOL[prec] and r["div_v"] < LIST_TOL[prec], r
