"""Lists that a probe builds, and probes of instances that a build's step did
not advance: the rows of every active instance are written, whatever its phase.

Counts and forces against the FP64 oracle at the tolerances of the other list
tests (counts exact; 1e-5 FP32, 1e-3 half2)."""
import numpy as np
import pytest

from tests.helpers import small_dam
from tests.test_lists_gpu import LIST_TOL, oracle_list_check
from weaklycompressiblesph_b200 import _native as N
from weaklycompressiblesph_b200 import cases
from weaklycompressiblesph_b200.sim import Solver

pytestmark = pytest.mark.gpu
PRECS = pytest.mark.parametrize("prec", [N.PREC_TILED, N.PREC_HALF2], ids=["tiled", "half2"])


def two_dams():
    return small_dam(dx=0.05, seed=1, vel_sigma=0.2), small_dam(dx=0.04, seed=2, vel_sigma=0.2, column=(0.3, 0.4, 0.6))


def check(oracle_lib, case, st, pr, prec):
    assert (st["alive"] == 1).all()
    r = oracle_list_check(oracle_lib, case, st, pr, 0)
    np.testing.assert_array_equal(pr["nbr"], r["cnt"])
    assert r["acc"] < LIST_TOL[prec] and r["div_v"] < LIST_TOL[prec], r
    return r["tot"]


@PRECS
def test_probe_on_stale_lists_builds_every_instance(prec, native, oracle_lib):
    a, b = two_dams()
    with Solver(a.n + b.n, max_instances=2, precision=prec, list_interval=20, autotune=False) as s:
        ka, kb = s.add(a), s.add(b)
        s.step(3)
        s.probe(ka)              # a search: the lists are dropped
        s.probe(ka, lists=True)  # builds them
        builds = s.list_stats()["builds"]
        check(oracle_lib, b, s.read(kb), s.probe(kb, lists=True), prec)
        s.step(2)  # reads the lists of the probe
        assert s.list_stats()["builds"] == builds
        pairs, states = s.last_pairs(), [s.read(ka), s.read(kb)]
        tot = [check(oracle_lib, c, st, s.probe(k, lists=True), prec) for c, st, k in zip((a, b), states, (ka, kb))]
    assert pairs == sum(tot)


@PRECS
def test_probe_of_a_finished_instance(prec, native, oracle_lib):
    """An instance past its t_end stays in the lists of the builds that follow."""
    a, b = two_dams()
    with Solver(a.n + b.n, max_instances=2, precision=prec, list_interval=2, autotune=False) as s:
        ka, kb = s.add(a, t_end=1e-9), s.add(b)
        s.step(7)  # builds at every other step
        assert s.status(ka)["finished"] and s.status(ka)["steps"] == 1 and s.status(kb)["steps"] == 7
        assert s.list_stats()["builds"] >= 3
        for c, k in ((a, ka), (b, kb)):
            check(oracle_lib, c, s.read(k), s.probe(k, lists=True), prec)


@pytest.mark.parametrize("density_pass", [1, 2], ids=["summation", "shepard"])
def test_probe_of_a_finished_instance_whose_lists_overflowed(density_pass, native, oracle_lib):
    """Its lists ask for no rebuild, and a partial build for the other instance keeps them."""
    a = small_dam(dx=0.05, seed=8, phys=cases.Physics(h_over_dx=2.5))
    b = cases.periodic_lattice(n_side=12, dx=0.01, seed=3, phys=cases.Physics(g=0.0, density_mode=N.DENSITY_CONTINUITY))
    b.vel = np.random.default_rng(4).normal(0.0, 2.0, size=b.vel.shape)
    with Solver(a.n + b.n, max_instances=2, precision=N.PREC_TILED, list_interval=1000, autotune=False) as s:
        ka, kb = s.add(a, t_end=1e-9), s.add(b)
        s.step(30)
        sched = s.list_schedule()
        assert s.status(ka)["steps"] == 1 and sched["partial_builds"] >= 2 and sched["list_steps"] >= 5, sched
        for _ in range(30):  # to a step that has just built in part
            s.step(1)
            if s.list_schedule()["partial_builds"] > sched["partial_builds"]:
                break
        assert s.list_schedule()["partial_builds"] == sched["partial_builds"] + 1
        st = s.read(ka)
        pr = s.probe(ka, density_pass=density_pass, lists=True)
        check(oracle_lib, b, s.read(kb), s.probe(kb, lists=True), N.PREC_TILED)
    r = oracle_list_check(oracle_lib, a, st, pr, density_pass)
    np.testing.assert_array_equal(pr["nbr"], r["cnt"])
    assert r["dens"] < 1e-5 and r["acc"] < 1e-5 and r["div_v"] < 1e-5, r


@pytest.mark.parametrize("density_pass", [1, 2], ids=["summation", "shepard"])
@PRECS
def test_probe_of_overflowed_lists(prec, density_pass, native, oracle_lib):
    """Particles with more neighbours than a list holds (about 500 at h = 2.5
    dx): the density pass of a probe searches for them as its pair sums do."""
    case = small_dam(dx=0.05, seed=8, phys=cases.Physics(h_over_dx=2.5))
    with Solver(case.n, precision=prec, list_interval=10, autotune=False) as s:
        k = s.add(case)
        s.step(2)
        assert s.list_stats()["overflows"] >= 1
        st = s.read(k)
        pr = s.probe(k, density_pass=density_pass, lists=True)
    r = oracle_list_check(oracle_lib, case, st, pr, density_pass)
    np.testing.assert_array_equal(pr["nbr"], r["cnt"])
    assert r["dens"] < 1e-5 and r["acc"] < LIST_TOL[prec] and r["div_v"] < LIST_TOL[prec], r
