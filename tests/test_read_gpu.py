"""Reads in original order (k_read_index, k_read_state, k_read_diag and the
ring their pieces pass through): what goes in comes out bit for bit, at sizes
of one piece, of ragged pieces and of several rounds of the ring (registered
blocks hold about 90,000 particles), with arrays left out, and with particles
that are in no slot any more, whose entries keep the caller's values."""
import ctypes as C

import numpy as np
import pytest

from tests.helpers import small_dam
from tests.test_scan_gpu import lone
from weaklycompressiblesph_b200 import _native as N
from weaklycompressiblesph_b200 import cases
from weaklycompressiblesph_b200.sim import Solver

pytestmark = pytest.mark.gpu


def shuffled(case, seed=8):
    order = np.random.default_rng(seed).permutation(case.n)
    for f in ("pos", "vel", "dens", "type"):
        setattr(case, f, getattr(case, f)[order])
    return case


@pytest.mark.parametrize("kind", ["lone1", "lone31", "lone33", "dam", "lattice"])
def test_state_comes_back_in_order(native, kind):
    if kind == "lattice":
        case = cases.periodic_lattice(n_side=69, dx=0.01, seed=6)
    else:
        case = small_dam(dx=0.02, seed=7) if kind == "dam" else lone(int(kind[4:]))
    case = shuffled(case)
    with Solver(case.n, precision=N.PREC_TILED) as s:
        k = s.add(case)
        for _ in range(2):
            st = s.read(k)
            np.testing.assert_array_equal(st["pos"], case.pos.astype(np.float32))
            np.testing.assert_array_equal(st["vel"], case.vel.astype(np.float32))
            assert (st["alive"] == 1).all()
        pr = s.probe(k)
        np.testing.assert_array_equal(pr["dens"], st["dens"])
        perm, _ = s.order(k)
        assert np.array_equal(np.sort(perm), np.arange(case.n))


@pytest.mark.parametrize("lists", [0, 10])
def test_particles_without_a_slot_keep_the_callers_values(native, lists):
    case, other = shuffled(small_dam(dx=0.05, vel_sigma=0.0, seed=9)), lone(40)
    fluid = np.nonzero(case.type == N.HYDRO)[0]
    gone = fluid[np.argsort(-case.pos[fluid, 2], kind="stable")][:5]  # the top of the column leaves the kill box
    case.vel[gone] = [0.0, 0.0, 200.0]
    case.kill_hi = (case.kill_hi[0], case.kill_hi[1], 1.2)
    with Solver(case.n + other.n, precision=N.PREC_TILED, list_interval=lists) as s:
        k = s.add(case)
        s.step(40)
        assert s.read(k)["alive"].sum() == case.n - 5
        s.add(other)  # takes the dead particles' slots
        s.step(2)
        n = case.n
        pos, dens, alive = np.full((n, 3), 7.5, np.float32), np.full(n, -3.0, np.float32), np.full(n, 9, np.int32)
        dt = np.full(n, 4.0, np.float32)
        N.call("wcsph_sim_read_instance", s._h, k, N.ptr(pos, C.c_float), None, N.ptr(dens, C.c_float), None, None,
               N.ptr(dt, C.c_float), N.ptr(alive, C.c_int32))
        full = s.read(k)
        rest = np.setdiff1d(np.arange(n), gone)
        assert (alive[gone] == 0).all() and (alive[rest] == 1).all()
        assert (pos[gone] == 7.5).all() and (dens[gone] == -3.0).all() and (dt[gone] == 4.0).all()
        assert (full["pos"][gone] == 0.0).all()
        np.testing.assert_array_equal(pos[rest], full["pos"][rest])
        np.testing.assert_array_equal(dens[rest], full["dens"][rest])
        assert (dt[rest] == 0.0).all() and (dens[rest] > 0.0).all()
        pr = s.probe(k)
        assert (pr["nbr"][rest] > 0).all() and (pr["nbr"][gone] == 0).all() and (pr["dens"][gone] == 0.0).all()
