"""The host blocks of a solver's reads: every order of small and large reads gives
the same bits (small ones in a large solver take blocks of their own size), and
particles in no slot any more in a read of several rounds of the blocks keep the
caller's values."""
import ctypes as C

import numpy as np
import pytest

from tests.helpers import small_dam
from tests.test_read_gpu import shuffled
from tests.test_scan_gpu import lone
from weaklycompressiblesph_b200 import _native as N
from weaklycompressiblesph_b200 import cases
from weaklycompressiblesph_b200.sim import Solver

pytestmark = pytest.mark.gpu


def test_reads_of_growing_and_shrinking_sizes(native):
    phys = cases.Physics(g=0.0, density_mode=N.DENSITY_CONTINUITY)
    cs = [lone(1), lone(33), small_dam(dx=0.05, seed=1), small_dam(dx=0.02, seed=2),
          shuffled(cases.periodic_lattice(n_side=69, dx=0.01, seed=6, phys=phys))]
    with Solver(sum(c.n for c in cs) + 1_000_000, precision=N.PREC_TILED, max_instances=8) as s:
        ks = [s.add(c) for c in cs]
        for i in (1, 0, 1, 2, 2, 2, 0, 3, 2, 3, 4, 1, 4, 3, 2, 1, 0, 4):
            st, c = s.read(ks[i]), cs[i]
            np.testing.assert_array_equal(st["pos"], c.pos.astype(np.float32))
            np.testing.assert_array_equal(st["vel"], c.vel.astype(np.float32))
            assert (st["alive"] == 1).all()


def test_particles_without_a_slot_in_a_large_read(native):
    case, other = shuffled(small_dam(dx=0.009, vel_sigma=0.0, seed=9)), lone(40)
    assert case.n > 300_000
    fluid = np.nonzero(case.type == N.HYDRO)[0]
    gone = fluid[np.argsort(-case.pos[fluid, 2], kind="stable")][:5]
    case.vel[gone] = [0.0, 0.0, 200.0]
    case.kill_hi = (case.kill_hi[0], case.kill_hi[1], 0.83)
    with Solver(case.n + other.n, precision=N.PREC_TILED) as s:
        k = s.add(case)
        s.step(40)
        s.add(other)  # takes the dead particles' slots
        s.step(2)
        n = case.n
        pos, div, alive = np.full((n, 3), 7.5, np.float32), np.full(n, -3.0, np.float32), np.full(n, 9, np.int32)
        N.call("wcsph_sim_read_instance", s._h, k, N.ptr(pos, C.c_float), None, None, None, N.ptr(div, C.c_float), None,
               N.ptr(alive, C.c_int32))
        full = s.read(k)
    rest = np.setdiff1d(np.arange(n), gone)
    assert (alive[gone] == 0).all() and (alive[rest] == 1).all()
    assert (pos[gone] == 7.5).all() and (div[gone] == -3.0).all() and (full["pos"][gone] == 0.0).all()
    np.testing.assert_array_equal(pos[rest], full["pos"][rest])
    np.testing.assert_array_equal(div[rest], full["div_v"][rest])
