"""Walk kernels at the edges of their tiles.

One batch holds walks of 1 to 129 i-particles (blocks of 32) against j-lists
of 1 to 2,049 records (mask words of 32, tiles of 512 and 1,024 records), in
random order, with a smoothing length that varies by particle.  Device-resident
walks, dispatched walks and the filter are compared with the FP64 oracle at
relative L2 1e-5: FP32 sums of at most a few hundred terms of size u stay
within a few hundred x 2^-24 of their values, far below it.
"""
import ctypes as C

import numpy as np
import pytest

from tests.helpers import rel_l2
from tests.test_zz_no_alloc import pack
from weaklycompressiblesph_b200 import fdps
from weaklycompressiblesph_b200 import _native as N

pytestmark = pytest.mark.gpu
TOL = 1e-5
SIZES = [(1, 1), (1, 33), (31, 31), (32, 32), (33, 64), (64, 511), (31, 512), (96, 513), (128, 1023), (129, 1024),
         (32, 1025), (65, 2049), (2, 160)]


def walks(vary_h, min_j=1):
    """(Walks, EPI, EPJ): walk w holds the n_i / n_j lattice particles nearest its own origin, shuffled."""
    rng = np.random.default_rng(17)
    ei, ej = [], []
    for n_i, n_j in SIZES:
        g = np.stack(np.meshgrid(*[np.arange(-8, 9)] * 3, indexing="ij"), -1).reshape(-1, 3) * 0.05
        pos = g + rng.uniform(-0.01, 0.01, g.shape)
        n = len(pos)
        order = np.argsort(np.linalg.norm(pos, axis=1))
        pos = pos[order] + rng.uniform(-1, 1, 3)
        e = np.zeros(n, fdps.EPJ_HYDRO)
        e["pos"] = pos
        e["vel"] = rng.normal(0, 0.3, (n, 3))
        e["dens"] = 1000.0 * rng.uniform(0.98, 1.02, n)
        e["mass"] = 1000.0 * 0.05**3
        e["smth"] = 0.06 * (rng.uniform(0.9, 1.1, n) if vary_h else 1.0)
        e["snds"] = 20.0 * rng.uniform(0.95, 1.05, n)
        e["pres"] = rng.uniform(0.0, 4.0e4, n)
        e["visc"] = 1.0e-3
        pick = rng.permutation(max(n_j, min_j))
        i = np.zeros(n_i, fdps.EPI_HYDRO)
        for f in i.dtype.names:
            if f in e.dtype.names:
                i[f] = e[f][:n_i]
        ei.append(i)
        ej.append(e[pick])
    n_i, n_j = [len(x) for x in ei], [len(x) for x in ej]
    off = lambda c: np.concatenate([[0], np.cumsum(c)])
    epi, epj = np.concatenate(ei), np.concatenate(ej)
    return fdps.Walks(np.arange(len(epi)), off(n_i), np.arange(len(epj)), off(n_j)), epi, epj


@pytest.mark.parametrize("vary_h", [False, True])
@pytest.mark.parametrize("kind", ["reference_gpu", "reference_cpu"])
def test_hydro_walks(native, oracle_lib, kind, vary_h):
    import torch

    w, epi, epj = walks(vary_h)
    pair = fdps.pair_params(kind)
    want = oracle_lib.hydro_walks(w.i_off, epi, w.j_off, epj,
                                  oracle_lib.PairParams(pair.alpha, pair.beta, pair.c_cfl, pair.eps, pair.vsig_mode,
                                                        pair.grad_mode))
    fdps.configure(pair)
    got = np.zeros(len(epi), fdps.RESULT_HYDRO)
    fdps.calc_force_multiwalk(w, epi, epj, got)
    assert rel_l2(got["acc"], want["acc"]) < TOL
    assert rel_l2(got["div_v"], want["div_v"]) < TOL
    np.testing.assert_allclose(got["dt"], want["dt"], rtol=TOL)

    dev = torch.device("cuda", 0)
    t = [torch.from_numpy(x.reshape(-1)).to(dev) for x in pack(w, epi, epj)]
    out = torch.full((len(epi) * 8,), float("nan"), device=dev)
    stream = torch.cuda.current_stream(dev).cuda_stream
    N.call("wcsph_hydro_walks_noalloc", w.n_walk, *(C.c_void_p(x.data_ptr()) for x in t), C.c_void_p(out.data_ptr()),
           C.byref(pair), C.c_void_p(stream))
    out = out.cpu().numpy().reshape(-1, 2, 4)
    assert rel_l2(out[:, 0, :3], want["acc"]) < TOL
    assert rel_l2(out[:, 0, 3], want["div_v"]) < TOL
    np.testing.assert_allclose(out[:, 1, 0], want["dt"], rtol=TOL)


@pytest.mark.parametrize("vary_h", [False, True])
def test_filter_walks(native, oracle_lib, vary_h):
    w, epi, epj = walks(vary_h, min_j=129)  # every i is in its walk's j-list
    epi_f = np.zeros(len(epi), fdps.EPI_FILTER)
    epi_f["pos"], epi_f["smth"] = epi["pos"], epi["smth"]
    epj_f = np.zeros(len(epj), fdps.EPJ_FILTER)
    for f in ("pos", "dens", "mass"):
        epj_f[f] = epj[f]
    out = np.zeros(len(epi), fdps.RESULT_FILTER)
    fdps.calc_force_multiwalk(w, epi_f, epj_f, out, kind="filter")
    np.testing.assert_allclose(out["dens"], oracle_lib.filter_walks(w.i_off, epi_f, w.j_off, epj_f), rtol=TOL)
    # a NaN weight anywhere in a j-list reaches every i of the walk, in support or not
    far = np.asarray(w.j_off[1:]) - 1
    epj_f["mass"][far[11]] = np.nan
    fdps.calc_force_multiwalk(w, epi_f, epj_f, out, kind="filter")
    lo, hi = w.i_off[11], w.i_off[12]
    assert np.all(np.isnan(out["dens"][lo:hi])) and not np.any(np.isnan(np.delete(out["dens"], slice(lo, hi))))
