"""v_sig of the GPU variant over a walk: the largest exact quotient, on the
device-resident walks as on the dispatched ones, at any scale of lengths.

Many j lie at one distance and approach at one speed, so that their quotients
-mu differ in the last bits only, out of the support as well as in it.  Both
paths round every quotient alike and take the largest, so their dt agree to
the bit; against the FP64 oracle within 20 x 2^-24, the roundings of one dt (7
in the numerator of mu, 7 in its denominator, the quotient, 4 in dt)."""
import ctypes as C

import numpy as np
import pytest

from tests.test_zz_no_alloc import pack
from weaklycompressiblesph_b200 import _native as N
from weaklycompressiblesph_b200 import fdps

pytestmark = pytest.mark.gpu


def near_ties(scale, n_walk=64, n_i=32, n_j=700, seed=5):
    """Walks of n_i particles near the origin and n_j on a shell that closes in at nearly the same rate."""
    rng = np.random.default_rng(seed)
    h = 0.06 * scale
    ei, ej = np.zeros(n_walk * n_i, fdps.EPI_HYDRO), np.zeros(n_walk * n_j, fdps.EPJ_HYDRO)
    for e, n in ((ei, n_i), (ej, n_j)):
        e["dens"] = 1000.0 * rng.uniform(0.98, 1.02, len(e))
        e["smth"], e["visc"] = h, 1.0e-3
        e["snds"] = rng.uniform(0.01, 0.02, len(e))  # small beside v_sig, so that dt shows its last bits
        e["pres"] = rng.uniform(0.0, 4.0e4, len(e))
    ei["pos"] = rng.uniform(-1e-9, 1e-9, (len(ei), 3)) * h
    u = rng.normal(size=(len(ej), 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    radius = np.repeat(rng.uniform(0.5, 6.0, n_walk), n_j)[:, None] * h
    ej["pos"], ej["vel"] = u * radius, -u * radius / h * rng.uniform(0.9, 1.1, n_walk).repeat(n_j)[:, None]
    ej["mass"] = 1000.0 * (h / 1.2) ** 3
    off = lambda n: np.arange(n_walk + 1) * n  # noqa: E731
    return fdps.Walks(np.arange(len(ei)), off(n_i), np.arange(len(ej)), off(n_j)), ei, ej


@pytest.mark.parametrize("scale", [2.0 ** -18, 1.0, 2.0 ** 24])
@pytest.mark.parametrize("eps", [0.01, 0.0])
def test_vsig_is_the_largest_exact_quotient(native, oracle_lib, scale, eps):
    import torch

    w, epi, epj = near_ties(scale)
    pair = fdps.pair_params("reference_gpu", eps=eps)
    fdps.configure(pair)
    got = np.zeros(len(epi), fdps.RESULT_HYDRO)
    fdps.calc_force_multiwalk(w, epi, epj, got)
    dev = torch.device("cuda", 0)
    t = [torch.from_numpy(x.reshape(-1)).to(dev) for x in pack(w, epi, epj)]
    out = torch.full((len(epi) * 8,), float("nan"), device=dev)
    N.call("wcsph_hydro_walks_noalloc", w.n_walk, *(C.c_void_p(x.data_ptr()) for x in t), C.c_void_p(out.data_ptr()),
           C.byref(pair), C.c_void_p(torch.cuda.current_stream(dev).cuda_stream))
    dt = out.cpu().numpy().reshape(-1, 2, 4)[:, 1, 0]
    want = oracle_lib.hydro_walks(w.i_off, epi, w.j_off, epj,
                                  oracle_lib.PairParams(pair.alpha, pair.beta, pair.c_cfl, pair.eps, pair.vsig_mode,
                                                        pair.grad_mode))
    np.testing.assert_allclose(dt, want["dt"], rtol=20 * 2.0 ** -24)
    np.testing.assert_array_equal(dt, got["dt"].astype(np.float32))


def test_particles_at_one_place_have_no_vsig(native):
    """r^2 = 0, be it that the squares underflow: no pair, though the particles approach (eps 0: a quotient by zero)."""
    import torch

    w, epi, epj = near_ties(1.0, n_walk=1, n_i=1, n_j=40)
    epi["pos"] = 0.0
    epj["vel"] = 0.0
    epj["pos"][7], epj["vel"][7] = [1.0e-25, 0.0, 0.0], [-5.0, 0.0, 0.0]
    pair = fdps.pair_params("reference_gpu", eps=0.0)
    dev = torch.device("cuda", 0)
    t = [torch.from_numpy(x.reshape(-1)).to(dev) for x in pack(w, epi, epj)]
    out = torch.full((8,), float("nan"), device=dev)
    N.call("wcsph_hydro_walks_noalloc", w.n_walk, *(C.c_void_p(x.data_ptr()) for x in t), C.c_void_p(out.data_ptr()),
           C.byref(pair), C.c_void_p(torch.cuda.current_stream(dev).cuda_stream))
    dt = out.cpu().numpy()[4]
    assert dt == np.float32(pair.c_cfl) * np.float32(epi["smth"][0]) / np.float32(epi["snds"][0])
