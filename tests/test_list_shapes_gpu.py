"""The list pass's launch shapes are timed within one summation order, chosen by
size: what the autotuner picks follows the rule on waves of blocks, at sizes on
both sides of its lines, and two tuned solvers agree to the bit."""
import numpy as np
import pytest

from weaklycompressiblesph_b200 import _native as N
from weaklycompressiblesph_b200 import cases
from weaklycompressiblesph_b200.sim import Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [N.PREC_TILED, N.PREC_HALF2], ids=["tiled", "half2"])
@pytest.mark.parametrize("side", [10, 36, 40, 47, 50])
def test_tuned_shape_follows_the_rule(side, prec, native):
    import torch

    case = cases.periodic_lattice(n_side=side, dx=0.01, seed=6)
    slots = 5 * torch.cuda.get_device_properties(0).multi_processor_count
    blocks = -(-case.n // 128)
    w1, w2 = -(-blocks // slots), -(-2 * blocks // slots)
    two = 4 * w2 < 5 * w1 if prec == N.PREC_TILED else 3 * w2 < 5 * w1
    got = []
    for _ in range(2):
        with Solver(case.n, precision=prec, list_interval=30) as s:
            k = s.add(case)
            s.step(6)
            assert s.tuning()["list_shape"] in ((1, 3) if two else (0, 2, 4))
            got.append(s.read(k))
    for f in ("pos", "vel", "dens", "acc", "div_v"):
        np.testing.assert_array_equal(got[0][f], got[1][f])
