"""The summation order of the list pass (one or two threads per particle) is a
rule on the solver's present size, whatever size it was tuned at."""
import pytest

from weaklycompressiblesph_b200 import _native as N
from weaklycompressiblesph_b200 import cases
from weaklycompressiblesph_b200.sim import Solver

pytestmark = pytest.mark.gpu


def two_threads(n, prec):
    import torch

    slots = 5 * torch.cuda.get_device_properties(0).multi_processor_count
    blocks = -(-n // 128)
    w1, w2 = -(-blocks // slots), -(-2 * blocks // slots)
    return 4 * w2 < 5 * w1 if prec == N.PREC_TILED else 3 * w2 < 5 * w1


@pytest.mark.parametrize("prec", [N.PREC_TILED, N.PREC_HALF2], ids=["tiled", "half2"])
@pytest.mark.parametrize("sides", [(33, 28), (45, 34)], ids=["36k-58k", "91k-130k"])
def test_order_follows_the_present_size(sides, prec, native):
    """Two sizes of one power of two: the solver is not tuned again in between."""
    a, b = (cases.periodic_lattice(n_side=k, dx=0.01, seed=k) for k in sides)
    with Solver(a.n + b.n, max_instances=2, precision=prec, list_interval=30) as s:
        n, buckets = 0, []
        for c in (a, b):
            s.add(c)
            n += c.n
            s.step(3)
            t = s.tuning()
            assert t["list_shape"] in ((1, 3) if two_threads(n, prec) else (0, 2, 4))
            buckets.append(t["bucket"])
        assert buckets[0] == buckets[1]
    with Solver(a.n, precision=prec, list_interval=30, list_shape=2) as s:  # a fixed shape stays
        s.add(a)
        s.step(3)
        assert s.tuning()["list_shape"] == 2
