"""The L1 roofline of the list pass: its minimum counts only the loads that the
measured counter sees, so that the fraction is one of a bound."""
import json
import os

import pytest

import bench

L1 = json.load(open(os.path.join(os.path.dirname(bench.__file__), "profiles", "hydro_list_l1.json")))


@pytest.mark.parametrize("prec", ["tiled", "half2"])
def test_l1_fraction_is_at_most_one(prec):
    r = L1[f"dam1m/{prec}"]
    out = bench.l1_roofline("dam1m", prec, {"lists": {"entries": r["entries"]}, "pairs_per_step": 0.875 * r["entries"]})
    assert out["min_wavefronts_per_launch"] * 128 == r["entries"] * (r["list_word_bytes"] + r["record_bytes"])
    assert 0.0 < out["frac"] <= 1.0
