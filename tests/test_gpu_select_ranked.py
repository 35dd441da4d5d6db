"""The selector's gain on the timings of the present kernels (select_timings_ranked.npz)."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_selector_gains_on_the_present_timings():
    import bench
    res = bench.select_leg()
    assert "select_timings_ranked" in res["data"]
    pol = res["policies"]
    assert pol["learned"]["ms"] < pol["cost_function"]["ms"], pol
    assert pol["learned"]["ms"] <= pol["fixed_default"]["ms"], pol


def test_same_graphs_as_the_earlier_timings():
    here = os.path.dirname(os.path.abspath(__file__))
    new, old = (np.load(os.path.join(here, "golden", "select_timings%s.npz" % x)) for x in ("_ranked", ""))
    assert np.allclose(new["features"], old["features"]) and new["times_ms"].shape == old["times_ms"].shape
