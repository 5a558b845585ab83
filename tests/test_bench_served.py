"""The plain path's side of the served benchmark (bench.plain_rate_at), on CPU: the
rate that it sustains at a p99, and none where no rate has that p99, for which the
bench then reports no ratio."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402

LAT_MS = np.linspace(0.5, 2.0, 200)


@pytest.mark.parametrize("p99", [0.4, 1.9])
def test_no_rate_below_the_service_times(p99):
    assert bench.plain_rate_at(LAT_MS, p99, 800.0) is None


def test_rate_at_a_p99_that_queueing_reaches():
    r = bench.plain_rate_at(LAT_MS, 6.0, 800.0)
    assert 100.0 < r < 800.0
    assert bench.plain_open_loop(LAT_MS, r)["p99_ms"] <= 6.0
    assert bench.plain_rate_at(LAT_MS, 12.0, 800.0) >= r
