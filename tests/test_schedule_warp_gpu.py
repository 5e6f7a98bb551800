"""Schedules whose average step is small: a warp sorts and merges a step of at
most 128 entries by itself, and its CTA the steps above that.  Steps on both
sides of every edge of that split, and averages on both sides of the rule's
line (96 entries a step), against the oracle's schedule bit for bit."""
import numpy as np
import pytest

from tests.helpers import input_graph as _graph
from tests.test_schedule_gpu import _check, _events

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [
    [0, 1, 31, 32, 33, 63, 64, 65],
    [95, 96, 97, 127, 128, 0, 1, 2],       # at the line below, the largest of a warp
    [129, 0, 128, 0, 2100, 3] + [0] * 40,  # steps left to the CTA, one above its tile
    [96] * 9, [96] * 8 + [97],             # the two sides of the rule
    [200] + [1] * 3000,
])
def test_steps_of_few_entries(sizes):
    rng = np.random.default_rng(len(sizes))
    rows = []
    for t, n in enumerate(sizes):
        # few channels: runs of equal neurons whose sums depend on their order
        rows += [(0, int(rng.integers(0, 12)), t, float(rng.standard_normal() * 10.0 ** int(rng.integers(-3, 4))))
                 for _ in range(n)]
    ev = _events([rows[i] for i in rng.permutation(len(rows))])
    _check(_graph(12), ev, np.array([len(sizes), 0], np.int32))
