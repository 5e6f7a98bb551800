"""Schedules whose average step is small but whose large steps are neighbours, of
fewer and of more steps than the device holds CTAs, against the oracle's schedule
bit for bit."""
import numpy as np
import pytest

from tests.helpers import input_graph as _graph
from tests.test_schedule_gpu import _check, _events

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [
    [784] * 6 + [0] * 44,
    [1] * 100 + [129] * 40 + [128, 130, 2100] + [2] * 60,
    [0] * 700 + [150] * 90 + [3] * 2000,
    [90] * 8 * 148 + [300, 0, 300],
])
def test_bursts(sizes):
    rng = np.random.default_rng(len(sizes))
    rows = []
    for t, n in enumerate(sizes):
        rows += [(0, int(rng.integers(0, 12)), t, float(rng.standard_normal() * 10.0 ** int(rng.integers(-3, 4))))
                 for _ in range(n)]
    ev = _events([rows[i] for i in rng.permutation(len(rows))])
    _check(_graph(12), ev, np.array([len(sizes)], np.int32))
