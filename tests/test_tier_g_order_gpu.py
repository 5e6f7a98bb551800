"""Waves of several samples on the all-SM kernel with weights whose sums depend
on their order (SORT), and where most neuron blocks receive nothing in most
steps: a sample that brings a block no events is followed at once by the next
one.  Equal to the oracle bit for bit, launch after launch."""
import numpy as np
import pytest

from oracle import oracle as O
from snc_b200 import runtime as R
from snc_b200 import workloads as W

pytestmark = pytest.mark.gpu

CASES = {
    # name: (n_in, n_hid, p, max_delay, rate)
    "quiet": (3000, 2500, 0.002, 3, 0.004),
    "few": (60, 200, 0.05, 6, 0.1),
    "ranked": (900, 500, 0.1, 5, 0.12),    # 64 to 256 descriptors
    "scanned": (900, 500, 0.1, 5, 0.5),    # more than 256
    "hubs": (300, 6, 1.0, 2, 0.5),         # long segments of few columns
}


@pytest.mark.parametrize("steps", [[9, 14], [12, 0, 7, 16, 5], [6, 11, 3, 8, 8, 2, 10, 4, 9, 12, 7, 5, 9]])
@pytest.mark.parametrize("name", sorted(CASES))
def test_wave(name, steps):
    n_in, n_hid, p, max_delay, rate = CASES[name]
    g = W.random_graph(11, n_in=n_in, n_hid=n_hid, n_out=5, p=p, max_delay=max_delay)
    g.weights[:] *= np.float32(min(1.0, 8.0 / max(1.0, g.num_synapses / g.num_neurons)))
    ev, t = W.random_events(12, g, len(steps), steps, rate=rate)
    lif = R.LIFParams(threshold=1.0, decay=0.9, reset=0.0, refractory=1, reset_mode=1)
    ref = O.forward_batched(g, ev, t, lif)
    assert ref["spikes"].sum() > 0
    dg = R.DeviceGraph(g)
    di = R.DeviceInputs(dg, ev, t)
    run = R.Run(dg, di, raster=True, vfinal=True, force_grid=True)
    for _ in range(5):
        run.launch(lif, mode=R.MODE_SORT)
        out = run.fetch(raster=True, vfinal=True)
        for k in ("spikes", "events", "logits", "raster"):
            np.testing.assert_array_equal(out[k], ref[k], err_msg=k)
        np.testing.assert_array_equal(out["v"].view(np.uint32), ref["v"].view(np.uint32))
