"""Waves of several samples on the all-SM kernel, which takes them side by side
in groups of threads: few and many descriptors a block and step (the ranked and
the scanned deliveries), more samples than groups, uneven and empty samples.
Equal to the oracle bit for bit; the weights' sums are exact in any order, so
BUCKET and ATOMIC have one result too."""
import numpy as np
import pytest

from oracle import oracle as O
from snc_b200 import runtime as R
from snc_b200 import workloads as W

pytestmark = pytest.mark.gpu

CASES = {
    # name: (n_in, n_hid, p, max_delay, rate)
    "few": (60, 200, 0.05, 6, 0.1),
    "ranked": (900, 500, 0.1, 5, 0.12),    # 64 to 256 descriptors
    "scanned": (900, 500, 0.1, 5, 0.5),    # more than 256
    "hubs": (300, 6, 1.0, 2, 0.5),         # long segments of few columns
}


@pytest.mark.parametrize("mode", [R.MODE_SORT, R.MODE_BUCKET, R.MODE_ATOMIC])
@pytest.mark.parametrize("steps", [[9, 14], [12, 0, 7, 16, 5], [6, 11, 3, 8, 8, 2, 10, 4, 9]])
@pytest.mark.parametrize("name", sorted(CASES))
def test_wave(name, steps, mode):
    n_in, n_hid, p, max_delay, rate = CASES[name]
    g = W.random_graph(11, n_in=n_in, n_hid=n_hid, n_out=5, p=p, max_delay=max_delay)
    scale = min(1.0, 8.0 / max(1.0, g.num_synapses / g.num_neurons))
    g.weights[:] = np.rint(g.weights * scale * 4096.0) / 4096.0
    ev, t = W.random_events(12, g, len(steps), steps, rate=rate, amp_jitter=False)
    ev["amplitude"] = np.rint(ev["amplitude"] * 4.0) / 4.0
    lif = R.LIFParams(threshold=1.0, decay=0.9, reset=0.0, refractory=1, reset_mode=1)
    ref = O.forward_batched(g, ev, t, lif)
    assert ref["spikes"].sum() > 0
    dg = R.DeviceGraph(g)
    di = R.DeviceInputs(dg, ev, t)
    run = R.Run(dg, di, raster=True, vfinal=True, force_grid=True)
    for _ in range(2):
        run.launch(lif, mode=mode)
        out = run.fetch(raster=True, vfinal=True)
        for k in ("spikes", "events", "logits", "raster"):
            np.testing.assert_array_equal(out[k], ref[k], err_msg=k)
        np.testing.assert_array_equal(out["v"].view(np.uint32), ref["v"].view(np.uint32))
