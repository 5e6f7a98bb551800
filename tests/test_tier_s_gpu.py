"""The sample-per-CTA kernel at the edges of its layouts, against the oracle:
rasters, potentials and counts equal bit for bit.  Weights lie on a 2^-12 grid
small enough that every sum is exact in any order, so ATOMIC delivery has one
result too."""
import numpy as np
import pytest

from oracle import oracle as O
from snc_b200 import runtime as R
from snc_b200 import workloads as W

pytestmark = pytest.mark.gpu

CASES = {
    # name: (n_in, n_hid, n_out, p, max_delay, samples, steps, rate)
    "one_warp": (6, 9, 2, 0.5, 3, 3, 20, 0.4),
    "one_chunk_exact": (300, 700, 24, 0.02, 5, 2, 12, 0.2),       # N = 1024: one neuron a thread
    "two_chunks": (500, 700, 9, 0.03, 7, 2, 12, 0.2),
    "four_chunks": (2400, 500, 11, 0.02, 9, 2, 10, 0.1),
    "state_in_shared": (4300, 200, 5, 0.02, 6, 2, 10, 0.1),
    "staged_in_rounds": (1500, 300, 8, 0.05, 6, 2, 8, 0.5),       # more than 256 fired rows a step
    "long_segments": (600, 300, 8, 0.9, 4, 1, 6, 0.6),            # more than 1024 events of a warp's batch
    "tags_per_warp": (150, 560, 8, 0.06, 68, 2, 80, 0.1),         # too many cells for a tag each
    "brimful": (40, 330, 10, 0.1, 149, 2, 160, 0.2),              # no room for scratch
    "cluster": (500, 700, 9, 0.12, 9, 3, 15, 0.1),                # 80,000 synapses and more
    "cluster_large": (2400, 600, 9, 0.06, 5, 2, 8, 0.15),
    "hubs": (700, 3, 2, 1.0, 2, 2, 10, 0.5),                      # hundreds of events a cell
}


# few samples run a cluster of CTAs each, many a CTA each
@pytest.mark.parametrize("many", [False, True])
@pytest.mark.parametrize("mode", [R.MODE_SORT, R.MODE_ATOMIC])
@pytest.mark.parametrize("name", sorted(CASES))
def test_layout(name, mode, many):
    n_in, n_hid, n_out, p, max_delay, samples, steps, rate = CASES[name]
    if many:
        samples, steps = 40, max(2, steps // 4)
    g = W.random_graph(5, n_in=n_in, n_hid=n_hid, n_out=n_out, p=p, max_delay=max_delay)
    scale = min(1.0, 8.0 / max(1.0, g.num_synapses / g.num_neurons))
    g.weights[:] = np.rint(g.weights * scale * 4096.0) / 4096.0
    ev, t = W.random_events(7, g, samples, np.arange(steps, steps + samples), rate=rate, amp_jitter=False)
    ev["amplitude"] = np.rint(ev["amplitude"] * 4.0) / 4.0
    lif = R.LIFParams(threshold=1.0, decay=0.9, reset=0.0, refractory=1)
    dg = R.DeviceGraph(g)
    di = R.DeviceInputs(dg, ev, t)
    run = R.Run(dg, di, raster=True, vfinal=True)
    run.configure(tier=0, mode=mode)
    ref = O.forward_batched(g, ev, t, lif)
    assert ref["spikes"].sum() > 0
    for _ in range(2):
        run.launch(lif, mode=mode)
        out = run.fetch(raster=True, vfinal=True)
        for k in ("spikes", "events", "logits", "raster"):
            np.testing.assert_array_equal(out[k], ref[k], err_msg=k)
        np.testing.assert_array_equal(out["v"].view(np.uint32), ref["v"].view(np.uint32))
