"""Batches around the number of clusters that the device holds at once (a cluster
of four CTAs a sample within it, one CTA a sample beyond): equal to the oracle
bit for bit, with weights whose sums depend on their order."""
import numpy as np
import pytest

from oracle import oracle as O
from snc_b200 import runtime as R
from snc_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("samples", [1, 31, 33, 34, 37, 38])
def test_samples(samples):
    g = W.random_graph(5, n_in=500, n_hid=700, n_out=9, p=0.12, max_delay=9)
    g.weights[:] *= np.float32(30.0 * g.num_neurons / g.num_synapses)
    assert g.num_synapses >= 80000
    ev, t = W.random_events(7, g, samples, np.arange(samples) % 5 + 14, rate=0.1)
    lif = R.LIFParams(threshold=1.0, decay=0.9, reset=0.0, refractory=1)
    ref = O.forward_batched(g, ev, t, lif)
    assert ref["logits"].sum() > 0
    dg = R.DeviceGraph(g)
    di = R.DeviceInputs(dg, ev, t)
    run = R.Run(dg, di, raster=True, vfinal=True)
    run.configure(tier=0, mode=R.MODE_SORT)
    run.launch(lif, mode=R.MODE_SORT)
    out = run.fetch(raster=True, vfinal=True)
    for k in ("spikes", "events", "logits", "raster"):
        np.testing.assert_array_equal(out[k], ref[k], err_msg=k)
    np.testing.assert_array_equal(out["v"].view(np.uint32), ref["v"].view(np.uint32))
