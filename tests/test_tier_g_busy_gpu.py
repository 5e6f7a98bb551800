"""Waves of several samples whose blocks receive hundreds of descriptors a step,
more than two for each thread of a group and up to what a block holds at once,
with weights whose sums depend on their order: equal to the oracle bit for bit."""
import numpy as np
import pytest

from oracle import oracle as O
from snc_b200 import runtime as R
from snc_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("samples", [2, 3, 6])
@pytest.mark.parametrize("rate", [0.1, 0.3, 0.8])
def test_busy(rate, samples):
    g = W.random_graph(5, n_in=1500, n_hid=4000, n_out=10, p=0.02, max_delay=4)
    g.weights[:] *= np.float32(8.0 / (g.num_synapses / g.num_neurons))
    steps = np.arange(samples, dtype=np.int32) % 3 + 7
    ev, t = W.random_events(7, g, samples, steps, rate=rate)
    lif = R.LIFParams(threshold=1.0, decay=0.9, reset=0.0, refractory=1)
    ref = O.forward_batched(g, ev, t, lif)
    assert (ref["spikes"] > 200 * steps * rate).all()
    dg = R.DeviceGraph(g)
    di = R.DeviceInputs(dg, ev, t)
    run = R.Run(dg, di, raster=True, vfinal=True, force_grid=True)
    run.launch(lif, mode=R.MODE_SORT)
    out = run.fetch(raster=True, vfinal=True)
    for k in ("spikes", "events", "logits", "raster"):
        np.testing.assert_array_equal(out[k], ref[k], err_msg=k)
    np.testing.assert_array_equal(out["v"].view(np.uint32), ref["v"].view(np.uint32))
