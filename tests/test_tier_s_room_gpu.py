"""The ordered sample-per-CTA delivery beside states that leave little shared
memory: few staged rows and few tags a warp, more fired rows than are staged at
once, weights whose sums depend on their order.  Equal to the oracle bit for
bit."""
import numpy as np
import pytest

from oracle import oracle as O
from snc_b200 import runtime as R
from snc_b200 import workloads as W

pytestmark = pytest.mark.gpu

CASES = {
    # name: (n_in, n_hid, n_out, ring slots, rate, weight gain)
    "64_rows_512_tags": (40, 330, 10, 141, 0.3, 16.0),
    "64_rows_256_tags": (40, 330, 10, 147, 0.3, 16.0),
    "32_rows_256_tags": (40, 330, 10, 151, 0.3, 16.0),
    "32_rows_128_tags": (5, 205, 5, 250, 0.9, 300.0),
}


@pytest.mark.parametrize("p", [0.12, 0.7])
@pytest.mark.parametrize("name", sorted(CASES))
def test_room(name, p):
    n_in, n_hid, n_out, slots, rate, gain = CASES[name]
    g = W.random_graph(9, n_in=n_in, n_hid=n_hid, n_out=n_out, p=p, max_delay=slots - 1)
    g.delays[0] = slots - 1
    g.weights[:] *= np.float32(min(4.0, gain / (g.num_synapses / g.num_neurons)))
    assert np.unique(g.post_ids).shape[0] == n_hid + n_out
    ev, t = W.random_events(3, g, 3, [slots + 40, 30, slots - 5], rate=rate)
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
