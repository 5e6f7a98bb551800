"""The sample-per-CTA kernel at the edges of its layouts with weights whose sums
depend on their order (SORT): rasters, potentials and counts equal the oracle's
bit for bit.  Few samples run on clusters where the net is large enough, many in
one CTA each."""
import numpy as np
import pytest

from oracle import oracle as O
from snc_b200 import runtime as R
from snc_b200 import workloads as W
from tests.test_tier_s_gpu import CASES

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("many", [False, True])
@pytest.mark.parametrize("name", sorted(CASES))
def test_layout(name, many):
    n_in, n_hid, n_out, p, max_delay, samples, steps, rate = CASES[name]
    if many:
        samples, steps = 40, max(2, steps // 4)
    g = W.random_graph(5, n_in=n_in, n_hid=n_hid, n_out=n_out, p=p, max_delay=max_delay)
    g.weights[:] *= np.float32(min(1.0, 8.0 / max(1.0, g.num_synapses / g.num_neurons)))
    ev, t = W.random_events(7, g, samples, np.arange(steps, steps + samples), rate=rate)
    lif = R.LIFParams(threshold=1.0, decay=0.9, reset=0.0, refractory=1)
    dg = R.DeviceGraph(g)
    di = R.DeviceInputs(dg, ev, t)
    run = R.Run(dg, di, raster=True, vfinal=True)
    run.configure(tier=0, mode=R.MODE_SORT)
    ref = O.forward_batched(g, ev, t, lif)
    assert ref["spikes"].sum() > 0
    for _ in range(2):
        run.launch(lif, mode=R.MODE_SORT)
        out = run.fetch(raster=True, vfinal=True)
        for k in ("spikes", "events", "logits", "raster"):
            np.testing.assert_array_equal(out[k], ref[k], err_msg=k)
        np.testing.assert_array_equal(out["v"].view(np.uint32), ref["v"].view(np.uint32))
