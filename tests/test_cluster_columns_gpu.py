"""Nets of 80,000 synapses and more whose neurons with incoming synapses all lie
in every fourth word of 32 neurons: a cluster of four CTAs a sample would leave
one of them all ring columns, more than fit beside the delivery's working
arrays.  They run in one CTA, forward and e-prop, equal to the oracle bit for
bit."""
import numpy as np
import pytest

from oracle import oracle as O
from snc_b200 import eprop as E
from snc_b200 import runtime as R
from snc_b200 import workloads as W
from snc_b200.graph import INPUT, INTERNAL, OUTPUT, SNNGraph

pytestmark = pytest.mark.gpu


def _graph(n, fan_out, max_delay, stride=4, w_std=1.5):
    """Inputs in the words without columns, hidden and 10 outputs in the others."""
    rng = np.random.default_rng(n)
    ids = np.arange(n)
    col = (ids // 32) % stride == 0
    cols = ids[col]
    pre = np.repeat(ids, fan_out)
    post = cols[rng.integers(0, cols.shape[0], pre.shape[0])]
    role = np.where(col, INTERNAL, INPUT).astype(np.uint8)
    role[cols[-10:]] = OUTPUT
    channel = np.full(n, -1, np.int32)
    channel[~col] = np.arange((~col).sum())
    channel[cols[-10:]] = np.arange(10)
    w = np.abs(rng.normal(0, w_std / np.sqrt(fan_out * n / cols.shape[0]), pre.shape[0])).astype(np.float32)
    sign = np.where(rng.random(n) < 0.4, -1, 1).astype(np.int8)
    d = rng.integers(1, max_delay + 1, pre.shape[0]).astype(np.int32)
    d[0] = max_delay
    return SNNGraph(n, np.arange(0, n * fan_out + 1, fan_out, dtype=np.int32), post.astype(np.int32), w, d,
                    role, sign, channel)


@pytest.mark.parametrize("n,fan_out,max_delay", [(2048, 40, 81), (1024, 80, 187)])
def test_forward(n, fan_out, max_delay):
    g = _graph(n, fan_out, max_delay)
    assert g.num_synapses >= 80000
    ev, t = W.random_events(7, g, 3, [max_delay + 20, 40, max_delay + 3], rate=0.05)
    lif = R.LIFParams(threshold=1.0, decay=0.9, reset=0.0, refractory=1)
    ref = O.forward_batched(g, ev, t, lif)
    assert ref["logits"].sum() > 20
    dg = R.DeviceGraph(g)
    di = R.DeviceInputs(dg, ev, t)
    run = R.Run(dg, di, raster=True, vfinal=True)
    run.configure(tier=0, mode=R.MODE_SORT)
    run.launch(lif, mode=R.MODE_SORT)
    out = run.fetch(raster=True, vfinal=True)
    for k in ("spikes", "events", "logits", "raster"):
        np.testing.assert_array_equal(out[k], ref[k], err_msg=k)
    np.testing.assert_array_equal(out["v"].view(np.uint32), ref["v"].view(np.uint32))


def test_eprop():
    g = _graph(1024, 80, 182)
    rng = np.random.default_rng(1)
    steps = np.array([200, 30], np.int32)
    ev, t = W.random_events(8, g, 2, steps, rate=0.03)
    labels = np.array([3, 7], np.int32)
    fb = rng.normal(0, 1.0, (int((g.role == INTERNAL).sum()), 10)).astype(np.float32)
    w0 = (g.weights * g.sign[g.pre_ids()]).astype(np.float32)
    lif = R.LIFParams(threshold=1.0, decay=0.9, reset=0.0, refractory=1)
    cfg = E.TrainConfig(lif=lif, lr=0.5, w_max=4.0, surrogate_scale=0.3, trace_decay=0.95)
    s = E.CudaTrainSession(g, cfg, batch=4, weights=w0, feedback=fb)
    assert not s.uses_grid()
    out = s.run_batch(ev, t, labels, train=True)
    ref = O.eprop_batch(g, w0, ev, t, lif, trace_decay=0.95, gamma=0.3, lr=0.5, w_max=4.0,
                        train_hidden=True, bmat=fb, labels=labels, want_elig=True)
    np.testing.assert_array_equal(out["counts"], ref["counts"])
    assert out["spikes"] == ref["spikes"] > 0 and out["events"] == ref["events"]
    np.testing.assert_array_equal(s.eligibility(2).view(np.uint32), ref["elig"].view(np.uint32))
