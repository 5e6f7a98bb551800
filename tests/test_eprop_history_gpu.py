"""Minibatches whose surrogate history exceeds its limit accumulate their
eligibility in the forward: the same bits as the CPU restatement, on nets whose
samples otherwise run on a cluster of CTAs (80,000 synapses and more) as on
those of one CTA, before and after minibatches that keep the history."""
import numpy as np
import pytest

from oracle import oracle as O
from snc_b200 import eprop as E
from snc_b200 import runtime as R
from snc_b200 import workloads as W
from snc_b200.graph import INTERNAL

pytestmark = pytest.mark.gpu

GRAPHS = {
    "one_cta": dict(n_in=30, n_hid=90, n_out=5, p=0.15, max_delay=6),
    "cluster": dict(n_in=500, n_hid=700, n_out=9, p=0.12, max_delay=9),
    "cluster_many_neurons": dict(n_in=2400, n_hid=600, n_out=9, p=0.06, max_delay=5),
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_history_limit(name):
    g = W.random_graph(11, **GRAPHS[name])
    assert (g.num_synapses >= 80000) == name.startswith("cluster")
    steps = np.array([14, 33, 20], np.int32)
    rng = np.random.default_rng(12)
    w0 = rng.normal(0, 4.0 / np.sqrt(g.num_synapses / g.num_neurons), g.num_synapses).astype(np.float32)
    fb = rng.normal(0, 1.0, (int((g.role == INTERNAL).sum()), g.num_output_channels)).astype(np.float32)
    lif = R.LIFParams(threshold=1.0, decay=0.9, reset=0.0, refractory=1)
    cfg = E.TrainConfig(lif=lif, lr=0.5, w_max=4.0, surrogate_scale=0.3, trace_decay=0.95)
    s = E.CudaTrainSession(g, cfg, batch=4, weights=w0, feedback=fb)
    assert not s.uses_grid()
    for k, limit in enumerate([1, 0, 1, 1]):
        ev, st = W.random_events(20 + k, g, 3, steps, rate=0.1)
        labels = rng.integers(0, g.num_output_channels, 3).astype(np.int32)
        w = s.get_weights()
        ref = O.eprop_batch(g, w, ev, st, lif, trace_decay=0.95, gamma=0.3, lr=0.5, w_max=4.0,
                            train_hidden=True, bmat=fb, labels=labels, want_elig=True)
        s.set_history_limit(limit)
        out = s.run_batch(ev, st, labels, train=True)
        np.testing.assert_array_equal(out["counts"], ref["counts"])
        assert out["spikes"] == ref["spikes"] > 0 and out["events"] == ref["events"]
        el = s.eligibility(3)
        assert np.count_nonzero(el) > el.size // 20
        np.testing.assert_array_equal(el.view(np.uint32), ref["elig"].view(np.uint32))
        assert np.abs(s.get_weights() - w).max() > 0
        np.testing.assert_allclose(s.get_weights(), ref["w"], rtol=1e-5, atol=1e-6)


def test_gradient_beyond_the_limit():
    import torch
    g = W.random_graph(11, **GRAPHS["cluster"])
    rng = np.random.default_rng(3)
    fb = rng.normal(0, 1.0, (int((g.role == INTERNAL).sum()), g.num_output_channels)).astype(np.float32)
    w0 = rng.normal(0, 0.4, g.num_synapses).astype(np.float32)
    cfg = E.TrainConfig(lif=R.LIFParams(), lr=0.5, trace_decay=0.95)
    s = E.CudaTrainSession(g, cfg, batch=4, weights=w0, feedback=fb)
    ev, st = W.random_events(21, g, 3, [25, 12, 30], rate=0.1)
    labels = rng.integers(0, g.num_output_channels, 3).astype(np.int32)
    got = []
    for limit in (0, 1):
        s.set_history_limit(limit)
        grad = torch.zeros(g.num_synapses, device="cuda")
        s.gradient(ev, st, labels, grad)
        got.append(grad.cpu().numpy())
    assert np.count_nonzero(got[0])
    np.testing.assert_array_equal(got[0].view(np.uint32), got[1].view(np.uint32))
