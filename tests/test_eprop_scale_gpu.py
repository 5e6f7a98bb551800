"""Eligibility at surrogate scales of either sign, at the largest and beyond
every finite one, against the CPU restatement: a step whose trace is zero adds
nothing, whatever the surrogate is."""
import numpy as np
import pytest

from oracle import oracle as O
from snc_b200 import eprop as E
from snc_b200 import runtime as R
from tests.test_eprop_gpu import make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gamma", [-0.3, 3e38, float("inf")])
def test_scale(gamma):
    steps = [30, 33, 5]
    g, ev, st, w0, fb, labels = make_case(6, len(steps), steps)
    lif = R.LIFParams(threshold=1.0, decay=0.9, reset=0.0, refractory=1)
    cfg = E.TrainConfig(lif=lif, lr=0.5, w_max=4.0, surrogate_scale=gamma, trace_decay=0.95)
    s = E.CudaTrainSession(g, cfg, batch=4, weights=w0, feedback=fb)
    ref = O.eprop_batch(g, w0, ev, st, lif, trace_decay=0.95, gamma=gamma, lr=0.5, w_max=4.0,
                        train_hidden=True, bmat=fb, labels=labels, want_elig=True)
    out = s.run_batch(ev, st, labels, train=True)
    np.testing.assert_array_equal(out["counts"], ref["counts"])
    el = s.eligibility(len(steps))
    # with an infinite scale the restatement multiplies it by the zero of a
    # neuron far from threshold, which the kernels do not
    known = ~np.isnan(ref["elig"])
    assert np.abs(ref["elig"][known]).max() > 0 and (known.all() or np.isinf(gamma))
    np.testing.assert_array_equal(el[known], ref["elig"][known])
    assert not np.isnan(el).any()
