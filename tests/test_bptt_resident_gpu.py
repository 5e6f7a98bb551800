"""The resident BPTT launches at the edges of their shapes: batch slices of 1,
2 and 4 words, batches whose last word or slice is partial (65 to 96 samples
take three words), in-degrees beyond the groups held at once, delay-1-only
graphs, no out-edges.  Forward spikes equal the CPU autograd restatement bit
for bit, gradients within 1e-4 of the largest, and the global-memory form
gives the same bits throughout."""
import numpy as np
import pytest
import torch

from oracle import bptt_ref as BR
from snc_b200 import bptt as BP

pytestmark = pytest.mark.gpu

CASES = {
    # name: (N, mean in-degree, max delay, hub in-degree, T, B, ckpt)
    "one_word": (60, 9, 4, 0, 11, 20, 3),
    "partial_third_word": (90, 12, 3, 0, 9, 70, 4),
    "five_slices": (80, 10, 5, 0, 7, 140, 0),
    "eight_slices": (50, 8, 2, 0, 6, 256, 4),
    "two_words": (2500, 6, 3, 180, 5, 50, 2),
    "two_words_two_slices": (1300, 7, 3, 170, 5, 100, 3),
    "four_words": (2450, 5, 2, 130, 4, 128, 3),
    "four_words_partial": (2450, 5, 2, 100, 4, 97, 0),
    "delay_one": (70, 40, 1, 0, 12, 33, 5),
    "hub_of_eight_groups": (300, 6, 1, 250, 8, 32, 10),
}


def _run(n, pre, post, d, w, ext, proj, ckpt, resident):
    core = BP.SpikingCore(n, pre, post, d, device="cuda")
    core.set_resident(resident)
    wt = torch.as_tensor(w, device="cuda").requires_grad_(True)
    et = ext.cuda().requires_grad_(True)
    s = BP.spiking_core(wt, et, core, 1.0, 0.9, 15.0, ckpt)
    gw, ge = torch.autograd.grad(s, (wt, et), proj.cuda())
    return [x.detach().cpu() for x in (s, gw, ge)]


@pytest.mark.parametrize("name", sorted(CASES))
def test_shapes(name):
    n, deg, max_delay, hub, t, b, ckpt = CASES[name]
    rng = np.random.default_rng(len(name))
    # the last tenth of the neurons have no outgoing synapse, the first tenth
    # no incoming one
    pre = rng.integers(0, n - n // 10, n * deg)
    post = rng.integers(n // 10, n, n * deg)
    if hub:
        pre = np.concatenate([pre, rng.integers(0, n - n // 10, hub)])
        post = np.concatenate([post, np.full(hub, n - 1)])
    d = rng.integers(1, max_delay + 1, pre.shape[0])
    w = rng.normal(0, 0.9 / np.sqrt(deg), pre.shape[0]).astype(np.float32)
    gen = torch.Generator().manual_seed(b)
    ext = (torch.rand(t, b, n, generator=gen) < 0.3).float() * 1.1
    proj = torch.randn(t, b, n, generator=gen)
    wr = torch.as_tensor(w).requires_grad_(True)
    er = ext.clone().requires_grad_(True)
    # the restatement sums the edges of a neuron in CSR order
    order = np.argsort(pre, kind="stable")
    lt = [torch.as_tensor(x[order]).long() for x in (pre, post, d)]
    s_ref = BR.core_forward(wr[torch.as_tensor(order)], er, *lt, 1.0, 0.9, 15.0)
    (s_ref * proj).sum().backward()
    got = _run(n, pre, post, d, w, ext, proj, ckpt, True)
    other = _run(n, pre, post, d, w, ext, proj, ckpt, False)
    assert s_ref.sum() > 0
    assert torch.equal(got[0], s_ref.detach())
    for x, y in zip(got[1:], (wr.grad, er.grad)):
        assert float((x - y).abs().max()) <= 1e-4 * float(y.abs().max())
    for x, y in zip(got, other):
        np.testing.assert_array_equal(x.numpy().view(np.uint32), y.numpy().view(np.uint32))
