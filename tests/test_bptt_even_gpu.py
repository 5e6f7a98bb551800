"""Resident BPTT launches over nets whose neurons have equally many synapses,
which deal the neurons to the CTAs in order: the last CTA partial, one and
several batch slices.  The same bits as the global-memory form, and the CPU
autograd restatement's spikes and gradients (within 1e-4 of the largest)."""
import numpy as np
import pytest
import torch

from oracle import bptt_ref as BR
from tests.test_bptt_resident_gpu import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,fan,B", [(31, 4, 5), (160, 8, 33), (1500, 6, 70), (2500, 6, 50)])
def test_ring(n, fan, B):
    rng = np.random.default_rng(n)
    off = rng.permutation(np.arange(1, 31))[:fan]
    pre = np.repeat(np.arange(n), fan)
    post = (pre + np.tile(off, n)) % n
    d = rng.integers(1, 4, pre.shape[0])
    w = rng.normal(0, 0.9 / np.sqrt(fan), pre.shape[0]).astype(np.float32)
    gen = torch.Generator().manual_seed(B)
    ext = (torch.rand(6, B, n, generator=gen) < 0.3).float() * 1.1
    proj = torch.randn(6, B, n, generator=gen)
    wr = torch.as_tensor(w).requires_grad_(True)
    er = ext.clone().requires_grad_(True)
    s_ref = BR.core_forward(wr, er, *[torch.as_tensor(x).long() for x in (pre, post, d)], 1.0, 0.9, 15.0)
    (s_ref * proj).sum().backward()
    got = _run(n, pre, post, d, w, ext, proj, 4, True)
    other = _run(n, pre, post, d, w, ext, proj, 4, False)
    assert s_ref.sum() > 0
    assert torch.equal(got[0], s_ref.detach())
    for x, y in zip(got[1:], (wr.grad, er.grad)):
        assert float((x - y).abs().max()) <= 1e-4 * float(y.abs().max())
    for x, y in zip(got, other):
        assert torch.equal(x, y)
