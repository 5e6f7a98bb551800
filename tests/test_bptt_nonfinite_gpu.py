"""Weights that are infinite or NaN: the resident launches and the global-memory
form give the same bits, and a synapse whose delay reaches beyond the last step
takes no part in anything, whatever its weight is."""
import numpy as np
import pytest
import torch

from snc_b200 import bptt as BP

pytestmark = pytest.mark.gpu


def _run(core, resident, w, ext, proj, ckpt):
    core.set_resident(resident)
    wt = torch.as_tensor(w, device="cuda").requires_grad_(True)
    et = ext.cuda().requires_grad_(True)
    s = BP.spiking_core(wt, et, core, 1.0, 0.9, 15.0, ckpt)
    gw, ge = torch.autograd.grad(s, (wt, et), proj.cuda())
    return [x.detach().cpu().numpy() for x in (s, gw, ge)]


def _same(a, b):
    for x, y in zip(a, b):
        np.testing.assert_array_equal(np.isnan(x), np.isnan(y))
        ok = ~np.isnan(x)
        np.testing.assert_array_equal(x[ok].view(np.uint32), y[ok].view(np.uint32))


# one, two and four words a slice; steps below, at and above the largest delay
@pytest.mark.parametrize("n,deg,b", [(60, 8, 20), (2500, 6, 50), (2450, 5, 128)])
@pytest.mark.parametrize("t", [1, 4, 6, 7, 15])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_nonfinite(n, deg, b, t, bad):
    rng = np.random.default_rng(t)
    pre, post = rng.integers(0, n, n * deg), rng.integers(0, n, n * deg)
    d = rng.integers(1, 7, pre.shape[0])
    d[:12] = np.arange(12) % 6 + 1
    w = rng.normal(0, 0.9 / np.sqrt(deg), pre.shape[0]).astype(np.float32)
    gen = torch.Generator().manual_seed(b)
    ext = (torch.rand(t, b, n, generator=gen) < 0.3).float() * 1.1
    proj = torch.randn(t, b, n, generator=gen)
    core = BP.SpikingCore(n, pre, post, d, device="cuda")
    # of every delay that reaches beyond the last step, and of all
    beyond = np.nonzero(d >= t)[0]
    w[beyond] = 0.0
    ref = _run(core, True, w, ext, proj, 3)
    assert all(np.isfinite(x).all() for x in ref)
    w[beyond] = bad
    for resident in (True, False):
        _same(_run(core, resident, w, ext, proj, 3), ref)
    w[:12] = bad
    _same(_run(core, True, w, ext, proj, 0), _run(core, False, w, ext, proj, 0))
