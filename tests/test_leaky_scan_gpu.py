"""The leaky scan over few and many columns, forwards and backwards, at step counts
around those it requests at once: equal to the step loop bit for bit."""
import numpy as np
import pytest
import torch

from snc_b200 import bptt as BP

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1), (3, 5), (2, 7001), (8, 148 * 1024 // 8)])
@pytest.mark.parametrize("t", [1, 7, 8, 9, 15, 16, 17, 31, 32, 33, 48, 61])
def test_steps(t, shape):
    gen = torch.Generator().manual_seed(t)
    x = torch.randn(t, *shape, generator=gen)
    g = torch.randn(t, *shape, generator=gen)
    xc = x.cuda().requires_grad_(True)
    y = BP.leaky_scan(xc, 0.9)
    (dx,) = torch.autograd.grad(y, xc, g.cuda())
    decay = np.float32(0.9)
    for got, src in ((y.detach(), x), (dx.flip(0), g.flip(0))):
        src, acc = src.numpy(), np.zeros(shape, np.float32)
        got = got.cpu().numpy()
        for k in range(t):
            acc = decay * acc + src[k]
            np.testing.assert_array_equal(got[k].view(np.uint32), acc.view(np.uint32))
