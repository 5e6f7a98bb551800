"""The layout transpose and the leaky scan at the edges of their tiles and
vector widths: equal to torch's permute and to the step-by-step loop bit for
bit, whatever the alignment of the rows."""
import numpy as np
import pytest
import torch

from snc_b200 import bptt as BP

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b", [1, 4, 31, 64, 66, 129])
@pytest.mark.parametrize("n", [1, 3, 60, 64, 65, 192])
def test_transpose(b, n):
    gen = torch.Generator(device="cuda").manual_seed(b * 1000 + n)
    for pad, off in ((0, 0), (4, 0), (3, 0), (5, 1)):
        # rows of n in a wider buffer: a view whose rows start at any alignment
        wide = torch.randn(3, b, n + pad + off, generator=gen, device="cuda")
        x = wide[:, :, off:off + n]
        y = BP._to_tnb(x)
        assert torch.equal(y, x.permute(0, 2, 1).contiguous())
        assert torch.equal(BP._from_tnb(y), x.contiguous())
    # time and batch swapped (a transposed embedding)
    x = torch.randn(b, 5, n, generator=gen, device="cuda").transpose(0, 1)
    assert torch.equal(BP._to_tnb(x), x.permute(0, 2, 1).contiguous())


@pytest.mark.parametrize("t", [1, 7, 8, 9, 17])
@pytest.mark.parametrize("n", [1, 6, 1030, 160000, 160002])
def test_leaky_scan(t, n):
    x = torch.randn(t, n, generator=torch.Generator().manual_seed(t)).cuda().requires_grad_(True)
    y = BP.leaky_scan(x, 0.9)
    g = torch.randn(t, n, generator=torch.Generator().manual_seed(n)).cuda()
    (gx,) = torch.autograd.grad(y, x, g)
    d = np.float32(0.9)
    for out, inp, order in ((y, x, range(t)), (gx, g, range(t - 1, -1, -1))):
        a = np.zeros(n, np.float32)
        o, i = out.detach().cpu().numpy(), inp.detach().cpu().numpy()
        for k in order:
            a = d * a + i[k]
            np.testing.assert_array_equal(o[k].view(np.uint32), a.view(np.uint32))
