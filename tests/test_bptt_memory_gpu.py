"""Scratch memory of the resident backward: rows of the batch's own size, not of
whole 32-sample words."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import numpy as np, torch
from snc_b200 import bptt as BP
n, t, b = 4000, 400, {b}
rng = np.random.default_rng(1)
pre, post = rng.integers(0, n, 3 * n), rng.integers(0, n, 3 * n)
core = BP.SpikingCore(n, pre, post, rng.integers(1, {delay} + 1, 3 * n), device='cuda')
w = torch.full((3 * n,), 0.3, device='cuda').requires_grad_(True)
def step(t, ckpt):
    ext = torch.full((t, b, n), 0.4, device='cuda')
    s = BP.spiking_core(w, ext, core, 1.0, 0.9, 15.0, ckpt)
    torch.autograd.grad(s.sum(), w)
torch.empty(300 << 20, dtype=torch.uint8, device='cuda')  # torch's own
step(2, 1)
free = torch.cuda.mem_get_info()[0]
step(t, t)
used = free - torch.cuda.mem_get_info()[0]
# the segment [t][n][b], with a tenth of slack, the ring and torch's tensors
assert used <= 4 * n * b * (t * 6.6 + {delay} + 1) + (64 << 20), used
"""


@pytest.mark.parametrize("b,delay", [(1, 5), (1, 200), (3, 5)])
def test_rows(b, delay):
    r = subprocess.run([sys.executable, "-c", CODE.format(b=b, delay=delay)], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
