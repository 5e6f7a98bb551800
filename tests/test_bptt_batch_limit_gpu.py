"""At most 256 samples a call, whatever form the net's launches take."""
import numpy as np
import pytest
import torch

from snc_b200 import _lib
from snc_b200 import bptt as BP

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,resident,smooth", [(40, True, False), (40, False, False), (40, True, True),
                                               (5000, True, False)])
def test_limit(n, resident, smooth):
    rng = np.random.default_rng(n)
    pre, post = rng.integers(0, n, 4 * n), rng.integers(0, n, 4 * n)
    core = BP.SpikingCore(n, pre, post, rng.integers(1, 4, 4 * n), device="cuda")
    core.set_resident(resident)
    w = torch.as_tensor(rng.normal(0, 0.5, 4 * n).astype(np.float32), device="cuda")
    for b in (256, 257, 300):
        ext = (torch.rand(3, b, n, device="cuda") < 0.3).float() * 1.1
        if b <= 256:
            assert BP.spiking_core(w, ext, core, 1.0, 0.9, 15.0, 2, smooth).shape == ext.shape
            continue
        with pytest.raises(_lib.SncB200Error) as e:
            BP.spiking_core(w, ext, core, 1.0, 0.9, 15.0, 2, smooth)
        assert e.value.status == _lib.EUNSUPPORTED
