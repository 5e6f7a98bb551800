"""The allocation pool: blocks that one object released serve another without
changing any result, from several threads at once, and all memory is given
back when the last object is released."""
import subprocess
import sys
import threading

import numpy as np
import pytest

from snc_b200 import runtime as R
from snc_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _evaluate(g, dg, seed, lif):
    rng = np.random.default_rng(seed)
    feats = rng.random((3 + seed % 5, g.num_input_channels), dtype=np.float32)
    steps = rng.integers(5, 40, feats.shape[0]).astype(np.int32)
    di = R.DeviceInputs.encode(dg, feats, steps, max_rate=0.4, seed=seed)
    run = R.Run(dg, di, vfinal=True)
    run.launch(lif)
    out = run.fetch(vfinal=True)
    run.release()
    di.release()
    return out


def test_threads_reuse_blocks():
    g = W.random_graph(3)
    lif = R.LIFParams()
    dg = R.DeviceGraph(g)
    ref = [_evaluate(g, dg, s, lif) for s in range(12)]
    bad = []

    def work(k):
        R.set_device(0)
        own = R.DeviceGraph(g)
        for rep in range(4):
            for s in range(k, 12, 2):
                out = _evaluate(g, own, s, lif)
                if any(not np.array_equal(out[n], ref[s][n]) for n in ("logits", "spikes", "events", "v")):
                    bad.append((k, rep, s))

    ts = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad


def test_memory_is_given_back():
    code = """
import numpy as np, torch
from snc_b200 import runtime as R, workloads as W
torch.zeros(1, device='cuda')
def cycle():
    g = W.random_graph(3); dg = R.DeviceGraph(g)
    ev, st = W.random_events(4, g, 400, 200)
    di = R.DeviceInputs(dg, ev, st); r = R.Run(dg, di); r.launch(R.LIFParams()); r.fetch()
    r.release(); di.release(); kept = torch.cuda.mem_get_info()[0]; dg.release(); return kept
cycle()
free = torch.cuda.mem_get_info()[0]
kept = cycle()
assert torch.cuda.mem_get_info()[0] == free and kept < free, (free, kept, torch.cuda.mem_get_info()[0])
"""
    subprocess.run([sys.executable, "-c", code], check=True, timeout=300)
