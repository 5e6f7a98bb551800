"""The allocation pool at its limits: what it holds, that released blocks serve
again, and that neither its size classes nor its kept blocks make an allocation
fail that fits the device.  In a process of its own, whose memory a ballast
leaves as little of as the case needs."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SETUP = """
import numpy as np, torch
from snc_b200 import eprop as E, runtime as R, workloads as W
MiB = 1 << 20
g = W.random_graph(3, n_in=20, n_hid=300, n_out=5, p=1.0)
dg = R.DeviceGraph(g)
def session(mib):  # the eligibility [batch][S] is the one large block
    return E.CudaTrainSession(g, E.TrainConfig(), batch=-(-mib * MiB // (4 * g.num_synapses)), device_graph=dg)
def free():
    return torch.cuda.mem_get_info()[0]
def leave(mib):
    return torch.empty(free() - mib * MiB, dtype=torch.uint8, device='cuda')
def train(s):
    ev, st = W.random_events(4, g, 2, 6)
    s.run_batch(ev, st, np.zeros(2, np.int32), train=True)
    assert np.count_nonzero(s.eligibility(2))
torch.zeros(1, device='cuda')
s = session(1); train(s); E.destroy(s)  # modules loaded
"""


def _run(code):
    r = subprocess.run([sys.executable, "-c", SETUP + code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


# a class is up to a quarter above: 5140 -> 6144 MiB, 130 -> 160 MiB
@pytest.mark.parametrize("mib,room", [(5140, 400), (130, 24)])
def test_a_block_that_fits_is_not_refused(mib, room):
    _run(f"b = leave({mib} + {room}); s = session({mib}); train(s); E.destroy(s); s = session({mib}); train(s)")


def test_kept_blocks_give_way():
    _run("""
s = session(200); E.destroy(s)          # kept
b = leave(100)
s = session(250); train(s)
""")


def test_kept_bytes_are_bounded_and_serve_again():
    _run("""
a = free()
many = [session(64) for _ in range(8)]  # 8 x 64 MiB
b = free()
assert a - b >= 8 * 64 * MiB
for s in many: E.destroy(s)
c = free()
assert 64 * MiB <= a - c <= (256 + 16) * MiB, (a - c) / MiB
s = session(64)
assert c - free() <= 16 * MiB           # from the kept blocks
train(s); E.destroy(s)
dg.release()
assert a - free() <= 16 * MiB
""")


def test_a_minibatch_that_outgrows_its_scratch():
    """The scratch that a longer minibatch replaces makes room for the new one
    before the call ends."""
    _run("""
s = session(1)
n = 2 * 305 * 4                          # bytes of surrogate history a step
long = 1200 * MiB // n
def run(T):
    ev = W.random_events(4, g, 2, 4)[0]
    s.run_batch(ev, np.full(2, T, np.int32), np.zeros(2, np.int32), train=True)
run(long * 2 // 3)                       # 800 MiB of history
b = leave(600)                           # the 1200 fit only in their place
run(long)
assert np.count_nonzero(s.eligibility(2))
""")
