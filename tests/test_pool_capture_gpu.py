"""Releasing an object waits for the device's work on every stream, and leaves a
stream capture alone that another thread, or the same one in relaxed mode, has
under way."""
import threading

import pytest
import torch

from snc_b200 import runtime as R
from snc_b200 import workloads as W

pytestmark = pytest.mark.gpu

LIF = R.LIFParams()


def _objects(dg, g):
    ev, st = W.random_events(4, g, 20, 50)
    di = R.DeviceInputs(dg, ev, st)
    run = R.Run(dg, di)
    run.launch(LIF)
    run.fetch()
    return run, di


@pytest.mark.parametrize("mode", ["thread_local", "relaxed"])
def test_release_during_a_capture(mode):
    g = W.random_graph(3)
    dg = R.DeviceGraph(g)
    x = torch.ones(4, device="cuda")
    objects = _objects(dg, g)
    begun, released = threading.Event(), threading.Event()

    def release():
        if mode == "thread_local":
            begun.wait(20)
            R.set_device(0)
        for o in objects:
            o.release()
        released.set()

    other = threading.Thread(target=release)
    if mode == "thread_local":
        other.start()
    cg = torch.cuda.CUDAGraph()
    with torch.cuda.graph(cg, capture_error_mode=mode):
        x.mul_(2)
        if mode == "thread_local":
            begun.set()
            released.wait(20)
        else:
            release()
        x.add_(1)
    if mode == "thread_local":
        other.join()
    assert released.is_set()
    cg.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [3.0] * 4
    for o in _objects(dg, g):  # the released blocks serve again
        o.release()


def test_release_waits_for_every_stream():
    g = W.random_graph(3)
    dg = R.DeviceGraph(g)
    _objects(dg, g)
    s = torch.cuda.Stream()  # not ordered with the legacy stream
    for k in range(3):
        run, di = _objects(dg, g)
        with torch.cuda.stream(s):
            torch.cuda._sleep(20_000_000)  # about 10 ms
        (run if k else di).release()
        assert s.query()
