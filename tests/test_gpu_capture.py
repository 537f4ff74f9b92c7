"""An engine is made while another stream of the process is captured.

A capture in the default (global) mode forbids allocations to every thread of
the process and is invalidated by them, so what an engine allocates for itself
when it is made has to be kept out of the capture's way; the captured graph
replays as if nothing had happened, and the new engine prices.
"""
import threading

import numpy as np
import pytest

from hestonexotics_gb300 import engine as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("other_thread", [False, True])
def test_engine_made_during_a_capture(engine, other_thread):
    torch = pytest.importorskip("torch")
    x = torch.zeros(64, device="cuda")
    torch.cuda.synchronize()
    prm, opts = E.Params(0.04, 0.04, -0.7, 1.5, 0.5, 0.02), E.Options(np.array([100.0]), 1.0, E.ASIAN)
    cfg = E.Config(n_paths=256, steps=8)
    want = engine.price(prm, 100.0, opts, cfg)
    made = []

    def make():
        made.append(E.Engine(0))

    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(torch.cuda.Stream()):
        graph.capture_begin()
        x.add_(1.0)
        if other_thread:
            t = threading.Thread(target=make)
            t.start()
            t.join()
        else:
            make()
        graph.capture_end()   # raises if the capture was invalidated
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [2.0] * 64
    (other,) = made
    got = other.price(prm, 100.0, opts, cfg)
    other.close()
    np.testing.assert_array_equal(got, want)
