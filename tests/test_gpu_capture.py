"""Calls beside a stream capture in the global mode, by the same and by another
thread: neither the calls nor the capture may fail, and the results are those of
calls without one."""
import threading

import numpy as np
import pytest

from mplb_b200 import Solver, config

pytestmark = pytest.mark.gpu


def solver():
    s = Solver(config.cavity(3, 48, 0.05, re=100.0))
    s.init_uniform()
    s.stream_collision(2)
    return s


@pytest.mark.parametrize("other_thread", [False, True])
def test_steps_beside_a_capture(gpu_lib, other_thread):
    import torch
    want = solver()
    for _ in range(8):
        want.stream_collision(20)
    got = solver()
    failed = []

    def steps():
        try:
            for _ in range(8):
                got.stream_collision(20)   # the last call's steps still run
        except Exception as e:             # noqa: BLE001
            failed.append(e)

    x = torch.ones(4, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="global"):
        x.add_(1)
        if other_thread:
            t = threading.Thread(target=steps)
            t.start()
            t.join()
        else:
            steps()
        x.add_(1)
    assert not failed, failed
    graph.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [3.0] * 4
    assert np.array_equal(got.f(0), want.f(0))
    assert got.last_step_ms() > 0
    got.close()
    want.close()
