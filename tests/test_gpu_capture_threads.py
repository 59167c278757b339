"""A call on one thread while another thread captures a graph on its own stream:
the capture goes on in every capture mode (the call's scratch may have to grow),
and both give their results."""
import ctypes
import threading

import numpy as np
import pytest
import torch

import arbor_b200 as ab
from gpu_util import dev, host, ok, render_buffers
from test_gpu_tight import Scene, batched, state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["global", "thread_local", "relaxed"])
def test_call_beside_another_threads_capture(cuda, mode):
    w, h, n = 320, 180, {"global": 7, "thread_local": 9, "relaxed": 11}[mode]  # (more scenes each time: the scratch grows)
    one, many, C = Scene([7]), Scene([20 + 13 * k for k in range(n)]), dev(state(w, h))
    want, r, got = batched(one, C, w, h), render_buffers(w, h), []
    of = (ctypes.c_int * 324)(*[t % n for t in range(324)])
    stream, ready, go, done = torch.cuda.Stream(), threading.Event(), threading.Event(), threading.Event()
    torch.cuda.synchronize()

    def other():
        ready.set()
        go.wait(60)
        for _ in range(3):
            got.append(ab.call("arbor_traceSpeciesPixels", many.P, many.Nodes, many.Order, n, of, C, r["Linear"], w, h, stream=stream))
            got.append(ab.call("arbor_tracePixels", one.P, one.Nodes, one.Order, C, r["Hit"], w, h, stream=stream))
        done.set()

    thread = threading.Thread(target=other)
    thread.start()
    ready.wait(60)
    x, graph, side = torch.zeros(64, device="cuda"), torch.cuda.CUDAGraph(), torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    try:
        with torch.cuda.graph(graph, stream=side, capture_error_mode=mode):
            x.add_(1.0)
            go.set()
            done.wait(60)
            x.mul_(2.0)
    finally:
        go.set()
        thread.join()
    graph.replay()
    torch.cuda.synchronize()
    assert got == [ab.OK] * 6 and bool((x == 2.0).all())
    assert np.array_equal(host(r["Hit"]).view(np.uint32), host(want["Hit"]).view(np.uint32))
