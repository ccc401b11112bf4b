"""The library's kept device memory, through the public entry points: what other threads, batches, the caller and a
new context see of it.  (test_device_memory.py tests the same code on a runtime of the host.)"""
import threading

import numpy as np
import pytest

import oracle as O
import pytrav as T

pytestmark = pytest.mark.gpu


def test_graphs_built_and_freed_in_one_thread_do_not_disturb_a_capture_in_another():
    """One handle per host thread: the first records a CUDA graph at every call (its arguments change), the second
    allocates and frees all the time."""
    import torch

    V = 1 << 10
    s, d, w = O.rmat(10, 8, seed=3)
    want = [O.bfs_levels(V, s, d, x) for x in range(4)]
    out = torch.empty((4, V), dtype=torch.int32, device="cuda")
    g = T.Graph.from_edges(V, s, d, w)
    g.bfs([0], out=out[:1])  # kernels loaded, workspace there
    g.set_capture(True)
    stop, errors = threading.Event(), []

    def build_and_free():
        try:
            torch.cuda.set_device(0)
            while not stop.is_set():
                T.Graph.from_edges(V, s, d, w).free()
        except Exception as e:  # noqa: BLE001 (reported by the test)
            errors.append(e)

    other = threading.Thread(target=build_and_free)
    other.start()
    try:
        for k in range(2000):
            x = k % 4
            g.bfs([x], out=out[x : x + 1], alpha=15.0 + k)  # a new key: captured again
    finally:
        stop.set()
        other.join()
    assert not errors, errors
    assert np.array_equal(out.cpu().numpy(), np.stack(want))
    g.free()
