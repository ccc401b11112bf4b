"""The library's kept device memory, through the public entry points: what other threads, batches, the caller and a
new context see of it.  (test_device_memory.py tests the same code on a runtime of the host.)"""
import subprocess
import sys
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


def test_a_batch_runs_in_the_memory_that_the_library_keeps():
    """Little is free beside kept blocks: the teams' scratch is sized as if they were free, as they were before
    blocks were kept."""
    import torch

    V = 1 << 10
    s, d, w = O.rmat(10, 8, seed=3)
    src, dst, _ = O.rmat(19, 16, seed=4)
    b = T.Batch([g := T.Graph.from_edges(V, s, d, w)])
    levels = torch.empty((8, V), dtype=torch.int32, device="cuda")
    queries = [(0, 0, x, 0.0, T.SCHEDULE_PLAIN, levels[x]) for x in range(8)]
    T.Graph.from_edges(1 << 19, src, dst, None).free()  # leaves some 600 MB of kept blocks
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    # less than the 1 GB that a batch leaves to the caller, more with the kept blocks
    filler = torch.empty(free - (900 << 20), dtype=torch.uint8, device="cuda")
    try:
        assert torch.cuda.mem_get_info()[0] < 1 << 30
        b.run(queries)
    finally:
        del filler
        torch.cuda.empty_cache()
    assert np.array_equal(levels.cpu().numpy(), np.stack([O.bfs_levels(V, s, d, x) for x in range(8)]))
    b.close()
    g.free()


def test_kept_memory_is_bounded_and_given_back_on_request():
    import torch

    V = 1 << 18
    s, d, w = O.rmat(18, 16, seed=9)
    hub = int(np.bincount(s, minlength=V).argmax())
    want = O.bfs_levels(V, s, d, hub)
    g = T.Graph.from_edges(V, s, d, w)
    g.bfs([hub])  # what a first call loads is there
    g.free()
    T.trim_memory()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    for _ in range(12):
        graphs = [T.Graph.from_edges(V, s, d, w) for _ in range(4)]
        assert np.array_equal(graphs[-1].bfs([hub])[0], want)  # in blocks of earlier handles
        for g in graphs:
            g.free()
    kept = free - torch.cuda.mem_get_info()[0]
    assert 0 < kept <= (1 << 30) + (64 << 20)  # the driver hands out pages of 2 MB
    assert T.trim_memory() > 0
    assert free - torch.cuda.mem_get_info()[0] <= 64 << 20
    assert T.trim_memory() == 0


def test_a_new_context_after_a_device_reset_starts_afresh():
    """A program that frees its handles and resets the device builds and runs on; nothing that was kept of the old
    context (blocks, streams, kernel attributes) is used in the new one."""
    code = """
import ctypes, sys
import numpy as np
sys.path[:0] = %r
import oracle as O, pytrav as T
rt = ctypes.CDLL("libcudart.so.12")
V = 1 << 14
s, d, w = O.rmat(14, 4, seed=2)
for k in range(3):
    g = T.Graph.from_edges(V, s, d, w)
    assert np.array_equal(g.bfs([1])[0], O.bfs_levels(V, s, d, 1)), k
    want = O.dijkstra(V, s, d, w, 1)
    for delta in (0.0, 0.1):
        assert np.array_equal(g.sssp([1], delta=delta)[0].view(np.uint32), want.view(np.uint32)), (k, delta)
    g.free()
    assert rt.cudaDeviceReset() == 0
print("fine")
""" % (sys.path,)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "fine", r.stdout + r.stderr
