"""Gathers of distances (SSSP) and of visited bits (BFS) through L1: graphs around the sizes at which all rows, or only the first ones, are read
there, with hubs that many edges improve at once.  Distances equal the oracle bit for bit, also when one handle answers
queries from different sources one after the other (an old distance must never outlive its query) and when one launch
answers them in turn."""
import numpy as np
import pytest

import oracle as O
import pytrav as T

pytestmark = pytest.mark.gpu


def _skewed(V, E, seed):
    rng = np.random.default_rng(seed)
    s = (V * rng.random(E) ** 3).astype(np.int32)
    d = (V * rng.random(E) ** 3).astype(np.int32)
    perm = rng.permutation(V).astype(np.int32)
    return perm[s], perm[d], rng.random(E, dtype=np.float32)


@pytest.mark.parametrize("V,E", [(8191, 120_000), (8192, 120_000), (8193, 120_000), (70_001, 1_000_000),
                                 (1 << 19, 4_500_000), ((1 << 19) + 1, 4_500_000), (700_000, 1_500_000)])
def test_distances_around_the_limits(V, E):
    import torch

    s, d, w = _skewed(V, E, V)
    g = T.Graph.from_edges(V, s, d, w)
    csr = O.csr(V, s, d, w)
    deg = np.bincount(s, minlength=V)
    srcs = [int(deg.argmax()), int(np.flatnonzero(deg)[-1])]
    want = [O.dijkstra(V, s, d, w, x, csr_arrays=csr).view(np.uint32) for x in srcs]
    for delta in (0.0, 0.05, 0.4):
        for _ in range(2):
            for x, ref in zip(srcs, want):
                assert np.array_equal(g.sssp([x], delta=delta)[0].view(np.uint32), ref), (delta, x)
        both = g.sssp(srcs, delta=delta).view(np.uint32)
        assert np.array_equal(both[0], want[0]) and np.array_equal(both[1], want[1])
    levels = [O.bfs_levels(V, s, d, x, csr_arrays=csr) for x in srcs]
    for force in (0, -1, 0):
        for x, ref in zip(srcs, levels):
            assert np.array_equal(g.bfs([x], force_direction=force)[0], ref), (force, x)
    g.set_grid(1, 5)
    assert np.array_equal(g.sssp([srcs[0]], delta=0.05)[0].view(np.uint32), want[0])
    g.set_grid(1, 0)
    outs = [torch.empty(V, dtype=torch.float32, device="cuda") for _ in range(4)]
    b = T.Batch([g])
    b.shape = (74, 64, 256)
    b.run([(0, 1, srcs[k % 2], 0.05, T.SCHEDULE_PLAIN, outs[k]) for k in range(4)])
    for k in range(4):
        assert np.array_equal(outs[k].cpu().numpy().view(np.uint32), want[k % 2])
    b.close()
    g.free()


@pytest.mark.parametrize("V,E", [(1 << 13, 1 << 18), ((1 << 19) + 3, 9_000_000)])
def test_pull_rounds_gather_sources_through_l1(V, E):
    """All rows near, and only the first 8,192: the source's distance of a pulled edge may be old, and the result must
    not be."""
    s, d, w = _skewed(V, E, V + 1)
    g = T.Graph.from_edges(V, s, d, w)
    csr = O.csr(V, s, d, w)
    deg = np.bincount(s, minlength=V)
    order = np.argsort(-deg, kind="stable")
    pulled = 0
    for x in (int(order[0]), int(order[5]), int(np.flatnonzero(deg)[-1])):
        ref = O.dijkstra(V, s, d, w, x, csr_arrays=csr).view(np.uint32)
        for delta in (0.02, 0.1):
            assert np.array_equal(g.sssp([x], delta=delta)[0].view(np.uint32), ref), (x, delta)
            pulled += int(np.sum(g.last_phase_log()[0] == 7))
    assert pulled > 0
    g.free()
