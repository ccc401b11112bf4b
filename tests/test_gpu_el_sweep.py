"""The edge-list sweeps behind bfs_wrapper, bellman_ford_wrapper and the masked reachability sweep, at the sizes
where they change path: edge counts around one 16-byte load and one CTA, arrays off a 16-byte boundary, bitmaps
too large for shared memory, and paths too long for sweeps (the CSR kernels take over).  Everything equals the
oracle bit for bit."""
import numpy as np
import pytest

import oracle as O
import pytrav as T

pytestmark = pytest.mark.gpu
FLT_MAX = np.finfo(np.float32).max


def _dev(torch, x, shift):
    """x on the GPU, starting `shift` elements past an allocation's start."""
    t = torch.zeros(len(x) + 4, dtype=torch.from_numpy(x[:0]).dtype, device="cuda")
    t[shift:shift + len(x)] = torch.from_numpy(x).cuda()
    return t[shift:shift + len(x)]


def _run(torch, V, s, d, w, src, trees=None, shift=0):
    ts, td, tw = _dev(torch, s, shift), _dev(torch, d, shift), _dev(torch, w, shift)
    vis = torch.full((V + 1,), 9, dtype=torch.uint8, device="cuda")
    dist = torch.empty(V, dtype=torch.float32, device="cuda")
    T.bfs_wrapper(ts, td, V, len(s), vis, src)
    T.init_distances(dist, V, src)
    T.bellman_ford_wrapper(ts, td, tw, V, len(s), src, dist)
    assert vis[V].item() == 9
    assert np.array_equal(vis[:V].cpu().numpy(), (O.bfs_levels(V, s, d, src) >= 0).astype(np.uint8))
    want = O.dijkstra(V, s, d, w, src)
    assert np.array_equal(dist.cpu().numpy().view(np.uint32), want.view(np.uint32))
    if trees is not None:
        tp = torch.tensor([src], dtype=torch.int32, device="cuda")
        tt = torch.from_numpy(trees).cuda()
        T._check(T.lib().trav_reach_el_masked(ts.data_ptr(), td.data_ptr(), V, len(s), tp.data_ptr(), tt.data_ptr(),
                                              vis.data_ptr()))
        assert np.array_equal(vis[:V].cpu().numpy(), O.reach_masked(V, s, d, src, trees))


@pytest.mark.parametrize("E,shift", [(0, 0), (1, 0), (3, 0), (4, 0), (5, 1), (8191, 0), (8192, 0), (8193, 3),
                                     (100_003, 0), (100_003, 2), (3_000_001, 0)])
def test_edge_counts_and_alignments(E, shift):
    import torch

    rng = np.random.default_rng(E + shift)
    V = max(2, E // 5 + 1)
    s, d = (rng.integers(0, V, E).astype(np.int32) for _ in range(2))
    w = rng.random(E, dtype=np.float32)
    _run(torch, V, s, d, w, int(s[0]) if E else 1, rng.integers(0, 2, V).astype(np.int32), shift)


@pytest.mark.parametrize("V", [31, 32, 33, 819_200, 819_201, 1_638_400, 1_638_401, 2_500_000])
def test_bitmaps_at_the_shared_memory_limits(V):
    import torch

    rng = np.random.default_rng(V)
    E = min(8 * V, 4_000_000)
    s, d = (rng.integers(0, V, E).astype(np.int32) for _ in range(2))
    w = (rng.integers(0, 5, E) / 4).astype(np.float32)  # zero weights and ties
    _run(torch, V, s, d, w, V - 1, rng.integers(0, 2, V).astype(np.int32))


@pytest.mark.parametrize("n", [40, 70, 20_000])
def test_long_paths_go_on_in_the_csr_kernels(n):
    import torch

    s = np.arange(n - 1, 0, -1).astype(np.int32)  # n-1 -> n-2 -> ... -> 0, listed backwards
    s, d = s[::-1].copy(), (s[::-1] - 1).astype(np.int32)
    w = np.full(n - 1, 0.5, np.float32)
    _run(torch, n, s, d, w, n - 1, np.zeros(n, np.int32))


def test_any_start_distances():
    """Seeds, infinities, NaN and negative values in d keep the meaning they had: only finite values >= 0 spread,
    and only a smaller sum replaces a value."""
    import torch

    V, s, d = 6, np.array([0, 1, 2, 3, 4], np.int32), np.array([1, 2, 3, 4, 5], np.int32)
    w = np.array([1.0, 1.0, 1.0, 1.0, 1.0], np.float32)
    start = np.array([3.0, FLT_MAX, np.inf, -1.0, 2.0, np.nan], np.float32)
    dist = torch.from_numpy(start.copy()).cuda()
    T.bellman_ford_wrapper(*(torch.from_numpy(x).cuda() for x in (s, d, w)), V, 5, 0, dist)
    want = np.array([3.0, 4.0, 5.0, -1.0, 2.0, np.nan], np.float32)
    assert np.array_equal(dist.cpu().numpy().view(np.uint32), want.view(np.uint32))


def test_bad_edges_are_refused_and_nothing_is_written():
    import torch

    V, s, d = 100, np.arange(99).astype(np.int32), np.arange(1, 100).astype(np.int32)
    for bad, msg in ((100, "outside"), (-1, "outside"), (np.float32(-1), "negative"), (np.float32(np.inf), "infinite"),
                     (np.float32(np.nan), "NaN")):
        w, d2 = np.ones(99, np.float32), d.copy()
        if isinstance(bad, int):
            d2[98] = bad
        else:
            w[98] = bad
        dist = torch.full((V,), 5.0, device="cuda")
        with pytest.raises(T.TravError) as e:
            T.bellman_ford_wrapper(*(torch.from_numpy(x).cuda() for x in (s, d2, w)), V, 99, 0, dist)
        assert e.value.code == T.TRAV_ERR_BAD_ARG and msg in str(e.value)
        assert bool((dist == 5.0).all())


def test_the_largest_vertex_count():
    """V = 2^31 - 1: vertex loops count past 2^31."""
    import torch

    V = (1 << 31) - 1
    path = [0, V - 1, V - 2, 5, 1 << 30]
    s, d = (torch.tensor(x, dtype=torch.int32, device="cuda") for x in (path[:-1], path[1:]))
    w = torch.full((4,), 0.5, device="cuda")
    vis = torch.full((V + 1,), 9, dtype=torch.uint8, device="cuda")
    T.bfs_wrapper(s, d, V, 4, vis, 0)
    assert vis[V].item() == 9 and vis[path].tolist() == [1] * 5 and int(vis[:V].sum(dtype=torch.int64)) == 5
    trees = torch.zeros(V, dtype=torch.int32, device="cuda")
    trees[5] = 1  # outside the pivot's tree, and on the way to the last vertex
    pivot = torch.zeros(1, dtype=torch.int32, device="cuda")
    T._check(T.lib().trav_reach_el_masked(s.data_ptr(), d.data_ptr(), V, 4, pivot.data_ptr(), trees.data_ptr(),
                                          vis.data_ptr()))
    assert vis[V].item() == 9 and vis[path].tolist() == [1, 1, 1, 0, 0] and int(vis[:V].sum(dtype=torch.int64)) == 3
    del vis, trees
    dist = torch.full((V + 1,), -7.0, device="cuda")
    T.init_distances(dist, V, 0)
    assert dist[V].item() == -7.0 and dist[0].item() == 0.0 and bool((dist[1:V] == float(FLT_MAX)).all())
    T.bellman_ford_wrapper(s, d, w, V, 4, 0, dist)
    assert dist[V].item() == -7.0 and dist[path].tolist() == [0.0, 0.5, 1.0, 1.5, 2.0]
    assert int((dist[:V] < float(FLT_MAX)).sum()) == 5
