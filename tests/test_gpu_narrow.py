"""Queries that run (or begin) in the narrow kernel, at the sizes where it changes path: rows around a segment and
around a whole queue, frontiers that outgrow the queue at once, after some phases or never, graphs around the sizes
that are initialised there and that run there alone.  Levels and distances equal the oracle bit for bit, and the
logs describe the same traversal."""
import numpy as np
import pytest

import oracle as O
import pytrav as T

pytestmark = pytest.mark.gpu


def _check(V, s, d, w, src, deltas=(0.0, 0.3, 40.0)):
    s, d, w = np.asarray(s, np.int32), np.asarray(d, np.int32), np.asarray(w, np.float32)
    g = T.Graph.from_edges(V, s, d, w)
    csr = O.csr(V, s, d, w)
    want = O.bfs_levels(V, s, d, src, csr_arrays=csr)
    for force in (-1, 0, 1):
        assert np.array_equal(g.bfs([src], force_direction=force)[0], want), force
        st = g.last_stats()
        dirs, frontier = g.last_bfs_trace()
        kind = g.last_phase_log()[0]
        assert st.steps == want.max() + 1
        n = len(dirs)  # the logs hold at most 4096 entries
        assert frontier.tolist() == [int((want == i).sum()) for i in range(n)]
        if len(kind) < 4096:
            assert [k for k in kind if k in (0, 1)] == dirs.tolist()
    ref = O.dijkstra(V, s, d, w, src, csr_arrays=csr).view(np.uint32)
    for delta in deltas:
        for _ in range(2):
            assert np.array_equal(g.sssp([src], delta=delta)[0].view(np.uint32), ref), delta
    g.free()


def _grid(h, wd, seed):
    idx = np.arange(h * wd).reshape(h, wd)
    p = [(idx[:, :-1], idx[:, 1:]), (idx[:, 1:], idx[:, :-1]), (idx[:-1], idx[1:]), (idx[1:], idx[:-1])]
    s, d = (np.concatenate([x[k].ravel() for x in p]) for k in (0, 1))
    return h * wd, s, d, np.random.default_rng(seed).integers(1, 100, len(s)).astype(np.float32)


@pytest.mark.parametrize("h,wd", [(1, 3), (64, 80), (64, 81), (64, 96), (64, 97), (5, 3000), (362, 362), (400, 331)])
def test_grids_stay_narrow(h, wd):
    _check(*_grid(h, wd, h), src=h * wd // 2)


@pytest.mark.parametrize("deg", [0, 1, 127, 128, 129, 640, 5119, 5120, 5121, 6143, 6144, 6145, 20_000])
def test_rows_at_the_segment_and_queue_limits(deg):
    """A hub behind a path, with `deg` out-edges to leaves that join again and go on."""
    V = deg + 8
    s = [0, 1] + [2] * deg + [3 + i for i in range(deg)] + [V - 3, V - 2]
    d = [1, 2] + [3 + i for i in range(deg)] + [V - 3] * deg + [V - 2, V - 1]
    rng = np.random.default_rng(deg)
    _check(V, s, d, (rng.integers(0, 9, len(s)) / 8).astype(np.float32), 0)


@pytest.mark.parametrize("V,E,seed", [(5120, 30_000, 8), (5121, 30_000, 9), (6144, 30_000, 1), (6145, 30_000, 2), (6144, 300_000, 3), (131_072, 400_000, 4),
                                      (131_073, 400_000, 5), (3000, 262_144, 6), (40_000, 60_000, 7)])
def test_random_graphs_change_over(V, E, seed):
    rng = np.random.default_rng(seed)
    s, d = rng.integers(0, V, E), rng.integers(0, V, E)
    s[0] = 7
    _check(V, s, d, rng.random(E, dtype=np.float32), 7, deltas=(0.0, 0.05, 0.5))


def test_learned_widths_and_several_sources():
    V, s, d, w = _grid(150, 170, 3)
    s, d = s.astype(np.int32), d.astype(np.int32)
    g = T.Graph.from_edges(V, s, d, w)
    g.set_mlp(1, np.random.default_rng(1).normal(scale=2.0, size=T.mlp_param_count(1)))
    srcs = [0, 77, V - 1]
    got = g.sssp(srcs, delta=3.0, schedule=T.SCHEDULE_LEARNED)
    x, ch, ph, lo, hi = g.last_decisions()
    assert len(ch) > 0 and np.all(hi > lo) and np.all(np.diff(lo) > 0) and np.all(np.isfinite(x))
    for k, src in enumerate(srcs):
        assert np.array_equal(got[k].view(np.uint32), O.dijkstra(V, s, d, w, src).view(np.uint32))
    g.free()


def test_masked_sweep_through_the_narrow_kernel():
    """The vertex mask reaches the BFS kernels when the edge-list sweeps give up (a long path)."""
    import torch

    n = 20_000
    s = np.arange(n - 1).astype(np.int32)[::-1].copy()
    d = (s + 1).astype(np.int32)
    trees = (np.arange(n) >= 15_000).astype(np.int32)
    vis = torch.full((n,), 9, dtype=torch.uint8, device="cuda")
    tp = torch.tensor([3], dtype=torch.int32, device="cuda")
    ts, td, tt = (torch.from_numpy(x).cuda() for x in (s, d, trees))
    T._check(T.lib().trav_reach_el_masked(ts.data_ptr(), td.data_ptr(), n, n - 1, tp.data_ptr(), tt.data_ptr(),
                                          vis.data_ptr()))
    assert np.array_equal(vis.cpu().numpy(), O.reach_masked(n, s, d, 3, trees))


@pytest.mark.parametrize("first,fan", [(127, 1980), (100, 2500), (60, 4000), (20, 6000), (3, 40_000)])
def test_long_rows_beyond_the_segments_of_a_queue(first, fan):
    # a small graph whose source has one short row, so that one block of the cluster finds all the long rows of the
    # next frontier: their segments outnumber the places of its queue
    V = 1200
    rng = np.random.default_rng(first)
    s = np.concatenate([np.zeros(first, np.int64), np.repeat(np.arange(1, first + 1), fan)])
    d = np.concatenate([np.arange(1, first + 1), rng.integers(0, V, first * fan)])
    assert len(s) <= 1 << 18
    _check(V, s, d, rng.uniform(0.01, 1.0, len(s)), 0, deltas=(0.0, 0.3))


@pytest.mark.parametrize("width", [1, 15, 16, 17, 500, 2500, 9000])
def test_frontiers_of_one_width(width):
    """Ladders: `width` paths side by side with a common root, so that every phase has as many rows; with cross edges
    that make the rows of one path longer than the others' (rows stay with their block, or are dealt round)."""
    n = 12
    idx = 1 + np.arange(n * width).reshape(n, width)
    s = [np.zeros(width), idx[:-1].ravel(), np.repeat(idx[:-1, 0], min(width, 400))]
    d = [idx[0], idx[1:].ravel(), np.concatenate([row[: min(width, 400)] for row in idx[1:]])]
    s, d = np.concatenate(s).astype(np.int64), np.concatenate(d)
    rng = np.random.default_rng(width)
    _check(1 + n * width, s, d, (rng.integers(1, 20, len(s)) / 4).astype(np.float32), 0, deltas=(0.0, 1.0, 3.0))


@pytest.mark.parametrize("where", ["apart", "first", "last"])
@pytest.mark.parametrize("deg", [511, 512, 513, 640, 641, 4000])
def test_long_in_rows_in_bottom_up_steps(deg, where):
    """An in-row around the length from which a whole warp scans it: without a parent that is ever reached, with one
    at its start, or at its end; beside rows of every lane's own."""
    rng = np.random.default_rng(deg)
    n = 400  # a dense part that is searched bottom-up, a hub, and `deg` sources of it
    hub = n
    s = np.concatenate([rng.integers(0, n, 20 * n), hub + 1 + np.arange(deg)])
    d = np.concatenate([rng.integers(0, n, 20 * n), np.full(deg, hub)])
    # in-rows are in the order of falling out-degree, then of ids
    if where == "first":
        s, d = np.concatenate([s, np.full(301, n - 1)]), np.concatenate([d, [hub], rng.integers(0, n, 300)])
    elif where == "last":
        s, d = np.concatenate([s, [3]]), np.concatenate([d, [hub + deg]])
    _check(n + 1 + deg, s, d, rng.random(len(s), dtype=np.float32), 0, deltas=(0.0,))


@pytest.mark.parametrize("n", [3, 4, 5, 8, 9, 127, 129, 1023, 2047, 2048, 2049, 4097, 5000])
def test_one_long_heavy_row_among_short_ones(n):
    """A star whose leaves point back: the hub's heavy row, of about 2 n / 3 edges, is expanded beside as many rows of
    one edge as there are leaves in the bucket, and gets up to a whole block's lanes."""
    leaf = 1 + np.arange(n)
    s = np.concatenate([np.zeros(n), leaf, leaf])
    d = np.concatenate([leaf, np.zeros(n), 1 + (leaf % n)])
    rng = np.random.default_rng(n)
    _check(n + 1, s, d, (rng.integers(0, 9, len(s)) / 8).astype(np.float32), 0, deltas=(0.0, 0.3))


@pytest.mark.parametrize("V,E,hub", [(5120, 32_768, 0), (5120, 32_769, 0), (5120, 65_536, 0), (5120, 65_537, 0),
                                     (3000, 65_536, 512), (3000, 65_536, 513), (3000, 262_144, 5120),
                                     (3000, 262_144, 5121), (3000, 262_145, 0), (20_000, 60_000, 5120),
                                     (20_000, 60_000, 5121)])
def test_queries_at_the_limits_of_where_they_run(V, E, hub):
    """Edge counts and longest rows around those that decide whether a query runs in the narrow kernel alone, begins
    there, or runs in the wide kernel; from the vertex of the longest row and from another, with forced directions."""
    rng = np.random.default_rng(E + hub)
    n = E - hub
    s, d = np.concatenate([np.arange(n) % (V - 1) + 1, np.zeros(hub)]), rng.integers(0, V, E)
    w = rng.random(E, dtype=np.float32)  # mean weight 0.5
    for src in (0, 7):
        _check(V, s, d, w, src, deltas=(0.0, 0.1, 0.6))


@pytest.mark.parametrize("hubs", [1, 8, 9, 10, 12])
def test_far_vertices_of_one_block_are_written_out_in_time(hubs):
    """A chain of hubs, each with a heavy row of 4,900 far leaves that two or three blocks expand, one bucket a hub.
    From the tenth on, the pile in memory, shared out over 16 blocks, and the 2,048 vertices that a block has staged
    could overflow its queue in the next bucket opening, and are written out first.  That is no phase of the query:
    the log is the one of the wide kernel."""
    leaves = 4900
    V = hubs * (1 + leaves)
    hub = np.arange(hubs)
    s = np.concatenate([np.repeat(hub, leaves), hub[:-1]]).astype(np.int32)
    d = np.concatenate([np.arange(hubs, V), hub[1:]]).astype(np.int32)
    w = np.concatenate([np.full(hubs * leaves, 30.0), np.full(hubs - 1, 1.5)]).astype(np.float32)
    want = []
    for i in range(hubs):
        want += [(5, 1), (4, (i + 1) * leaves + (i + 1 < hubs))]
    want += [(4, i * leaves) for i in range(hubs - 1, 0, -1)]
    g = T.Graph.from_edges(V, s, d, w)
    ref = O.dijkstra(V, s, d, w, 0).view(np.uint32)
    for ctas in (0, 5):  # 0: begins in the narrow kernel; the caller's shape: wide only
        g.set_grid(1, ctas)
        assert np.array_equal(g.sssp([0], delta=1.0)[0].view(np.uint32), ref)
        kind, size, end_us, _ = g.last_phase_log()
        # (the wide kernel may check for pulling, and pull, in a heavy round)
        got = [(5 if k == 7 else int(k), int(x)) for k, x in zip(kind, size) if k != 6]
        assert got == want, ctas
        assert np.all(np.diff(end_us) >= 0)
    g.free()
