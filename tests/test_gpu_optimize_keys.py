"""The optimisation pass where its packed sort keys change width: vertex and segment counts around powers of two, one
vertex, one segment and as many segments as vertices.  The arrays equal the oracle's exactly."""
import numpy as np
import pytest

import oracle as O
import pytrav as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [1, 2, 3, 255, 256, 257, 65_535, 65_536, 65_537])
def test_packed_keys(V):
    import torch

    rng = np.random.default_rng(V)
    E = 30_000
    s, d = rng.integers(0, V, E).astype(np.int32), rng.integers(0, V, E).astype(np.int32)
    s[:50], d[50:100] = V - 1, V - 1
    w = (rng.integers(0, 5, E) / 4).astype(np.float32)
    for segment in (0, 1, 2, max(V // 256, 1), max(V - 1, 1), V, V + 1, 2**31 - 1):
        want = O.el_optimize(s, d, w, segment=segment)
        t = [torch.from_numpy(x.copy()).cuda() for x in (s, d, w)]
        n = T.el_optimize(*t, V, segment)
        assert n == len(want[0])
        for a, b in zip(t, want):
            assert np.array_equal(a[:n].cpu().numpy().view(np.uint32), b.view(np.uint32)), segment
