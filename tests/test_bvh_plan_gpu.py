"""The planned collapse into 8-wide nodes (ff_bvh.cu) on triangle sets whose
binary trees are as lopsided as they come: sizes and distances that halve from
one triangle to the next, single triangles up to counts around the leaf size
(3) and the node width (8).  Hits equal the oracle's brute force bit for bit
(the trace tests' tolerance: none)."""
from __future__ import annotations

import numpy as np
import pytest

from firefly_b200 import scenes
from tests.test_trace_gpu import _check_any, _check_closest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 7, 8, 9, 17, 33, 60, 257])
@pytest.mark.parametrize("ratio", [0.5, 0.97])
def test_lopsided_trees(ctx, oracle, n, ratio):
    import firefly_b200 as ff
    rng = np.random.default_rng(n)
    size = np.maximum(ratio ** np.arange(n), 1e-6)[:, None]
    centre = rng.uniform(-1, 1, (n, 3)) * size + np.array([8.0, 0.0, 0.0]) * size
    P = np.stack([centre + rng.uniform(-1, 1, (n, 3)) * size * 0.4 for _ in range(3)], 1)
    scn = scenes.Scene(positions=P.reshape(-1, 3).astype(np.float32),
                       indices=np.arange(3 * n, dtype=np.uint32).reshape(n, 3))
    ds = ff.dScene(ctx, scn)
    m = 4000
    k = rng.integers(0, n, m)
    target = P[k].mean(1) + rng.normal(size=(m, 3)) * size[k] * 0.1
    o = target + rng.normal(size=(m, 3)) * 5.0
    d = target - o
    rays = np.zeros((m, 8), np.float32)
    rays[:, 0:3], rays[:, 4:7] = o, d / np.linalg.norm(d, axis=1, keepdims=True)
    rays[:, 7] = np.inf
    _check_closest(scn, ds, oracle, rays)
    _check_any(scn, ds, oracle, rays)
    st = ds.stats()
    assert st["num_nodes"] <= max(1, n - 1) and st["bvh_depth"] <= 64
    ds.close()
