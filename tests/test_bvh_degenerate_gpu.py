"""The collapse where boxes have no area, or one that overflows: duplicates of
one point, points on a line along an axis (evenly spaced, and halving), and
triangles spread over 1e25.  Every split costs the same there, so the tree has
to be kept wide by count: a node that has an internal child uses all 8 slots,
and the tree stays shallow.  With ordinary triangles beside them, hits equal the
oracle's brute force bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from firefly_b200 import scenes
from tests.test_trace_gpu import _check_any, _check_closest

pytestmark = pytest.mark.gpu


def _points(what, n, rng):
    """n triangles (n x 3 x 3) of zero area, or large ones far apart."""
    c = np.zeros((n, 3))
    if what == "line":
        c[:, 1] = np.linspace(-3.0, 5.0, n)
    elif what == "halving":
        c[:, 2] = 0.5 ** (np.arange(n) % 60)
    elif what == "huge":
        return rng.uniform(-1e25, 1e25, (n, 1, 3)) + rng.uniform(-1e22, 1e22, (n, 3, 3))
    return np.repeat(c[:, None], 3, 1)


def _scene(T):
    return scenes.Scene(positions=T.reshape(-1, 3).astype(np.float32),
                        indices=np.arange(3 * len(T), dtype=np.uint32).reshape(-1, 3))


@pytest.mark.parametrize("what", ["point", "line", "halving", "huge"])
@pytest.mark.parametrize("n", [4, 25, 5000])
def test_trees_without_areas_stay_wide(ctx, what, n):
    import firefly_b200 as ff
    ds = ff.dScene(ctx, _scene(_points(what, n, np.random.default_rng(n))))
    nodes, _ = ds.read_bvh()
    used = (nodes[:, 24:32] != 0).sum(1)
    inner = nodes[:, 15] != 0
    assert (used[inner] == 8).all(), np.bincount(used[inner])
    # equal keys split by position: 5000 < 8^4 leaf-sized subtrees; each halving of the distance is one level at most
    assert ds.stats()["bvh_depth"] <= (8 if what != "halving" else 21)
    ds.close()


@pytest.mark.parametrize("what", ["point", "line", "halving"])
def test_hits_beside_triangles_without_area(ctx, oracle, what):
    import firefly_b200 as ff
    rng = np.random.default_rng(3)
    T = rng.uniform(-2, 2, (300, 1, 3)) + rng.uniform(-0.6, 0.6, (300, 3, 3))
    scn = _scene(rng.permutation(np.concatenate([T, _points(what, 700, rng)])))
    ds = ff.dScene(ctx, scn)
    m = 4000
    o = rng.normal(size=(m, 3)) * 4.0
    d = rng.uniform(-2, 2, (m, 3)) - o
    rays = np.zeros((m, 8), np.float32)
    rays[:, 0:3], rays[:, 4:7], rays[:, 7] = o, d / np.linalg.norm(d, axis=1, keepdims=True), np.inf
    _check_closest(scn, ds, oracle, rays)
    _check_any(scn, ds, oracle, rays)
    ds.close()
