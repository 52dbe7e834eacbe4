"""Scenes whose build temporaries exceed what a context keeps between calls (256
MiB: 1.4M triangles take more): loaded twice, they give the same hits, and the
device gets everything back but that block."""
from __future__ import annotations

import numpy as np
import pytest

from firefly_b200 import scenes

pytestmark = pytest.mark.gpu


def test_large_scene_loaded_twice(ctx):
    import torch
    import firefly_b200 as ff
    rng = np.random.default_rng(0)
    n = 1_400_000
    T = (rng.uniform(-5, 5, (n, 1, 3)) + rng.uniform(-0.05, 0.05, (n, 3, 3))).astype(np.float32)
    scn = scenes.Scene(positions=T.reshape(-1, 3), indices=np.arange(3 * n, dtype=np.uint32).reshape(n, 3))
    rays = np.zeros((50_000, 8), np.float32)
    rays[:, 0:3] = rng.uniform(-5, 5, (len(rays), 3))
    d = rng.normal(size=(len(rays), 3))
    rays[:, 4:7], rays[:, 7] = d / np.linalg.norm(d, axis=1, keepdims=True), np.inf
    small = ff.dScene(ctx, scenes.small_room(seed=0))
    small.trace(rays)     # the staging of this many rays
    small.close()
    before = torch.cuda.mem_get_info(0)[0]
    hits = []
    for _ in range(2):
        ds = ff.dScene(ctx, scn)
        hits.append(ds.trace(rays).view(np.uint32))
        ds.close()
        assert torch.cuda.mem_get_info(0)[0] >= before - (256 << 20)
    assert np.array_equal(*hits)
    assert (hits[0].reshape(-1, 4)[:, 3].view(np.int32) >= 0).any()
