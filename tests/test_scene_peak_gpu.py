"""A large scene's load holds no more memory at once than the tree's build needs
beside positions, indices and the tree itself: what comes after the tree (shading
attributes, normals, textures) is allocated after it, and the build's
temporaries are gone by then.  In bytes a triangle: positions and indices 48
(no shared vertices), nodes 40, triangle records 48, and of temporaries the
records 48, boxes 24, sorted keys and order 12, unsorted ones with the
centroids 24 and the sort's own 12 and a little, binary nodes 40, parents and
arrivals 12, queues 8, the check of the references 4."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from firefly_b200 import scenes

pytestmark = pytest.mark.gpu


def test_peak_of_a_large_load(ctx):
    import firefly_b200 as ff
    rng = np.random.default_rng(0)
    n = 7_000_000
    T = rng.random((n, 1, 3), dtype=np.float32) * 10 + rng.random((n, 3, 3), dtype=np.float32) * np.float32(0.05)
    N = np.zeros((3 * n, 3), np.float32)
    N[:, 1] = 1
    scn = scenes.Scene(positions=T.reshape(-1, 3), indices=np.arange(3 * n, dtype=np.uint32).reshape(n, 3), normals=N)
    peak = C.c_uint64()
    ff.lib().ff_debug_alloc_peak(None)
    ff.lib().ff_debug_alloc_peak(C.byref(peak))
    held = peak.value
    ds = ff.dScene(ctx, scn)
    ff.lib().ff_debug_alloc_peak(C.byref(peak))
    assert peak.value - held <= 320 * n * 1.01 + (64 << 20), (peak.value - held) / n
    rays = scenes.incoherent_rays(scn, 10_000, seed=1)
    assert (ds.trace(rays)["prim"] >= 0).any()
    ds.close()
