"""A cache whose copy of the coarse levels by cells was refused (its last
allocation, refused on the host) is created all the same, answers bit for bit
as one that has it, and trains."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from firefly_b200 import scenes
from tests.test_cache_gpu import random_records

pytestmark = pytest.mark.gpu


def test_refused_cells_change_no_answer(ctx):
    import firefly_b200 as ff
    from firefly_b200.cache import RadianceCache
    ds = ff.dScene(ctx, scenes.small_room(seed=0, width=64, height=64))
    total = C.c_uint64()
    count = lambda: (ff.lib().ff_debug_alloc_stats(C.byref(total), None), total.value)[1]
    before = count()
    full = RadianceCache(ds, log2_table_size=16, seed=3)
    made = count() - before
    ff.lib().ff_debug_fail_alloc_after(made - 1)
    try:
        bare = RadianceCache(ds, log2_table_size=16, seed=3)
    finally:
        ff.lib().ff_debug_fail_alloc_after(-1)
    rng = np.random.default_rng(5)
    mlp = rng.uniform(-1, 1, (5, 64, 64)).astype(np.float32) * np.float32(0.2)
    grid = rng.uniform(-1, 1, (16, 1 << 16, 2)).astype(np.float32)
    recs = random_records(ds.stats(), 5000, seed=4)
    for c in (full, bare):
        c.write_params(mlp=mlp, grid=grid)
    assert np.array_equal(full.query(recs), bare.query(recs))
    first = bare.train(recs)
    for _ in range(20):
        last = bare.train(recs)
    assert np.isfinite(last) and last < first
    bare.close()
    full.close()
    ds.close()
