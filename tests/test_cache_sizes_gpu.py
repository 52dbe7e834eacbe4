"""Cache queries and gradients at the edges of tiles (128 rows), of the switch
from one tile a CTA to several (296 tiles on 148 SMs) and of the levels kept by
cells (none, some, all dense levels of small and large tables), against the
float32 restatement of test_cache_gpu and against each other.  Tolerances: an
answer does not depend on the batch it is in (equal bits).  Against the
restatement: sums in another order (relative 1e-7) can round an activation to
the other of two bf16 neighbours (2^-8 apart), about once in 10^4 activations,
i.e. in some percent of the records; such a record is off by at most a few
2^-8 of the output scale, the mean by 1e-4 of it."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from firefly_b200 import scenes
from tests.test_cache_gpu import Ref, random_records

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log2_T,base,maxres", [(10, 2, 64), (12, 16, 16), (14, 16, 512), (19, 16, 2048), (20, 90, 128)])
def test_sizes_and_levels(ctx, log2_T, base, maxres):
    import firefly_b200 as ff
    from firefly_b200.cache import RadianceCache
    scn = scenes.small_room(seed=0, width=64, height=64)
    ds = ff.dScene(ctx, scn)
    cache = RadianceCache(ds, log2_table_size=log2_T, base_resolution=base, max_resolution=maxres)
    ref = Ref(ds.stats(), log2_T=log2_T, base=base, maxres=maxres)
    rng = np.random.default_rng(5)
    mlp = rng.uniform(-1, 1, (5, 64, 64)).astype(np.float32) * np.float32(0.2)
    mlp[4, 3:] = 0
    grid = rng.uniform(-1, 1, (16, 1 << log2_T, 2)).astype(np.float32)
    cache.write_params(mlp=mlp, grid=grid)
    n = 296 * 128 + 129
    recs = random_records(ds.stats(), n, seed=4)
    recs["pos"][:8] = [[x, y, z] for x in (-9, 9) for y in (-9, 19) for z in (-9, 9)]     # outside: clamped corners
    full = cache.query(recs)
    grid_h = torch.from_numpy(grid.reshape(-1, 2)).half().float()
    want = ref.forward(recs[:3000], torch.from_numpy(mlp), grid_h).numpy()
    err, scale = np.abs(full[:3000] - want), np.abs(want).max()
    assert err.max() <= 2 ** -6 * scale and err.mean() <= 1e-4 * scale
    for k in (1, 127, 128, 129, 296 * 128, 296 * 128 + 1):
        assert np.array_equal(cache.query(recs[:k]), full[:k]), k
    # one step moves the table; the copy by cells follows: the answers equal those of a cache given the same parameters
    cache.train(recs[:500])
    p = cache.read_params()
    other = RadianceCache(ds, log2_table_size=log2_T, base_resolution=base, max_resolution=maxres)
    other.write_params(mlp=p["mlp"], grid=p["grid"])
    assert np.array_equal(other.query(recs[:3000]), cache.query(recs[:3000]))
    other.close()
    cache.close()
    ds.close()
