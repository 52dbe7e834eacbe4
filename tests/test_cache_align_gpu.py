"""Device records of the radiance cache are read in 32-byte accesses where they
sit on a 32-byte boundary, in 16-byte ones where they sit 16 bytes past one:
the same answers and, from one tile of records (one atomic per weight), the same
weight gradients, bit for bit."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from firefly_b200 import scenes
from tests.test_cache_gpu import random_records

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 128, 1000])
def test_records_off_the_sector_boundary(ctx, n):
    import torch
    import firefly_b200 as ff
    from firefly_b200 import _abi as A
    from firefly_b200.cache import RadianceCache
    ds = ff.dScene(ctx, scenes.small_room(seed=0, width=64, height=64))
    cache = RadianceCache(ds, log2_table_size=14)
    recs = torch.from_numpy(random_records(ds.stats(), n, seed=4).view(np.float32).reshape(n, 16))
    rgb, grads = [], []
    for off in (0, 4):      # floats past the allocation's start
        buf = torch.zeros(16 * n + 8, device="cuda")
        buf[off:off + 16 * n] = recs.reshape(-1).cuda()
        out = torch.empty((n, 3), device="cuda")
        torch.cuda.synchronize()
        p = C.c_void_p(buf.data_ptr() + 4 * off)
        assert ff.lib().ff_cache_query(cache.handle, p, n, C.c_void_p(out.data_ptr()), A.FF_MEM_DEVICE) == A.FF_OK
        cache.reset()
        loss = C.c_float()
        assert ff.lib().ff_cache_train(cache.handle, p, min(n, 128), A.FF_MEM_DEVICE | A.FF_CACHE_GRADIENTS_ONLY,
                                       C.byref(loss)) == A.FF_OK
        rgb.append(out.cpu())
        grads.append(cache.read_params()["grad_mlp"])
    assert torch.equal(*rgb)
    assert np.abs(grads[0]).max() > 0 and np.array_equal(*grads)
    cache.close()
    ds.close()
