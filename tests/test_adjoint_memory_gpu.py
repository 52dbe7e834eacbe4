"""The adjoint's vertex records are workspace, not the caller's loss: those of a
large call are freed when it returns, and those kept for the next one, like the
block of the scene builds' temporaries, go back to the device when an
allocation of the context is refused (on the host, before cudaMalloc), before
that call fails.  Free memory is the driver's (cudaMemGetInfo)."""
from __future__ import annotations

import numpy as np
import pytest

from firefly_b200 import scenes

pytestmark = pytest.mark.gpu

W = H = 512
SPP = 16
SLOTS = W * H * SPP


def test_records_go_back():
    import torch
    import firefly_b200 as ff
    from firefly_b200 import _abi as A
    free = lambda: torch.cuda.mem_get_info(0)[0]
    ctx = ff.Context(0)
    scn = scenes.textured_room(seed=2, width=W, height=H, tex_res=16, env_w=32, env_h=16)
    ds = ff.dScene(ctx, scn)
    dimg = np.full((H, W, 3), 1e-3, np.float32)

    def grad(depth):
        g = np.zeros_like(scn.textures[0])
        ds.render_adjoint(W, H, dimg, grad_texture=g, spp=SPP, max_depth=depth, seed=5)
        return g

    first = grad(3)
    kept = free()
    # 2.0 GB of records: as much memory is free after the call as with none held
    grad(15)
    assert free() >= kept
    again = grad(3)
    held = SLOTS * 3 * 32
    before = free()
    ff.lib().ff_debug_fail_alloc_after(0)
    try:
        with pytest.raises(ff.FireflyError) as e:
            ff.PathTracer(ctx, 64, 64)
    finally:
        ff.lib().ff_debug_fail_alloc_after(-1)
    assert e.value.status == A.FF_ERR_OOM
    assert free() >= before + held, "the refused call kept the records"
    last = grad(3)
    for g in (again, last):
        assert np.allclose(g, first, rtol=1e-4, atol=1e-5 * np.abs(first).max())
    ds.close()
    ctx.close()
