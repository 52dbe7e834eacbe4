"""Traversal errors of device-pointer traces, which nothing waits for, stay
counted on the context until a call that waits reports them: every host-pointer
ff_trace, through either staging (up to 8,192 rays and more), and
ff_trace_count.  The count is set from the host."""
from __future__ import annotations

import numpy as np
import pytest

from firefly_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 8192, 8193])
@pytest.mark.parametrize("any_hit", [False, True])
def test_a_host_trace_reports_and_clears_the_count(ctx, n, any_hit):
    import firefly_b200 as ff
    from firefly_b200 import _abi as A
    scn = scenes.small_room(seed=0)
    ds = ff.dScene(ctx, scn)
    rays = scenes.incoherent_rays(scn, n, seed=1)
    want = ds.trace(rays, any_hit=any_hit)
    assert ff.lib().ff_debug_trace_errors(ctx.handle, 3) == A.FF_OK
    with pytest.raises(ff.FireflyError) as e:
        ds.trace(rays, any_hit=any_hit)
    assert e.value.status == A.FF_ERR_INTERNAL
    assert np.array_equal(ds.trace(rays, any_hit=any_hit).view(np.uint32), want.view(np.uint32)), "reported once"
    ds.close()
