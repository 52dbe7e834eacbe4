"""Few rays (eight lanes a ray) give the same bits as many (a lane a ray):
the first n of a set traced alone, at the edges of the blocks (16 rays), of the
switch (40,960 rays) and at one ray, equal the same rays inside a set large
enough for the other kernel; closest, two-sided and any hits (occluder and t
included)."""
from __future__ import annotations

import numpy as np
import pytest

from firefly_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sets(ctx):
    import firefly_b200 as ff
    out = {}
    for name, scn in (("room", scenes.small_room(seed=0)),
                      ("mesh", scenes.displaced_icosphere(subdiv=4, width=64, height=64, env_w=16, env_h=8))):
        ds = ff.dScene(ctx, scn)
        rays = scenes.incoherent_rays(scn, 60_000, seed=9)
        rays[::7, 4:7] = np.eye(3, dtype=np.float32)[np.arange(len(rays[::7])) % 3]      # along the axes
        rays[::11, 3] = 0.5
        rays[::13, 7] = 3.0
        out[name] = ds, rays, scenes.with_random_tmax(rays, scn)
    yield out
    for ds, _, _ in out.values():
        ds.close()


@pytest.mark.parametrize("scene", ["room", "mesh"])
@pytest.mark.parametrize("kind", ["closest", "two_sided", "any"])
def test_few_rays_equal_many(sets, scene, kind):
    ds, rays, anyr = sets[scene]
    r = anyr if kind == "any" else rays
    kw = dict(any_hit=kind == "any", two_sided=kind == "two_sided")
    many = ds.trace(r, **kw)
    for n in (1, 2, 15, 16, 17, 1000, 40960, 40961):
        few = ds.trace(r[:n], **kw)
        assert np.array_equal(few.view(np.uint32), many[:n].view(np.uint32)), n


@pytest.mark.parametrize("kind", ["closest", "two_sided", "any"])
def test_rays_taken_by_the_pool(sets, kind):
    """Sets large enough for the warps to take 64 rays at a time, ending at and
    around the sizes where they begin to (two rays a resident thread): the
    60,000 rays over and over give each time the bits that they give alone."""
    ds, rays, anyr = sets["room"]
    r = anyr if kind == "any" else rays
    kw = dict(any_hit=kind == "any", two_sided=kind == "two_sided")
    one = ds.trace(r, **kw).view(np.uint32).reshape(-1, 4)
    for n in (606_207, 606_208, 606_273, 1_000_003):
        got = ds.trace(r[np.arange(n) % len(r)], **kw).view(np.uint32).reshape(-1, 4)
        assert np.array_equal(got, one[np.arange(n) % len(r)]), n
