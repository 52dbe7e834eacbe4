"""The wavefront replay (FF_ADJOINT_REPLAY, and where the vertex records are
refused) against the one-thread-per-sample replay and the records: albedo,
roughness and environment gradients, odd films.  A call whose slots take one
sample each runs at most depth + 2 frames with records and more when it traces
every sample twice, so the frames tell which it was.  Tolerances as in
test_adjoint_gpu: the same terms, summed by float atomics in another order."""
from __future__ import annotations

import numpy as np
import pytest

from firefly_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture
def lab(ctx, request):
    import firefly_b200 as ff
    w, h, spp, depth, kind = request.param
    k = {"mix": ff.FF_MAT_MIX, "conductor": ff.FF_MAT_CONDUCTOR, "dielectric": ff.FF_MAT_DIELECTRIC,
         "coat": ff.FF_MAT_COAT}[kind]
    sky = scenes.sky_env(32, 16, seed=3, sun_radiance=8.0, sun_diameter_deg=20.0)
    scn = scenes.textured_room(seed=2, width=w, height=h, tex_res=16, env=sky, sphere_kind=k)
    ds = ff.dScene(ctx, scn)
    dimg = np.random.default_rng(1).standard_normal((h, w, 3)).astype(np.float32)

    def run(**kw):
        g = {"albedo": np.zeros_like(scn.textures[0]), "rough": np.zeros_like(scn.textures[1]),
             "env": np.zeros_like(scn.env_rgb)}
        st = ds.render_adjoint(w, h, dimg, texture=0, grad_texture=g["albedo"], grad_env=g["env"], spp=spp,
                               max_depth=depth, seed=5, light=-1, roughness_texture=1, grad_roughness=g["rough"], **kw)
        return g, st
    yield run, depth
    ds.close()


def _same(a, b):
    for name, floor in (("albedo", 1e-6), ("rough", 1e-6), ("env", 1e-5)):
        assert np.abs(b[name]).max() > 0, name
        assert np.allclose(a[name], b[name], rtol=1e-4, atol=floor * np.abs(b[name]).max()), name


CASES = [(33, 7, 3, 2, "mix"), (17, 31, 5, 7, "coat"), (65, 9, 2, 4, "dielectric"), (129, 3, 4, 3, "conductor")]


@pytest.mark.parametrize("lab", CASES, indirect=True)
def test_replay_matches_megakernel_and_records(lab):
    run, depth = lab
    g, st = run(replay=True)
    mega, sm = run(megakernel=True)
    rec, sr = run()
    _same(g, mega)
    _same(rec, mega)
    assert sr["frames"] <= depth + 2 < st["frames"]
    # both count the rays of both passes, traced once where the vertices are kept
    assert st["extension_rays"] + st["shadow_rays"] == sm["extension_rays"] == sr["extension_rays"] + sr["shadow_rays"]


@pytest.mark.parametrize("lab", CASES[:1], indirect=True)
def test_refused_records_are_replayed(lab):
    import firefly_b200 as ff
    run, depth = lab
    want, st = run(replay=True)      # the workspace is there, no records are held
    ff.lib().ff_debug_fail_alloc_after(0)
    try:
        g, sf = run()
    finally:
        ff.lib().ff_debug_fail_alloc_after(-1)
    assert sf["frames"] == st["frames"] > depth + 2
    _same(g, want)


@pytest.mark.parametrize("lab", [(256, 256, 16, 8, "mix")], indirect=True)
def test_replay_gives_the_records_back(lab):
    import torch
    run, depth = lab
    run()
    before = torch.cuda.mem_get_info(0)[0]
    run(replay=True)
    assert torch.cuda.mem_get_info(0)[0] >= before + 256 * 256 * 16 * depth * 48
