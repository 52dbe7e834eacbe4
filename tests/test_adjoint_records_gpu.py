"""The adjoint with vertex records (one trace per sample) against the
one-thread-per-sample replay, where records and film do not line up with
blocks: odd films, depths 1 to 7, albedo, roughness and environment gradients
alone and together.  Tolerances as in test_adjoint_gpu: the same terms, summed
by float atomics in another order (1e-4 relative, floors of 1e-6 of the largest
texel, 1e-5 for the environment, whose texels sum the most atomics)."""
from __future__ import annotations

import numpy as np
import pytest

from firefly_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,spp,depth,kind", [(1, 1, 1, 1, "conductor"), (33, 7, 3, 2, "mix"), (17, 31, 5, 7, "coat"),
                                                (65, 9, 2, 4, "dielectric")])
@pytest.mark.parametrize("want", ["albedo", "rough", "env", "all"])
def test_records_match_megakernel(ctx, w, h, spp, depth, kind, want):
    import firefly_b200 as ff
    k = {"mix": ff.FF_MAT_MIX, "conductor": ff.FF_MAT_CONDUCTOR, "dielectric": ff.FF_MAT_DIELECTRIC,
         "coat": ff.FF_MAT_COAT}[kind]
    sky = scenes.sky_env(32, 16, seed=3, sun_radiance=8.0, sun_diameter_deg=20.0)
    scn = scenes.textured_room(seed=2, width=w, height=h, tex_res=16, env=sky, sphere_kind=k)
    ds = ff.dScene(ctx, scn)
    dimg = np.random.default_rng(1).standard_normal((h, w, 3)).astype(np.float32)
    got = []
    for mega in (False, True):
        g = {"albedo": np.zeros_like(scn.textures[0]), "rough": np.zeros_like(scn.textures[1]),
             "env": np.zeros_like(scn.env_rgb)}
        on = lambda name: g[name] if want in (name, "all") else None
        st = ds.render_adjoint(w, h, dimg, texture=0 if want in ("albedo", "all") else -1, grad_texture=on("albedo"),
                               grad_env=on("env"), spp=spp, max_depth=depth, seed=5, light=-1,
                               roughness_texture=1 if want in ("rough", "all") else -1, grad_roughness=on("rough"),
                               megakernel=mega)
        got.append((g, st["extension_rays"] + st["shadow_rays"]))
    assert got[0][1] == got[1][1]
    for name, floor in (("albedo", 1e-6), ("rough", 1e-6), ("env", 1e-5)):
        a, b = got[0][0][name], got[1][0][name]
        assert np.allclose(a, b, rtol=1e-4, atol=floor * max(np.abs(b).max(), 1e-30)), name
    ds.close()


def test_replay_beyond_the_record_budget(ctx):
    """8.4M slots at depth 15 with a roughness texture would take 6 GB of
    records: the samples are replayed.  Positive image gradients, so that no
    texel's sum cancels; the floor is the environment's above, as each texel
    sums thousands of atomics."""
    import firefly_b200 as ff
    w, h, spp, depth = 512, 512, 32, 15
    scn = scenes.textured_room(seed=2, width=w, height=h, tex_res=16, env_w=32, env_h=16, sphere_kind=ff.FF_MAT_COAT)
    ds = ff.dScene(ctx, scn)
    dimg = np.full((h, w, 3), 1e-3, np.float32)
    g = [[np.zeros_like(t) for t in scn.textures] for _ in range(2)]
    st = [ds.render_adjoint(w, h, dimg, grad_texture=g[m][0], roughness_texture=1, grad_roughness=g[m][1], spp=spp,
                            max_depth=depth, seed=5, megakernel=bool(m)) for m in (0, 1)]
    assert st[0]["extension_rays"] + st[0]["shadow_rays"] == st[1]["extension_rays"]
    assert np.allclose(g[0][0], g[1][0], rtol=1e-4, atol=1e-5 * np.abs(g[1][0]).max())
    ds.close()
