"""The work a program has this framework do, as cases that can be timed and compared.

listed() names them, draw() makes more of the same ranges, prepare() builds what the program holds before the call
(scene, film, cache, device buffers), run() is one pass through the public entry points (the Python classes, and the C
ABI with device pointers where those classes take host arrays only), work() the bytes and operations a pass cannot do
without, exact() the results in 64 bits where plain tensor code can state them.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

import firefly_b200 as ff
from firefly_b200 import _abi as A
from firefly_b200 import scenes
from firefly_b200.cache import RadianceCache

ROOM_TRIS, NODE_FLOPS = 4120, 400       # triangles of the small room; about the arithmetic of one ray in a shallow BVH
LEVELS, WIDTH = 16, 64                  # the cache's grid levels and its layer width
KINDS = {"mix": ff.FF_MAT_MIX, "diffuse": ff.FF_MAT_DIFFUSE, "conductor": ff.FF_MAT_CONDUCTOR,
         "dielectric": ff.FF_MAT_DIELECTRIC, "coat": ff.FF_MAT_COAT}


def listed():
    return [
        # a click in a viewer: what lies under a brush of some hundred pixels (host arrays, latency)
        dict(name="pick", op="trace", scene="room", rays=100, any=False, two=False, host=True),
        # the benchmark's trace micro workload: incoherent closest hits from device memory
        dict(name="trace_incoherent", op="trace", scene="room", rays=16777216, any=False, two=False, host=False),
        # visibility of an odd number of point pairs in the large mesh, as for baking occlusion
        dict(name="trace_shadow", op="trace", scene="mesh", subdiv=8, rays=3000017, any=True, two=False, host=False),
        # loading an asset of ordinary size under a sky, to its first hits
        dict(name="load", op="load", subdiv=6, env=1024, probe=4096),
        # an interactive preview: the reference's defaults (1 sample, depth 3, parity), image on the host
        dict(name="preview", op="draw", scene="room", kind="mix", w=256, h=256, spp=1, depth=3, corrected=False, light=0),
        # the small plain-tracer benchmark
        dict(name="draw_room", op="draw", scene="room", kind="mix", w=256, h=256, spp=16, depth=5, corrected=False,
             light=0),
        # the headline benchmark: the 1.3M-triangle mesh with five material kinds, full HD, 64 samples, depth 8
        dict(name="draw_scale", op="draw", scene="mesh", subdiv=8, kind="mix", w=1920, h=1080, spp=64, depth=8,
             corrected=True, light=-1),
        # one step of the inverse-rendering benchmark: new parameters in, primal render, gradients out (device)
        dict(name="inverse_step", op="inverse", w=512, h=512, spp=16, depth=3, tex=512, env=256),
        # gradients of a roughness texture on an odd film through host arrays (the tests' sizes)
        dict(name="adjoint_rough", op="rough", kind="conductor", w=97, h=61, spp=4, depth=5, tex=64, env=128),
        # radiance-cache queries of one full-HD frame
        dict(name="cache_query", op="query", n=2000003, table=19),
        # one optimiser step of the cache and its answers afterwards, the default batch
        dict(name="cache_train", op="train", n=16384, table=19, probe=4096),
        # the cached render of the benchmark: full HD, four frames with online training
        dict(name="cache_render", op="cached", w=1920, h=1080, frames=4, depth=5),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["trace", "trace", "load", "draw", "draw", "inverse", "rough", "query", "train", "cached"])
    if op == "trace":
        any_hit = rng.random() < 0.5
        host = rng.random() < 0.4
        c = dict(op=op, scene=rng.choice(["room", "mesh"]), rays=_log(rng, 1, 500_000 if host else 12_000_000), any=any_hit,
                 two=not any_hit and rng.random() < 0.3, host=host)
        return dict(c, subdiv=rng.randint(3, 6)) if c["scene"] == "mesh" else c
    if op == "load":
        return dict(op=op, subdiv=rng.randint(2, 6), env=_log(rng, 16, 2048), probe=_log(rng, 64, 20000))
    if op == "draw":
        scene = rng.choice(["room", "sky", "mesh", "pbr"])
        w, h = _log(rng, 33, 1600), _log(rng, 33, 1000)
        corrected = scene == "mesh" or rng.random() < 0.5
        light = 0 if scene == "room" else -1
        if corrected and rng.random() < 0.25:
            light = -2      # one light per vertex, chosen uniformly
        return dict(op=op, scene=scene, subdiv=rng.randint(3, 6), kind=rng.choice(sorted(KINDS)), w=w, h=h,
                    spp=max(1, min(_log(rng, 1, 64), 20_000_000 // (w * h))), depth=rng.randint(1, 8), corrected=corrected,
                    light=light)
    if op == "inverse":
        return dict(op=op, w=_log(rng, 31, 600), h=_log(rng, 31, 600), spp=_log(rng, 1, 16), depth=rng.randint(2, 5),
                    tex=_log(rng, 16, 512), env=_log(rng, 16, 1024))
    if op == "rough":
        return dict(op=op, kind=rng.choice(["mix", "conductor", "dielectric", "coat"]), w=_log(rng, 17, 300),
                    h=_log(rng, 17, 300), spp=_log(rng, 1, 16), depth=rng.randint(1, 6), tex=_log(rng, 8, 256),
                    env=_log(rng, 16, 512))
    if op == "query":
        return dict(op=op, n=_log(rng, 1, 4_000_000), table=rng.randint(14, 19))
    if op == "train":
        return dict(op=op, n=_log(rng, 64, 65536), table=rng.randint(14, 19), probe=_log(rng, 1, 8192))
    return dict(op=op, w=_log(rng, 200, 1920), h=_log(rng, 100, 1080), frames=rng.randint(1, 4), depth=rng.randint(2, 6))


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=None)
def _context():
    """One context for the program, on a torch stream so that tensor code and the library's launches keep their order."""
    stream = torch.cuda.Stream()
    return ff.Context(0, stream=stream.cuda_stream), stream


@functools.lru_cache(maxsize=None)
def _mesh(subdiv):
    """The displaced mesh (seconds to make at 8 subdivisions, so its geometry is made once in a process)."""
    return scenes.displaced_icosphere(subdiv=subdiv, seed=0, width=64, height=64, env_w=64, env_h=32)


@functools.lru_cache(maxsize=None)
def _sky(width, height):
    return scenes.sky_env(width, height, seed=0)


def _scene(c, seed):
    """The case's scene, with a camera, materials or sky of the seed's own."""
    rng = np.random.default_rng(seed)
    w, h = c.get("w", 64), c.get("h", 64)
    kind = KINDS[c.get("kind", "mix")]
    what = c.get("scene", "room")
    if what == "sky":
        return scenes.sphere_under_sky(seed=seed, width=w, height=h, kind=kind)
    if what == "pbr":
        return scenes.pbr_textured_room(seed=seed, width=w, height=h)
    if what == "mesh":
        base = _mesh(c["subdiv"])
        turn = rng.uniform(-0.5, 0.5)
        cam = scenes.make_camera(eye=(7.4 * math.sin(turn), 3.2, 7.4 * math.cos(turn)), center=(0.0, 2.2, 0.0), fovy=50.0,
                                 aspect=w / h, near=0.05, far=100.0)
        ew = c.get("env", 2048)
        env = _sky(ew, max(1, ew // 2)) * np.float32(rng.uniform(0.8, 1.2))
        return scenes.Scene(positions=base.positions, indices=base.indices, normals=base.normals,
                            material_ids=base.material_ids, materials=base.materials, env_rgb=env, camera=cam, width=w,
                            height=h)
    return scenes.small_room(seed=seed, width=w, height=h, kind=kind)


def _rays(scn, n, seed, any_hit):
    """Origins uniform in the scene's box, directions uniform on the sphere; any-hit rays end within some diagonals."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    lo, hi = (torch.tensor(b, device="cuda") for b in scn.bounds())
    r = torch.empty((n, 8), device="cuda")
    r[:, 0:3] = lo + (hi - lo) * torch.rand((n, 3), generator=g, device="cuda")
    r[:, 3] = 0
    r[:, 4:7] = torch.nn.functional.normalize(torch.randn((n, 3), generator=g, device="cuda"), dim=1)
    r[:, 7] = math.inf
    if any_hit:
        r[:, 7] = torch.linalg.norm(hi - lo) * (0.1 + 9.9 * torch.rand(n, generator=g, device="cuda"))
    return r


def _records(scn, n, seed):
    """Vertices on the scene's surfaces (n x 16 floats, ff_cache_record): what a frame asks the cache about, with a
    target radiance that varies smoothly over the scene."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    tri = torch.from_numpy(scn.triangle_soup()).cuda().reshape(-1, 3, 3)
    e1, e2 = tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    cross = torch.linalg.cross(e1, e2)
    area = torch.linalg.norm(cross, dim=1)
    k = torch.searchsorted(torch.cumsum(area, 0) / area.sum(), torch.rand(n, generator=g, device="cuda"))
    k = k.clamp(max=len(tri) - 1)
    u, v = torch.rand((2, n, 1), generator=g, device="cuda")
    u, v = torch.where(u + v > 1, 1 - u, u), torch.where(u + v > 1, 1 - v, v)
    pos = tri[k, 0] + u * e1[k] + v * e2[k]
    nrm = torch.nn.functional.normalize(cross[k], dim=1)
    wo = torch.nn.functional.normalize(torch.randn((n, 3), generator=g, device="cuda"), dim=1)
    wo = torch.where((wo * nrm).sum(1, keepdim=True) < 0, -wo, wo)
    val = 0.6 + 0.4 * torch.sin(pos * 0.7 + torch.tensor([0.0, 1.0, 2.0], device="cuda"))
    r = torch.zeros((n, 16), device="cuda")
    r[:, 0:3], r[:, 3] = pos, 0.25 + 0.75 * torch.rand(n, generator=g, device="cuda")
    r[:, 4:7], r[:, 7] = wo, val[:, 0]
    r[:, 8:11], r[:, 11], r[:, 13] = nrm, val[:, 1], val[:, 2]
    return r


def _params(table, seed):
    """Weights and grid features of a cache that has trained for a while."""
    g = torch.Generator(device="cuda").manual_seed(seed + 77)
    mlp = (torch.rand((5, WIDTH, WIDTH), generator=g, device="cuda") * 2 - 1) * math.sqrt(6 / (2 * WIDTH))
    mlp[4, 3:] = 0
    grid = (torch.rand((LEVELS, 1 << table, 2), generator=g, device="cuda") * 2 - 1) * 0.5
    return mlp.cpu().numpy(), grid.cpu().numpy()


class _State(dict):
    __getattr__ = dict.__getitem__


def prepare(case, seed):
    c = dict(case)
    ctx, stream = _context()
    op = c["op"]
    s = _State(case=c, ctx=ctx, stream=stream, seed=seed)
    if op == "load":
        s["scn"] = _scene(dict(c, scene="mesh"), seed)
        s["rays"] = _rays(s.scn, c["probe"], seed, False).cpu().numpy()
        return s
    if op in ("inverse", "rough"):
        rng = np.random.default_rng(seed)
        ew, eh = c["env"], max(1, c["env"] // 2)
        sky = scenes.sky_env(ew, eh, seed=seed, sun_radiance=8.0, sun_diameter_deg=20.0)
        scn = scenes.textured_room(seed=seed, width=c["w"], height=c["h"], tex_res=c["tex"], env=sky,
                                   sphere_kind=KINDS[c["kind"]] if op == "rough" else None)
        s["ds"] = ff.dScene(ctx, scn)
        if op == "rough":
            s["d_image"] = (rng.standard_normal((c["h"], c["w"], 3)) / (c["w"] * c["h"])).astype(np.float32)
            s["grad"] = np.zeros_like(scn.textures[1])
            s["grad_env"] = np.zeros_like(scn.env_rgb)
            return s
        s["pt"] = ff.PathTracer(ctx, c["w"], c["h"])
        # the fit's state part of the way: a flat albedo and the hazy sky, and a target image
        s["albedo"] = torch.full((c["tex"], c["tex"], 3), 0.5, device="cuda")
        s["env"] = torch.from_numpy(scn.env_rgb).cuda()
        s["target"] = torch.rand((c["h"], c["w"], 3), generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda")
        s["rgba"] = torch.empty((c["h"], c["w"], 4), device="cuda")
        s["count"] = torch.empty((c["h"], c["w"]), dtype=torch.int32, device="cuda")
        s["g_tex"], s["g_env"] = torch.zeros_like(s.albedo), torch.zeros_like(s.env)
        return s
    scn = _scene(c, seed)
    s["ds"] = ff.dScene(ctx, scn)
    if op == "trace":
        rays = _rays(scn, c["rays"], seed, c["any"])
        s["rays"] = rays.cpu().numpy() if c["host"] else rays
        if not c["host"]:
            s["hits"] = torch.empty((c["rays"], 4), device="cuda")
    elif op == "draw":
        s["pt"] = ff.PathTracer(ctx, c["w"], c["h"])
        s["device"] = c["w"] * c["h"] > 500_000
        if s.device:
            s["rgba"] = torch.empty((c["h"], c["w"], 4), device="cuda")
            s["count"] = torch.empty((c["h"], c["w"]), dtype=torch.int32, device="cuda")
    elif op in ("query", "train"):
        s["cache"] = RadianceCache(s.ds, log2_table_size=c["table"], seed=seed)
        mlp, grid = _params(c["table"], seed)
        s.cache.write_params(mlp=mlp, grid=grid)
        s["recs"] = _records(scn, c["n"], seed)
        n = c["n"] if op == "query" else c["probe"]
        s["rgb"] = torch.empty((n, 3), device="cuda")
        if op == "train":
            s["probe"] = _records(scn, n, seed + 1)
            s["loss"] = C.c_float()
    else:
        # past its first frames, as in all of a render but these, with the rate lowered for the fine fit
        s["cache"] = RadianceCache(s.ds, seed=seed, lr=1e-3)
        mlp, grid = _params(19, seed)
        s.cache.write_params(mlp=mlp, grid=grid)
        s["pt"] = ff.PathTracer(ctx, c["w"], c["h"])
        s["rgba"] = torch.empty((c["h"], c["w"], 4), device="cuda")
        s["count"] = torch.empty((c["h"], c["w"]), dtype=torch.int32, device="cuda")
    return s


# -------------------------------------------------------------------- passes
def _p(t):
    return C.c_void_p(t.data_ptr())


def _ok(status, ctx):
    if status != A.FF_OK:
        raise ff.FireflyError(status, ff.lib().ff_last_error_message(ctx.handle).decode())


def _film(s):
    """The film's sums and counts in the program's device tensors."""
    _ok(ff.lib().ff_film_read(s.pt.film, _p(s.rgba), _p(s.count), A.FF_MEM_DEVICE), s.ctx)
    return s.rgba, s.count


def run(s):
    c, L = s["case"], ff.lib()
    with torch.cuda.stream(s.stream):
        return _RUN[c["op"]](s, c, L)


def _run_trace(s, c, L):
    if c["host"]:
        h = s.ds.trace(s.rays, any_hit=c["any"], two_sided=c["two"])
        # any-hit queries answer whether something lies in the way (which occluder they met is open)
        return {"occluded": h["prim"] >= 0} if c["any"] else {k: h[k] for k in ("t", "u", "v", "prim")}
    s.ds.trace_device(s.rays.data_ptr(), c["rays"], s.hits.data_ptr(), any_hit=c["any"], two_sided=c["two"])
    prim = s.hits.view(torch.int32)[:, 3]
    if c["any"]:
        return {"occluded": prim >= 0}
    return {"t": s.hits[:, 0], "u": s.hits[:, 1], "v": s.hits[:, 2], "prim": prim}


def _run_load(s, c, L):
    ds = ff.dScene(s.ctx, s.scn)
    h = ds.trace(s.rays)
    st = ds.stats()
    ds.close()
    return {"t": h["t"], "u": h["u"], "v": h["v"], "prim": h["prim"], "box": np.array([st["scene_lo"], st["scene_hi"]])}


def _run_draw(s, c, L):
    s.pt.clear_buffer()
    s.pt.draw(s.ds, spp=c["spp"], max_depth=c["depth"], rr_depth=3, seed=s.seed, light=c["light"],
              mode=ff.FF_MODE_CORRECTED if c["corrected"] else ff.FF_MODE_PARITY)
    rgba, count = _film(s) if s.device else s.pt.read()
    return {"rgba": rgba, "count": count}


def _run_inverse(s, c, L):
    _ok(L.ff_scene_set_texture(s.ds.handle, 0, _p(s.albedo), A.FF_MEM_DEVICE), s.ctx)
    _ok(L.ff_scene_set_environment(s.ds.handle, _p(s.env), A.FF_MEM_DEVICE), s.ctx)
    s.pt.clear_buffer()
    s.pt.draw(s.ds, spp=c["spp"], max_depth=c["depth"], rr_depth=3, seed=s.seed, light=-1, mode=ff.FF_MODE_CORRECTED)
    rgba, count = _film(s)
    img = rgba[..., :3] / count[..., None]
    d_image = (img - s.target) / img.numel()
    s.g_tex.zero_()
    s.g_env.zero_()
    st = A.ff_render_settings(spp=c["spp"], max_depth=c["depth"], rr_depth=3, seed=s.seed + 0x40000000,
                              mode=A.FF_MODE_CORRECTED, light=-1, max_paths=0, sample_offset=0, flags=0, shadow_offset=0.001)
    d = A.ff_adjoint_desc(width=c["w"], height=c["h"], d_image=d_image.data_ptr(), texture=0,
                          grad_texture=s.g_tex.data_ptr(), grad_env=s.g_env.data_ptr(), flags=A.FF_MEM_DEVICE)
    _ok(L.ff_render_adjoint(s.ctx.handle, s.ds.handle, C.byref(st), C.byref(d), None), s.ctx)
    return {"image": img, "g_tex": s.g_tex, "g_env": s.g_env}


def _run_rough(s, c, L):
    s.grad[:] = 0
    s.grad_env[:] = 0
    s.ds.render_adjoint(c["w"], c["h"], s.d_image, texture=-1, grad_env=s.grad_env, spp=c["spp"], max_depth=c["depth"],
                        seed=s.seed, light=-1, roughness_texture=1, grad_roughness=s.grad)
    return {"g_rough": s.grad, "g_env": s.grad_env}


def _run_query(s, c, L):
    _ok(L.ff_cache_query(s.cache.handle, _p(s.recs), c["n"], _p(s.rgb), A.FF_MEM_DEVICE), s.ctx)
    return s.rgb


def _run_train(s, c, L):
    _ok(L.ff_cache_train(s.cache.handle, _p(s.recs), c["n"], A.FF_MEM_DEVICE, C.byref(s.loss)), s.ctx)
    _ok(L.ff_cache_query(s.cache.handle, _p(s.probe), c["probe"], _p(s.rgb), A.FF_MEM_DEVICE), s.ctx)
    return {"loss": float(s.loss.value), "answers": s.rgb}


def _run_cached(s, c, L):
    s.pt.clear_buffer()
    s.cache.render(s.ds, s.pt, frames=c["frames"], max_depth=c["depth"], rr_depth=3, seed=s.seed, light=0)
    rgba, count = _film(s)
    return {"rgba": rgba, "count": count}


_RUN = {"trace": _run_trace, "load": _run_load, "draw": _run_draw, "inverse": _run_inverse, "rough": _run_rough,
        "query": _run_query, "train": _run_train, "cached": _run_cached}


# ---------------------------------------------------------------------- work
def _tris(c):
    return 20 * 4 ** c["subdiv"] + 12 if c.get("scene") == "mesh" or c["op"] == "load" else ROOM_TRIS


def work(case):
    c, op = case, case["op"]
    if op == "trace":       # a ray in, a hit out; a scene is read once only where the rays can have visited it
        n = c["rays"]
        return {"bytes": 48 * n + min(_tris(c), n) * 48, "flops": n * NODE_FLOPS}
    if op == "load":        # vertices, indices and the sky in; triangles, normals and tables out
        texels = c["env"] * max(1, c["env"] // 2)
        return {"bytes": _tris(c) * (24 + 12 + 48 + 80 + 20) + texels * (12 + 28) + 48 * c["probe"], "flops": _tris(c) * 500}
    if op in ("draw", "cached"):    # the film out, the scene in; about two bounces of three rays a sample
        n = c["w"] * c["h"] * c.get("spp", c.get("frames"))
        tris = _tris(c) if c.get("scene") == "mesh" else ROOM_TRIS
        return {"bytes": c["w"] * c["h"] * 20 + min(tris, 2 * n) * 128, "flops": n * min(c["depth"], 3) * 3 * NODE_FLOPS}
    if op in ("inverse", "rough"):
        n, texels = c["w"] * c["h"] * c["spp"], c["tex"] ** 2 * 24 + c["env"] ** 2 * 12
        return {"bytes": c["w"] * c["h"] * 32 + texels, "flops": n * min(c["depth"], 3) * 9 * NODE_FLOPS}
    n = c["n"]
    net = 2 * (4 * WIDTH * WIDTH + 3 * WIDTH)
    if op == "query":       # a record in, three floats out, the grid's half-precision entries that it reads at most once each
        return {"bytes": n * 76 + min(LEVELS << c["table"], n * 128) * 4, "flops": n * net}
    touched = min(LEVELS << c["table"], n * 128)
    return {"bytes": n * 64 + c["probe"] * 76 + touched * 2 * 4 * 7, "flops": 3 * n * net + c["probe"] * net}


# --------------------------------------------------------------------- exact
def _exact_hits(scn, rays):
    """Closest front-facing hits by testing every triangle in 64 bits."""
    tri = torch.from_numpy(scn.triangle_soup()).cuda().double().reshape(-1, 3, 3)
    v0, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    out = []
    for r in torch.from_numpy(rays).cuda().double().split(256):
        o, d = r[:, None, 0:3], r[:, None, 4:7].expand(-1, len(v0), -1)
        p = torch.linalg.cross(d, e2[None].expand_as(d))
        det = (p * e1).sum(-1)
        tv = o - v0
        q = torch.linalg.cross(tv, e1[None].expand_as(tv))
        u, v, t = ((tv * p).sum(-1) / det, (d * q).sum(-1) / det, (q * e2).sum(-1) / det)
        hit = (det > 1e-6) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= 0)
        best = torch.where(hit, t, math.inf).min(1)
        k = best.indices[:, None]
        out.append(torch.stack([best.values, u.gather(1, k)[:, 0], v.gather(1, k)[:, 0]]))
    t, u, v = torch.cat(out, 1).cpu().numpy()
    return {"t": t, "u": u, "v": v, "prim": None}


def _exact_answers(scn, recs, mlp, grid, table):
    """The cache's network on the records, in 64 bits with unrounded weights, features and activations."""
    lo, hi = (torch.tensor(b, device="cuda").double() for b in scn.bounds())
    grow = (hi - lo) * 0.01 + 1e-4
    mlp, grid = torch.from_numpy(mlp).cuda().double(), torch.from_numpy(grid).cuda()
    base = math.exp(math.log(2048 / 16) / (LEVELS - 1))
    out = []
    for r in recs.double().split(1 << 17):
        p = ((r[:, 0:3] - (lo - grow)) / (hi - lo + 2 * grow)).clamp(0, 1)
        feats = []
        for l in range(LEVELS):
            cells = int(math.floor(16 * base ** l + 1e-9))
            f = p * cells
            i = f.floor().long().clamp(0, cells - 1)
            t = (f - i).clamp(0, 1)
            acc = 0
            for k in range(8):
                bit = [(k >> a) & 1 for a in range(3)]
                x, y, z = (i[:, a] + bit[a] for a in range(3))
                if (cells + 1) ** 3 <= 1 << table:
                    h = x + (cells + 1) * (y + (cells + 1) * z)
                else:
                    h = x ^ ((y * 2654435761) & 0xFFFFFFFF) ^ ((z * 805459861) & 0xFFFFFFFF)
                wt = math.prod(t[:, a] if bit[a] else 1 - t[:, a] for a in range(3))
                acc = acc + grid[l][h & ((1 << table) - 1)].double() * wt[:, None]
            feats.append(acc)
        x, y, z = r[:, 4], r[:, 5], r[:, 6]
        pi, xx, yy, zz = math.pi, x * x, y * y, z * z
        s15, s105 = math.sqrt(15 / pi) / 2, math.sqrt(105 / pi)
        a, b, e = math.sqrt(3 / (4 * pi)), math.sqrt(35 / (2 * pi)) / 4, math.sqrt(21 / (2 * pi)) / 4
        sh = torch.stack([torch.full_like(x, 0.5 / math.sqrt(pi)), -a * y, a * z, -a * x, s15 * x * y, -s15 * y * z,
                          math.sqrt(5 / pi) / 4 * (3 * zz - 1), -s15 * x * z, s15 / 2 * (xx - yy), -b * y * (3 * xx - yy),
                          s105 / 2 * x * y * z, -e * y * (5 * zz - 1), math.sqrt(7 / pi) / 4 * z * (5 * zz - 3),
                          -e * x * (5 * zz - 1), s105 / 4 * z * (xx - yy), -b * x * (xx - 3 * yy)], 1)
        act = torch.cat(feats + [sh, r[:, 8:11], r[:, 3:4], torch.ones_like(r[:, :1]), torch.zeros_like(r[:, :11])], 1)
        for l in range(4):
            act = torch.relu(act @ mlp[l].T)
        out.append(act @ mlp[4, :3].T)
    return torch.cat(out)


def exact(case, seed):
    c = case
    if c["op"] == "trace" and c["scene"] == "room" and not c["any"] and not c["two"] and c["rays"] <= 4096:
        scn = _scene(c, seed)
        out = _exact_hits(scn, _rays(scn, c["rays"], seed, False).cpu().numpy())
        return out
    if c["op"] in ("query", "train"):
        scn = _scene(c, seed)
        recs = _records(scn, c["n"], seed)
        y = _exact_answers(scn, recs, *_params(c["table"], seed), c["table"])
        if c["op"] == "query":
            return y
        target = recs[:, [7, 11, 13]].double()
        return {"loss": float((((y - target) ** 2) / (y * y + 0.01)).sum(1).mean()), "answers": None}
    return None     # path-traced estimates: a 64-bit tracer takes other paths where a rounding decides
