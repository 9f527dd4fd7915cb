"""The renders, ray casts and job mixes whose speed is measured.

Each case is a call (or the few calls) that a program using the package makes
over and over, through its public entry points: `Scene.render`,
`Scene.render_paths`, `Scene.trace`, `Scene.refit`, `Context.batch_render`
and the job `Server`.  The scenes are the seeded synthetic ones of
`raytracer_gb300.scenes`; a case's seed moves their geometry, colours or sky
and chooses the sample streams.
"""
import math
import random

import numpy as np
import torch

import raytracer_gb300 as R
from raytracer_gb300 import desc as D
from raytracer_gb300 import scenes as S


def listed():
    return [
        # The plugin's per-sample Integrator::li: a host renderer asks for the
        # radiance of a few path samples at a time.
        dict(name="li_33_paths", kind="li", scene="cornell", width=256, height=256, paths=33),
        # Ray casting for a caller with rays of its own (picking, visibility,
        # baking): closest hits, then occlusion of the same rays.
        dict(name="cast_300k_rays", kind="rays", level=5, rays=300_000),
        # An interactive preview of moving geometry: new vertex positions in
        # device memory, then a few samples of a small odd-sized frame.
        dict(name="refit_preview", kind="preview", level=5, width=171, height=121, spp=4, depth=8),
        # The Cornell-box configuration: a whole small frame, diffuse, one
        # area light.
        dict(name="cornell_256_16spp", kind="frame", scene="cornell", width=256, height=256, spp=16, depth=8,
             filter="box", host=False),
        # A scene file's usual options together: textures, the Gaussian
        # reconstruction filter, an odd frame size, the film back on the host
        # as the command line renders it.
        dict(name="textured_gauss_301x203", kind="frame", scene="textured", width=301, height=203, spp=25, depth=10,
             filter="gauss", host=True),
        # Every light sampled at every vertex (the reference's default
        # strategy), with a mesh, a point and a spot light.
        dict(name="all_lights_333x257", kind="frame", scene="delta", width=333, height=257, spp=32, depth=8,
             filter="box", host=False),
        # The furnished room: every smooth BSDF, a large frame.
        dict(name="smooth_room_1024", kind="frame", scene="smooth", width=1024, height=1024, spp=16, depth=12,
             filter="box", host=False),
        # The large-mesh configuration (1.31 M triangles, four BSDF families,
        # environment light) at its full size: the headline frame.
        dict(name="icosphere_l8_1024_64spp", kind="frame", scene="icosphere", level=8, width=1024, height=1024,
             spp=64, depth=16, filter="box", host=False),
        # A small volumetric frame of ragged size, film on the host.
        dict(name="volume_133x97_9spp", kind="frame", scene="volume", level=64, width=133, height=97, spp=9, depth=64,
             filter="box", host=True),
        # The grid-medium configuration at its full size.
        dict(name="volume_512_128spp", kind="frame", scene="volume", level=128, width=512, height=512, spp=128,
             depth=64, filter="box", host=False),
        # A render farm's batch: scenes of uneven size in one call, films in
        # device memory.
        dict(name="batch_12_jobs", kind="batch", jobs=12, mix=5, max_level=6, max_spp=48),
        # A burst of jobs at the server, each rendered to a target error on
        # the displayed image; one in five volumetric.
        dict(name="serve_6_jobs", kind="serve", jobs=6, mix=3, max_level=5, max_spp=96),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _odd_size(rng, lo, hi):
    """A frame side: any number of pixels, a power of two now and then."""
    n = _log_int(rng, lo, hi)
    return 1 << (n.bit_length() - 1) if rng.random() < 0.25 else n


def draw(rng):
    kind = rng.choice(["li", "rays", "preview", "frame", "frame", "frame", "frame", "volume", "volume", "batch", "serve"])
    if kind == "li":
        return dict(kind="li", scene=rng.choice(["cornell", "smooth", "textured"]), width=_odd_size(rng, 64, 512),
                    height=_odd_size(rng, 64, 512), paths=_log_int(rng, 1, 4096))
    if kind == "rays":
        return dict(kind="rays", level=rng.randint(3, 6), rays=_log_int(rng, 1000, 1_000_000))
    if kind == "preview":
        return dict(kind="preview", level=rng.randint(4, 6), width=_odd_size(rng, 64, 400),
                    height=_odd_size(rng, 64, 400), spp=rng.randint(1, 8), depth=rng.randint(3, 16))
    if kind == "batch":
        return dict(kind="batch", jobs=rng.randint(2, 16), mix=rng.randrange(1000), max_level=6,
                    max_spp=_log_int(rng, 8, 64))
    if kind == "serve":
        return dict(kind="serve", jobs=rng.randint(2, 8), mix=rng.randrange(1000), max_level=5,
                    max_spp=_log_int(rng, 24, 128))
    if kind == "volume":
        w, h = _odd_size(rng, 48, 512), _odd_size(rng, 48, 512)
        return dict(kind="frame", scene="volume", level=rng.choice([32, 64]), width=w, height=h,
                    spp=_log_int(rng, 2, 64), depth=rng.choice([16, 64]), filter="box", host=rng.random() < 0.5)
    scene = rng.choice(["cornell", "textured", "delta", "smooth", "icosphere", "icosphere", "icosphere"])
    w, h = _odd_size(rng, 64, 1024), _odd_size(rng, 64, 1024)
    filt = rng.choice(["box", "box", "box", "gauss", "mitchell"])
    c = dict(kind="frame", scene=scene, width=w, height=h, spp=_log_int(rng, 1, 64 if filt == "box" else 16),
             depth=rng.choice([5, 8, 12, 16]), filter=filt, host=rng.random() < 0.5)
    if scene == "icosphere":
        c["level"] = rng.randint(3, 7)
    return c


# ------------------------------------------------------------------ scenes
def _tint(s, rng):
    """Other wall colours for another seed."""
    for b in s.bsdfs:
        if b["type"] == D.BSDF_DIFFUSE:
            b["albedo"] = tuple(float(np.clip(a * rng.uniform(0.85, 1.1), 0.0, 0.95)) for a in b["albedo"])


def _icosphere(level, width, height, depth, seed, env=None):
    if env is None:
        env, _ = S.sky_env(1024, 512, sun_azim_deg=20.0 + 37.0 * (seed % 8), sun_elev_deg=25.0 + 3.0 * (seed % 5))
    return S.displaced_icosphere(level=level, width=width, height=height, seed=seed % 100003, max_depth=depth, env=env)


def _scene(name, width, height, depth, seed, level=None):
    rng = np.random.default_rng(seed)
    if name == "icosphere":
        return _icosphere(level, width, height, depth, seed)
    if name == "volume":
        return S.volume_grid(width, height, res=level, seed=seed % 100003, max_depth=depth)
    if name == "cornell":
        s = S.cornell_box(width, height)
    elif name == "smooth":
        s = S.cornell_smooth(width, height)
    elif name == "textured":
        s = S.textured_room(width, height)
    else:
        s = S.cornell_delta_lights(width, height)
        s.integrator = dict(s.integrator, strategy=D.STRATEGY_ALL_LIGHTS)
    _tint(s, rng)
    s.integrator = dict(s.integrator, max_depth=depth)
    return s


def _rays(n, rng):
    """Rays from a shell around the sphere toward it, half of them aimed to
    pass near its surface; a tenth start on the ground."""
    o = rng.normal(size=(n, 3))
    o *= (rng.uniform(1.8, 6.0, (n, 1)) / np.linalg.norm(o, axis=1, keepdims=True))
    o[:, 1] = np.abs(o[:, 1]) + 0.05
    g = rng.random(n) < 0.1
    o[g, 1] = 1e-3
    t = rng.normal(size=(n, 3))
    t *= rng.uniform(0.0, 1.3, (n, 1)) / np.linalg.norm(t, axis=1, keepdims=True)
    t += np.array([0.0, 1.15, 0.0])
    d = t - o
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    r = np.zeros(n, D.RAY_DTYPE)
    r["o"], r["d"], r["mint"], r["maxt"] = o, d, 1e-4, 1e4
    return r


def _mix(case):
    """Sizes of a job mix: fixed by the case, so that every seed costs alike."""
    rng = random.Random(case["mix"])
    jobs = []
    for _ in range(case["jobs"]):
        jobs.append(dict(level=rng.randint(3, case["max_level"]), res=rng.choice([128, 192, 256, 512]),
                         spp=_log_int(rng, 4, case["max_spp"]), volume=rng.random() < 0.2))
    return jobs


# ------------------------------------------------------------------ prepare / run
def prepare(case, seed):
    ctx = R.Context(0)
    k = case["kind"]
    if k == "li":
        rng = np.random.default_rng(seed)
        s = R.Scene(ctx, _scene(case["scene"], case["width"], case["height"], 8, seed))
        n = case["paths"]
        return dict(kind=k, scene=s, seed=seed % (1 << 31),
                    pixels=rng.integers(0, case["width"] * case["height"], n).astype(np.int32),
                    samples=rng.integers(0, 64, n).astype(np.int32))
    if k == "rays":
        s = R.Scene(ctx, _icosphere(case["level"], 64, 64, 4, seed))
        return dict(kind=k, scene=s, rays=_rays(case["rays"], np.random.default_rng(seed)))
    if k == "preview":
        data = _icosphere(case["level"], case["width"], case["height"], case["depth"], seed)
        s = R.Scene(ctx, data)
        v = data.vertices
        moved = v + np.float32(0.03) * np.sin(np.float32(3.0) * v[:, ::-1])
        film = torch.zeros((case["height"], case["width"], 4), device="cuda")
        st = dict(kind=k, scene=s, vertices=torch.from_numpy(np.ascontiguousarray(moved, np.float32)).cuda(), film=film, spp=case["spp"],
                  seed=seed % (1 << 31))
        torch.cuda.synchronize()
        return st
    if k == "frame":
        data = _scene(case["scene"], case["width"], case["height"], case["depth"], seed, case.get("level"))
        if case["filter"] == "gauss":
            data.camera["filter"] = D.gaussian_filter(2.0, 2.0)
        elif case["filter"] == "mitchell":
            data.camera["filter"] = D.mitchell_filter(1.5, 1.5)
        s = R.Scene(ctx, data)
        shape = (case["height"], case["width"], 4)
        film = np.zeros(shape, np.float32) if case["host"] else torch.zeros(shape, device="cuda")
        torch.cuda.synchronize()
        return dict(kind=k, scene=s, film=film, host=case["host"], spp=case["spp"], seed=seed % (1 << 31))
    env, _ = S.sky_env(1024, 512, sun_azim_deg=20.0 + 37.0 * (seed % 8))
    if k == "batch":
        jobs, films = [], []
        for j, m in enumerate(_mix(case)):
            s = R.Scene(ctx, _icosphere(m["level"], m["res"], m["res"], 12, seed + 31 * j, env=env))
            jobs.append((s, m["spp"], dict(seed=(seed + j) % (1 << 31))))
            films.append(torch.zeros((m["res"], m["res"], 4), device="cuda"))
        torch.cuda.synchronize()
        return dict(kind=k, ctx=ctx, jobs=jobs, films=films)
    jobs = []
    for j, m in enumerate(_mix(case)):
        if m["volume"]:
            data = S.volume_grid(128, 128, res=32, seed=(seed + 31 * j) % 100003, max_depth=64)
        else:
            res = min(m["res"], 256)
            data = _icosphere(m["level"], res, res, 12, seed + 31 * j, env=env)
        jobs.append((R.Scene(ctx, data), m["spp"], (seed + j) % (1 << 31)))
    return dict(kind=k, jobs=jobs, server=R.Server(ctx, lanes=2, rmse_display=True))


def run(state):
    k = state["kind"]
    if k == "li":
        return state["scene"].render_paths(state["pixels"], state["samples"], seed=state["seed"])
    if k == "rays":
        h = state["scene"].trace(state["rays"])
        o = state["scene"].trace(state["rays"], anyhit=True)
        return dict(t=h["t"], u=h["u"], v=h["v"], prim=h["prim"], occluded=o["prim"])
    if k == "preview":
        state["scene"].refit(state["vertices"])
        state["scene"].render(state["spp"], seed=state["seed"], film=state["film"].data_ptr())
        return state["film"]
    if k == "frame":
        if state["host"]:
            return state["scene"].render(state["spp"], seed=state["seed"], out=state["film"])
        state["scene"].render(state["spp"], seed=state["seed"], film=state["film"].data_ptr())
        return state["film"]
    if k == "batch":
        state["ctx"].batch_render(state["jobs"], device_films=[f.data_ptr() for f in state["films"]])
        return state["films"]
    srv = state["server"]
    ids = [srv.submit(s, spp, target_rmse=0.05, seed=seed) for s, spp, seed in state["jobs"]]
    return [srv.wait(i)[1] for i in ids]


# ------------------------------------------------------------------ work
def _triangles(scene, level):
    return dict(cornell=36, smooth=40, textured=36, delta=36, volume=24).get(scene) or 20 * 4 ** level + 2


def _render_work(tris, pixels, samples, scene, film_bytes=16, extra=0):
    """A frame reads its scene once and writes its film once; every sample
    traces at least its camera ray and, where that hits, one shadow ray: two
    descents of the tree (a box test of 18 operations per level) and a
    triangle test of 50 each, and the sample's shading, about 400."""
    env = 1024 * 512 * 12 if scene == "icosphere" else 0
    depth = math.log2(max(2, tris))
    return dict(bytes=tris * 36 + env + extra + pixels * film_bytes,
                flops=samples * (2 * (2 * depth * 18 + 50) + 400))


def _add(a, b):
    return {k: a[k] + b[k] for k in a}


def work(case):
    k = case["kind"]
    if k == "rays":
        tris = _triangles("icosphere", case["level"])
        n = case["rays"]
        return dict(bytes=2 * n * (32 + 16) + tris * 36, flops=2 * n * (2 * math.log2(tris) * 18 + 50))
    if k == "li":
        n = case["paths"]
        return _render_work(_triangles(case["scene"], None), n, n, case["scene"], film_bytes=20)
    if k == "preview":
        tris = _triangles("icosphere", case["level"])
        pix = case["width"] * case["height"]
        return _render_work(tris, pix, pix * case["spp"], "icosphere", extra=tris * 6)
    if k == "frame":
        lv = case.get("level")
        pix = case["width"] * case["height"]
        grid = 4 * lv ** 3 if case["scene"] == "volume" else 0
        return _render_work(_triangles(case["scene"], lv), pix, pix * case["spp"], case["scene"], extra=grid)
    total = dict(bytes=0, flops=0)
    for m in _mix(case):
        if k == "serve" and m["volume"]:
            total = _add(total, _render_work(24, 128 * 128, 128 * 128 * 8, "volume", extra=4 * 32 ** 3))
            continue
        res = min(m["res"], 256) if k == "serve" else m["res"]
        spp = min(m["spp"], 8) if k == "serve" else m["spp"]   # a served job may stop at its target
        total = _add(total, _render_work(_triangles("icosphere", m["level"]), res * res, res * res * spp, "icosphere"))
    return total


# ------------------------------------------------------------------ 64-bit results
def exact(case, seed):
    """Ray casts: every ray against every triangle, in 64 bits.  A path-traced
    film has no such value: a path whose branch is decided by the last bit of
    a distance or of a density goes elsewhere in another precision, so a
    64-bit film is a film of other paths."""
    if case["kind"] != "rays" or case["rays"] * 4 ** case["level"] > 2e9:
        return None
    data = _icosphere(case["level"], 64, 64, 4, seed)
    rays = _rays(case["rays"], np.random.default_rng(seed))
    tri = torch.from_numpy(data.vertices.astype(np.float64)[data.indices]).cuda()
    p0, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    n = torch.linalg.cross(e1, e2)
    o = torch.from_numpy(rays["o"].astype(np.float64)).cuda()
    d = torch.from_numpy(rays["d"].astype(np.float64)).cuda()
    mint = 1e-4 * torch.clamp(o.abs().amax(1), min=1.0)
    best_t = torch.full((len(o),), float("inf"), dtype=torch.float64, device="cuda")
    best_u, best_v = torch.zeros_like(best_t), torch.zeros_like(best_t)
    step = max(1, int(4e7) // len(tri))
    m1, m2 = torch.linalg.cross(e2, p0), torch.linalg.cross(p0, e1)
    for a in range(0, len(o), step):
        oo, dd = o[a:a + step], d[a:a + step]
        mo = torch.linalg.cross(oo, dd)
        # det = -d.n; with s = o - p0: t det = s.n, u det = d.(e2 x s), v det = d.(s x e1)
        det = -(dd @ n.T)
        t = (oo @ n.T - (p0 * n).sum(1)) / det
        u = (mo @ e2.T - dd @ m1.T) / det
        v = (-(mo @ e1.T) - dd @ m2.T) / det
        ok = (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= mint[a:a + step, None]) & (t <= 1e4) & (det.abs() > 1e-8)
        t = torch.where(ok, t, torch.inf)
        tb, k = t.min(1)
        best_t[a:a + step] = tb
        best_u[a:a + step] = u.gather(1, k[:, None])[:, 0]
        best_v[a:a + step] = v.gather(1, k[:, None])[:, 0]
    miss = torch.isinf(best_t)
    zero = torch.zeros_like(best_t)
    out = [torch.where(miss, zero, x).cpu().numpy() for x in (best_t, best_u, best_v)]
    return dict(t=out[0], u=out[1], v=out[2], prim=None, occluded=None)
