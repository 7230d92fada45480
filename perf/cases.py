"""Performance cases of the path-tracing core, run through the Python API (``petrichor_gb300.capi``).

A case is a dict of plain values; ``kind`` picks the entry point:

* ``frame``   one image of a resident scene: ``Context.render`` (film in host memory) where
              ``host`` is set, else ``Context.render_device``;
* ``batch``   several images of several resident scenes in one ``Context.batch_render``;
* ``serve``   a burst of requests through the resident serving loop (``Context.serve_*``);
* ``rays``    closest hits of caller rays (``Context.trace_closest``);
* ``replay``  one image with the reference renderer's own random streams (bit parity mode);
* ``aov``     one denoiser guide (or uv) pass with the reference's streams
              (``Context.render_aov_device``);
* ``denoise`` the image filter on device buffers (``Context.denoise_device``);
* ``dropin``  ``capi.render_scene``: upload, BVH build, render, film copy and release in one
              call, as the reference's ``Petrichor::Render(scene)`` works.

Scenes, skies and requests come from ``petrichor_gb300.synth`` with the given seed: the
benchmark's own generators at its sizes, or below them where making the input would take
longer than the work (the 20M-triangle terrain and the 4M-triangle serving scene are cut to
about 2M and 1M triangles; the batch of 64 scenes to 8).
"""
import math

import torch

from petrichor_gb300 import capi, synth
from petrichor_gb300.scene_io import INTEGRATOR_PT, INTEGRATOR_SIMPLE


def listed():
    return [
        # a viewport preview: one sample per pixel of a light scene, film back on the host.
        # The smallest call: launches and host latency count.
        dict(name="preview_128x72_1spp", kind="frame", scene="spheres", tris=20_000, width=128, height=72, spp=1,
             bounces=8, env=512, host=True),
        # the reference's own small scene and default integrator (Russian roulette, no depth
        # limit), film on the host
        dict(name="cornell_256_16spp", kind="frame", scene="cornell_simple", tris=36, width=256, height=256, spp=16,
             bounces=3, env=0, host=True),
        # an interior with an area light, a thin lens and every material kind: bounded shadow
        # rays, no common ray origin; odd image size
        dict(name="interior_lens_803x601", kind="frame", scene="cornell_lens", tris=36, width=803, height=601,
             spp=16, bounces=8, env=0, host=False),
        # the flagship still: the benchmark's 1.0M-triangle workload
        dict(name="still_1080p_64spp", kind="frame", scene="spheres", tris=1_000_000, width=1920, height=1080,
             spp=64, bounces=16, env=2048, host=False),
        # terrain in 4K: the benchmark's memory-bound scene, fewer samples, every bounce traced
        dict(name="terrain_4k_4spp", kind="frame", scene="terrain", tris=2_400_000, width=3840, height=2160, spp=4,
             bounces=12, env=2048, host=False),
        # a batch of uneven images (the benchmark's ranges)
        dict(name="batch_8_uneven", kind="batch", mix=3, count=8, tris_lo=10_000, tris_hi=500_000, side_lo=256,
             side_hi=1024, bounces=16, env=512),
        # a burst of render requests on textured resident scenes (the benchmark's stream)
        dict(name="serve_24_requests", kind="serve", mix=5, count=24, scenes=3, tris_lo=100_000, tris_hi=1_000_000,
             side_lo=128, side_hi=1024, env=1024, maps=512),
        # ray queries of another program (visibility, picking, baking): incoherent rays
        dict(name="rays_4m", kind="rays", tris=300_000, rays=4_000_000),
        # the parity mode: the reference's stream, one per 16x16 tile
        dict(name="replay_cornell_256", kind="replay", scene="cornell_mixed", tris=36, width=256, height=256, spp=2,
             bounces=5, env=0),
        # the denoiser's albedo guide of a still
        dict(name="aov_albedo_960x540", kind="aov", aov=capi.AOV_DENOISING_ALBEDO, tris=200_000, width=960,
             height=540, spp=4, bounces=16, env=512),
        # the denoiser on a noisy 1080p HDR film with both guides
        dict(name="denoise_1080p_hdr", kind="denoise", width=1920, height=1080, hdr=True, albedo=True, normal=True),
        # the whole drop-in call on a mid-size scene: build and upload weigh as much as the render
        dict(name="dropin_400k_640x360", kind="dropin", tris=400_000, width=640, height=360, spp=16, bounces=16,
             env=1024),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "frame", "batch", "serve", "rays", "rays", "replay", "aov",
                       "denoise", "denoise", "dropin"])
    env = rng.choice([256, 500, 512, 1024])  # equirect width; 500: not a power of two
    if kind == "frame":
        scene = rng.choice(["spheres", "spheres", "terrain", "cornell_simple", "cornell_lens"])
        w, h = _log(rng, 65, 1920), _log(rng, 41, 1080)
        spp = max(1, min(_log(rng, 1, 64), 60_000_000 // (w * h)))
        return dict(kind="frame", scene=scene, width=w, height=h, spp=spp, env=env, host=rng.random() < 0.5,
                    tris=36 if scene.startswith("cornell") else _log(rng, 5_000, 1_000_000),
                    bounces=3 if scene == "cornell_simple" else rng.randint(2, 16))
    if kind == "batch":
        return dict(kind="batch", mix=rng.randrange(1000), count=rng.randint(2, 8), tris_lo=10_000,
                    tris_hi=_log(rng, 20_000, 300_000), side_lo=_log(rng, 96, 256), side_hi=_log(rng, 300, 900),
                    bounces=rng.randint(4, 16), env=env)
    if kind == "serve":
        return dict(kind="serve", mix=rng.randrange(1000), count=rng.randint(3, 24), scenes=rng.randint(1, 3),
                    tris_lo=50_000, tris_hi=_log(rng, 60_000, 500_000), side_lo=64, side_hi=_log(rng, 128, 900),
                    env=env, maps=_log(rng, 33, 512))
    if kind == "rays":
        return dict(kind="rays", tris=_log(rng, 1_000, 500_000), rays=_log(rng, 1_000, 4_000_000))
    if kind == "replay":
        return dict(kind="replay", scene=rng.choice(["cornell_mixed", "cornell_lens"]), tris=36,
                    width=_log(rng, 40, 256), height=_log(rng, 40, 256), spp=rng.randint(1, 2),
                    bounces=rng.randint(2, 5), env=0)
    if kind == "aov":
        return dict(kind="aov", aov=rng.choice([capi.AOV_UV, capi.AOV_DENOISING_ALBEDO, capi.AOV_DENOISING_NORMAL]),
                    tris=_log(rng, 5_000, 200_000), width=_log(rng, 97, 960), height=_log(rng, 61, 540),
                    spp=rng.randint(1, 4), bounces=rng.randint(2, 16), env=env)
    if kind == "denoise":
        albedo = rng.random() < 0.7
        return dict(kind="denoise", width=_log(rng, 33, 1920), height=_log(rng, 33, 1080), hdr=rng.random() < 0.7,
                    albedo=albedo, normal=albedo and rng.random() < 0.8)
    return dict(kind="dropin", tris=_log(rng, 10_000, 400_000), width=_log(rng, 97, 640),
                height=_log(rng, 61, 360), spp=_log(rng, 1, 16), bounces=rng.randint(4, 16), env=env)


# ---------------------------------------------------------------- inputs
def _scene(case, seed):
    w, h, spp, b = case["width"], case["height"], case["spp"], case["bounces"]
    env = case["env"]
    kind = case.get("scene", "spheres")
    if kind == "cornell_simple":
        return synth.cornell(seed=seed, width=w, height=h, spp=spp, max_bounces=b, integrator=INTEGRATOR_SIMPLE)
    if kind == "cornell_mixed":
        return synth.cornell(seed=seed, width=w, height=h, spp=spp, max_bounces=b, integrator=INTEGRATOR_PT,
                             mixed=True, env_texture=True)
    if kind == "cornell_lens":
        return synth.cornell(seed=seed, width=w, height=h, spp=spp, max_bounces=b, integrator=INTEGRATOR_PT,
                             mixed=True, aperture=0.1)
    if kind == "terrain":
        rocks = max(4, min(1000, case["tris"] // 5000))
        n = max(16, int(math.sqrt(0.5 * max(2_000, case["tris"] - 400 * rocks))))
        return synth.terrain_rocks(seed=seed, terrain_n=n, n_rocks=rocks, rock_tris=400, width=w, height=h, spp=spp,
                                   max_bounces=b, env_width=env, env_height=env // 2)
    return synth.spheres_grids(seed=seed, tri_budget=case["tris"], width=w, height=h, spp=spp, max_bounces=b,
                               env_width=env, env_height=env // 2)


def _film(width, height):
    return torch.zeros(height, width, 3, dtype=torch.float32, device="cuda")


def _host_film(width, height):
    return torch.zeros(height, width, 3, dtype=torch.float32, pin_memory=True).numpy()


# The sizes of a batch and the requests of a burst are the case's (drawn from its ``mix``),
# the scenes and random streams the seed's.
def _batch_params(case):
    return synth.batch_instance_params(case["mix"], case["count"], tri_lo=case["tris_lo"], tri_hi=case["tris_hi"],
                                       px_lo=case["side_lo"] ** 2, px_hi=case["side_hi"] ** 2, spps=(4, 16))


def _requests(case):
    return synth.request_stream(case["mix"], 500.0, case["count"], n_scenes=case["scenes"], px_lo=case["side_lo"] ** 2,
                                px_hi=case["side_hi"] ** 2, spps=(1, 8, 32))


def _denoise_images(case, seed):
    """A noisy film and its guides: smooth regions with albedo and normal edges, and
    multiplicative noise with a heavy tail (a few fireflies), as few samples leave it."""
    w, h = case["width"], case["height"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    y = torch.linspace(0, 1, h, device="cuda")[:, None]
    x = torch.linspace(0, 1, w, device="cuda")[None, :]
    cells = torch.rand(16, 16, 3, device="cuda", generator=g) * 0.8 + 0.05
    cy = (y * 15.999).long().expand(h, w)
    cx = (x * 15.999).long().expand(h, w)
    albedo = cells[cy, cx]
    facets = torch.randn(16, 16, 3, device="cuda", generator=g)
    facets = facets / facets.norm(dim=-1, keepdim=True)
    normal = facets[cx, cy]
    light = 0.4 + torch.sin(7 * x + 3 * y).abs() + 0.5 * torch.cos(5 * y - 2 * x).abs()
    noise = torch.exp(0.8 * torch.randn(h, w, 1, device="cuda", generator=g))
    spikes = (torch.rand(h, w, 1, device="cuda", generator=g) < 1e-3) * 50.0
    color = albedo * light[..., None] * (noise + spikes)
    return color.contiguous(), albedo.contiguous(), normal.contiguous()


def prepare(case, seed):
    kind = case["kind"]
    ctx = capi.Context(0)
    s = {"kind": kind, "ctx": ctx}
    if kind in ("frame", "replay", "aov"):
        sc = _scene(case, seed)
        s["sid"] = ctx.upload(sc)
        s["cam"] = capi.camera_from_scene(sc)
        mode = capi.MODE_REPLAY if kind == "replay" else capi.MODE_WAVEFRONT
        s["st"] = capi.settings_from_scene(sc, mode, seed & 0x7FFFFFFF, denoising_spp=case["spp"])
        s["host"] = bool(case.get("host"))
        s["film"] = (_host_film if s["host"] else _film)(case["width"], case["height"])
        s["aov"] = case.get("aov")
    elif kind == "batch":
        s["jobs"], s["films"] = [], []
        for k, (tris, w, h, spp) in enumerate(_batch_params(case)):
            sc = synth.spheres_grids(seed=seed + 17 * k, tri_budget=tris, width=w, height=h, spp=spp,
                                     max_bounces=case["bounces"], env_width=case["env"], env_height=case["env"] // 2)
            film = _film(w, h)
            s["films"].append(film)
            s["jobs"].append((ctx.upload(sc), capi.camera_from_scene(sc),
                              capi.settings_from_scene(sc, capi.MODE_WAVEFRONT, seed & 0x7FFFFFFF), film.data_ptr()))
    elif kind == "serve":
        scenes = synth.serving_scenes(seed=seed, n=case["scenes"], tri_lo=case["tris_lo"], tri_hi=case["tris_hi"],
                                      env_width=case["env"], env_height=case["env"] // 2, map_size=case["maps"])
        ids = [ctx.upload(sc) for sc in scenes]
        cams = [capi.camera_from_scene(sc) for sc in scenes]
        s["reqs"] = []
        for k, (_, i, w, h, spp, depth) in enumerate(_requests(case)):
            st = capi.settings_from_scene(scenes[i], capi.MODE_WAVEFRONT, (seed + k) & 0x7FFFFFFF, width=w, height=h,
                                          spp=spp, max_bounces=depth)
            s["reqs"].append((ids[i], cams[i], st, _host_film(w, h)))
        ctx.serve_start()
    elif kind == "rays":
        sc = synth.spheres_grids(seed=seed, tri_budget=case["tris"], env_width=64, env_height=32)
        s["sid"] = ctx.upload(sc)
        n = case["rays"]
        g = torch.Generator(device="cuda").manual_seed(seed)
        lo = torch.tensor(sc.positions.min(0), device="cuda")
        hi = torch.tensor(sc.positions.max(0), device="cuda")
        org = lo + (hi - lo) * torch.rand(n, 3, device="cuda", generator=g)
        d = torch.randn(n, 3, device="cuda", generator=g)
        s["rays"] = torch.cat([org, d / d.norm(dim=1, keepdim=True)], 1).contiguous()
        s["n"] = n
        s["tri"] = torch.zeros(n, dtype=torch.int32, device="cuda")
        s["dist"] = torch.zeros(n, dtype=torch.float32, device="cuda")
    elif kind == "denoise":
        c, a, nrm = _denoise_images(case, seed)
        s["images"] = (c, a if case["albedo"] else None, nrm if case["normal"] else None)
        s["hdr"] = bool(case["hdr"])
        s["out"] = torch.zeros_like(c)
    else:
        s["scene"] = _scene(case, seed)
        s["seed"] = seed & 0x7FFFFFFF
    torch.cuda.synchronize()  # the inputs are made on torch's stream, the context has its own
    return s


# ---------------------------------------------------------------- one pass
def run(s):
    kind, ctx = s["kind"], s["ctx"]
    if kind == "frame":
        if s["host"]:
            return ctx.render(s["sid"], s["cam"], s["st"], s["film"])
        ctx.render_device(s["sid"], s["cam"], s["st"], s["film"].data_ptr())
        return s["film"]
    if kind == "replay":
        ctx.render_device(s["sid"], s["cam"], s["st"], s["film"].data_ptr())
        return s["film"]
    if kind == "aov":
        ctx.render_aov_device(s["sid"], s["cam"], s["st"], s["aov"], s["film"].data_ptr())
        return s["film"]
    if kind == "batch":
        ctx.batch_render(s["jobs"])
        return s["films"]
    if kind == "serve":
        ids = [ctx.serve_submit(sid, cam, st, film_host=film) for sid, cam, st, film in s["reqs"]]
        states = [ctx.serve_wait(r, 60.0).state for r in ids]
        for r in ids:
            ctx.serve_release(r)
        return {"states": states, "films": [q[3] for q in s["reqs"]]}
    if kind == "rays":
        ctx.trace_closest(s["sid"], s["n"], s["rays"].data_ptr(), 0.0, 1e30, s["tri"].data_ptr(),
                          s["dist"].data_ptr())
        return {"tri": s["tri"], "dist": s["dist"]}
    if kind == "denoise":
        c, a, n = s["images"]
        ctx.denoise_device(c.shape[1], c.shape[0], c.data_ptr(), a.data_ptr() if a is not None else 0,
                           n.data_ptr() if n is not None else 0, s["hdr"], s["out"].data_ptr())
        return s["out"]
    return capi.render_scene(s["scene"], capi.MODE_WAVEFRONT, seed=s["seed"], ctx=ctx)


# ---------------------------------------------------------------- what a pass cannot do without
# Per closest-hit or visibility query in a tree of T triangles: one box test for each of two
# children on each of log2(T) levels (25 operations a box), four triangle tests of 45.
# Shading a hit (BSDF, next event, sky lookup): about 400. A sample is one camera query, and
# on these scenes about 0.5 further bounces with as many visibility rays outside, about 3 of
# each in a closed box.
def _query_flops(tris):
    return 2.0 * 25.0 * math.log2(max(2, tris)) + 4 * 45.0


def _image_work(tris, width, height, spp, env, closed=False):
    """(bytes, flops): triangles (vertices, normals, indices) and sky read once, film written."""
    n = float(width) * height * spp
    bounces = 3.0 if closed else 0.5
    flops = n * ((1 + 2 * bounces) * _query_flops(tris) + (1 + bounces) * 400.0)
    return tris * 60.0 + env * (env // 2) * 12.0 + width * height * 12.0, flops


def work(case):
    kind = case["kind"]
    b = f = 0.0
    if kind in ("frame", "replay", "dropin", "aov"):
        b, f = _image_work(case["tris"], case["width"], case["height"], case["spp"], case["env"],
                           case.get("scene", "").startswith("cornell"))
        if kind == "aov":  # the camera query and its shading point
            f = float(case["width"]) * case["height"] * case["spp"] * (_query_flops(case["tris"]) + 100.0)
        if kind == "dropin":  # the build: every level bins and sorts every triangle
            f += case["tris"] * math.log2(case["tris"]) * 40.0
    elif kind == "batch":
        for tris, w, h, spp in _batch_params(case):
            x, y = _image_work(tris, w, h, spp, case["env"])
            b, f = b + x, f + y
    elif kind == "serve":
        for _, i, w, h, spp, _depth in _requests(case):
            t = case["tris_lo"] * (case["tris_hi"] / case["tris_lo"]) ** (i / max(1, case["scenes"] - 1))
            x, y = _image_work(t, w, h, spp, 0)
            b, f = b + x - 60.0 * t, f + y
        b += case["scenes"] * (case["env"] * (case["env"] // 2) * 12.0 + 3 * case["maps"] ** 2 * 12.0)
    elif kind == "rays":
        b, f = case["rays"] * (24.0 + 8.0) + case["tris"] * 36.0, case["rays"] * _query_flops(case["tris"])
    elif kind == "denoise":
        px = float(case["width"]) * case["height"]
        guides = int(case["albedo"]) + int(case["normal"])
        b, f = px * 12.0 * (2 + guides), px * 5 * 25 * (20.0 + 10.0 * guides)
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------- 64-bit values
def exact(case, seed):
    """The denoiser's output in 64 bits. The other outputs are sums over random paths (or
    closest hits over whole scenes), whose every branch depends on single-precision
    comparisons: they have no 64-bit value, and equal their earlier films instead."""
    if case["kind"] != "denoise":
        return None
    c, a, n = _denoise_images(case, seed)
    return _denoise64(c.double(), a.double() if case["albedo"] else None, n.double() if case["normal"] else None,
                      bool(case["hdr"]))


def _lum(c):
    return 0.2126 * c[..., 0] + 0.7152 * c[..., 1] + 0.0722 * c[..., 2]


def _denoise64(c, albedo, normal, hdr):
    """Edge-avoiding a-trous wavelet filter (Dammertz et al., HPG 2010) with a variance-scaled
    luminance stop carried through the passes (Schied et al., HPG 2017)."""
    H, W = c.shape[:2]
    yy, xx = torch.arange(H, device=c.device), torch.arange(W, device=c.device)

    def shift(t, dy, dx):  # clamped edges
        return t[(yy + dy).clamp(0, H - 1)][:, (xx + dx).clamp(0, W - 1)]

    def edge(t):
        y = _lum(t).clamp(min=0)
        return torch.log1p(y) if hdr else y.clamp(max=1)

    factor = torch.ones_like(c)
    if albedo is not None:
        lit = (_lum(albedo) > 0.01)[..., None]
        factor = torch.where(lit, albedo.clamp(min=1e-3), factor)
    c = c / factor
    if normal is not None:
        l2 = (normal * normal).sum(-1, keepdim=True)
        known = (l2 > 0.25)[..., 0]
        normal = torch.where(l2 > 0.25, normal / l2.clamp(min=0.25).sqrt(), torch.zeros_like(normal))
    lum = edge(c)
    near = [(dy, dx) for dy in (-1, 0, 1) for dx in (-1, 0, 1)]
    m1 = sum(shift(lum, *d) for d in near) / 9
    m2 = sum(shift(lum * lum, *d) for d in near) / 9
    var = (m2 - m1 * m1).clamp(min=0)
    kernel = [1 / 16, 1 / 4, 3 / 8, 1 / 4, 1 / 16]
    sigma = 4.0 if (albedo is not None or normal is not None) else 2.0
    for k in range(5):
        scale = 1.0 / (sigma * (sum(shift(var, *d) for d in near) / 9).sqrt() + 1e-4)
        sc, sw, sv = torch.zeros_like(c), torch.zeros_like(lum), torch.zeros_like(lum)
        for i in range(5):
            for j in range(5):
                dy, dx = (i - 2) << k, (j - 2) << k
                w = torch.ones_like(lum)
                if i != 2 or j != 2:
                    w = torch.exp(-(lum - shift(lum, dy, dx)).abs() * scale)
                    if normal is not None:
                        dot = (normal * shift(normal, dy, dx)).sum(-1).clamp(min=0)
                        w = torch.where(known & shift(known, dy, dx), w * dot ** 128, w)
                    if albedo is not None:
                        da = factor - shift(factor, dy, dx)
                        w = w * torch.exp(-(da * da).sum(-1) * 100.0)
                w = w * (kernel[i] * kernel[j])
                sc += w[..., None] * shift(c, dy, dx)
                sw += w
                sv += w * w * shift(var, dy, dx)
        c = sc / sw[..., None]
        var = sv / (sw * sw)
        lum = edge(c)
    return c * factor
