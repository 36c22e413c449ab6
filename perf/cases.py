"""The calls this renderer is used for, with the sizes they are used at.

Every case is one call sequence a program makes through the public interface
(`aperturerendererv3_gb300.scene.SceneRenderer`, `torch_render.render_textures`):
progressive frames, headless renders, guided renders, the differentiable step,
raw ray queries, mesh refits and rebuilds, and the denoiser.  `prepare` builds
the scene (what a program keeps between calls), `run` makes the calls.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from aperturerendererv3_gb300 import SceneRenderer, TriangleMesh, configs
from aperturerendererv3_gb300._lib import DENOISE_GBUF_DTYPE, DENOISE_STAT_DTYPE
from aperturerendererv3_gb300.torch_render import render_textures

DEV = "cuda"

# the denoiser's weights of a squared difference, 1 / (2 sigma^2)
SIGMA = {"albedo": 0.5, "normal": 2.0, "depth": 8.0, "metallic": 2.0, "rough": 2.0, "model": 50.0, "spatial": 0.125}

# closest-hit and shadow rays one sample of each scene casts, about: what the estimate in work() counts
RAYS_PER_SAMPLE = {"cornell": 6.0, "reference": 6.0, "glass": 5.0, "terrain": 2.0, "combined": 4.0, "textured": 6.0}


def listed():
    return [
        # an interactive viewport: one progressive frame per call, where latency and launches count
        {"name": "frame_256", "kind": "frame", "scene": "cornell", "width": 256, "height": 256, "depth": 8,
         "denoise": False},
        # a preview written to a file: a small headless render to host memory and its display image
        {"name": "file_256x16", "kind": "file", "scene": "cornell", "width": 256, "height": 256, "spp": 16, "depth": 8},
        # glass, dispersion and absorption at the default depth limit, an odd image size
        {"name": "glass_413x307x8", "kind": "render", "scene": "glass", "width": 413, "height": 307, "spp": 8,
         "depth": 1000, "res": 0},
        # the headline workload: a large heightfield, GGX, many lights and the sky
        {"name": "terrain_1080p", "kind": "render", "scene": "terrain", "width": 1920, "height": 1080, "spp": 32,
         "depth": 16, "res": 2048},
        # terrain, smooth-union SDF and a participating medium together
        {"name": "combined_640x360", "kind": "render", "scene": "combined", "width": 640, "height": 360, "spp": 4,
         "depth": 24, "res": 512},
        # a guided render that resumes from saved probes: one update window sampled from them, then learning
        {"name": "guided_480x270", "kind": "guided", "scene": "reference", "width": 480, "height": 270, "spp": 16,
         "depth": 16},
        # a step of texture fitting: forward, L2 loss, replay adjoint
        {"name": "texture_step_256", "kind": "texture", "width": 256, "height": 256, "spp": 64, "depth": 8, "res": 512},
        # a large batch of ray queries against random triangles: camera rays and incoherent ones
        {"name": "rays_1m_tris", "kind": "rays", "scene": "triangles", "tris": 1000000, "rays": 2073600, "any": False},
        # a picking or visibility query: few rays, a small scene
        {"name": "rays_few", "kind": "rays", "scene": "triangles", "tris": 5000, "rays": 1000, "any": True},
        # an animation frame: the mesh moves, the tree is refit, rays are cast
        {"name": "refit_513", "kind": "refit", "grid": 513, "rays": 65536},
        # an edit that changes the mesh: rebuilt on the GPU, rays are cast
        {"name": "rebuild_200k", "kind": "rebuild", "tris": 200000, "rays": 65536},
        # the denoiser on an image of display size
        {"name": "denoise_1080p", "kind": "denoise", "width": 1920, "height": 1080, "spp": 8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "file", "render", "render", "guided", "texture", "rays", "rays", "refit", "rebuild",
                       "denoise"])
    w = _log(rng, 48, 1920)
    h = max(16, min(1080, int(w * rng.uniform(0.5, 1.1))))
    if kind == "frame":
        return {"kind": kind, "scene": rng.choice(["cornell", "reference", "glass"]), "width": w, "height": h,
                "depth": rng.randint(2, 24), "denoise": rng.random() < 0.5}
    if kind == "file":
        return {"kind": kind, "scene": rng.choice(["cornell", "reference"]), "width": w, "height": h,
                "spp": max(1, min(64, _log(rng, 1, 64) * 16384 // (w * h) + 1)), "depth": rng.randint(2, 16)}
    if kind == "render":
        scene = rng.choice(["cornell", "reference", "glass", "terrain", "combined"])
        most = 230400 * 4 if scene == "combined" else 1920 * 1080 * 4
        return {"kind": kind, "scene": scene, "width": w, "height": h,
                "spp": max(1, min(_log(rng, 1, 64), most // (w * h))), "depth": rng.choice([2, 5, 8, 16, 24, 1000]),
                "res": rng.choice([65, 128, 257, 512]) if scene in ("terrain", "combined") else 0}
    if kind == "guided":
        w, h = min(w, 640), min(h, 360)
        return {"kind": kind, "scene": rng.choice(["cornell", "reference"]), "width": w, "height": h,
                "spp": rng.randint(1, 16), "depth": rng.randint(4, 16)}
    if kind == "texture":
        w, h = _log(rng, 32, 320), _log(rng, 32, 320)
        return {"kind": kind, "width": w, "height": h, "spp": rng.choice([4, 9, 16, 40]), "depth": rng.randint(2, 12),
                "res": rng.choice([31, 64, 256, 512])}
    if kind == "rays":
        return {"kind": kind, "scene": "triangles", "tris": _log(rng, 1000, 500000), "rays": _log(rng, 100, 2000000),
                "any": rng.random() < 0.5}
    if kind == "refit":
        return {"kind": kind, "grid": _log(rng, 17, 600), "rays": _log(rng, 256, 65536)}
    if kind == "rebuild":
        return {"kind": kind, "tris": _log(rng, 500, 200000), "rays": _log(rng, 256, 65536)}
    return {"kind": kind, "width": w, "height": h, "spp": rng.randint(2, 64)}


# ------------------------------------------------------------------ scenes
@functools.lru_cache(maxsize=3)
def _terrain_base(res):
    """The benchmark's terrain, read once like a mesh file; each seed stretches its heights."""
    return configs.terrain_scene(res=res)


def _renderer(scene, seed, res=0):
    """(renderer, camera, render keywords) of a named scene."""
    rng = np.random.default_rng(seed)
    kw = {"seed": int(rng.integers(1, 1 << 62))}
    if scene in ("terrain", "combined"):
        objs, base = _terrain_base(res)
        v = base.vertices.copy()
        v[:, 1] *= np.float32(rng.uniform(0.9, 1.1))
        mesh = TriangleMesh(v, base.indices, base.material_ids, base.materials)
        if scene == "terrain":
            cam, r = dict(configs.TERRAIN_CAMERA), SceneRenderer(objs, mesh=mesh)
        else:
            cam = dict(configs.COMBINED_CAMERA)
            r = SceneRenderer(objs, mesh=mesh, sdf=configs.sdf_blobs(), medium=configs.COMBINED_MEDIUM)
    elif scene == "cornell":
        cam, r = dict(configs.CORNELL_CAMERA), SceneRenderer(configs.cornell_triangles())
    elif scene == "reference":
        cam, r = dict(configs.REFERENCE_CORNELL_CAMERA), SceneRenderer(configs.reference_cornell())
    else:
        cam, r = dict(configs.GLASS_TEST_CAMERA), SceneRenderer(configs.glass_test_scene())
    o = cam["origin"]
    cam["origin"] = (o[0] + float(rng.uniform(-0.02, 0.02)), o[1] + float(rng.uniform(-0.02, 0.02)), o[2])
    r.build()
    return r, cam, kw


def _rays(n, seed, lo, hi, any_hit):
    """n rays (o, tmin, d, tmax): the first half through a camera's pixels, the rest from inside the box [lo, hi]
    in random directions; visibility queries end at a limit."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    lo, hi = torch.tensor(lo, device=DEV), torch.tensor(hi, device=DEV)
    k = n // 2
    side = max(1, math.isqrt(max(1, k)))
    i = torch.arange(k, device=DEV)
    px, py = ((i % side) + 0.5) / side, ((i // side) + 0.5) / max(1, -(-k // side))
    eye = 0.5 * (lo + hi) + (hi - lo).max() * torch.tensor([0.0, 0.35, 1.3], device=DEV)
    at = lo + (hi - lo) * torch.stack([px, 1.0 - py, torch.full_like(px, 0.5)], 1)
    o = torch.cat([eye.expand(k, 3), lo + (hi - lo) * torch.rand(n - k, 3, generator=g, device=DEV)])
    d = torch.cat([at - eye, torch.randn(n - k, 3, generator=g, device=DEV)])
    d = d / d.norm(dim=1, keepdim=True)
    rays = torch.empty(n, 8, device=DEV)
    rays[:, 0:3], rays[:, 4:7] = o, d
    rays[:, 3] = 0.0
    rays[:, 7] = 0.5 if any_hit else math.inf
    return rays


def _triangle_mesh(n, seed):
    v = configs.random_triangles(n, seed=seed)
    mats = [configs.Material.CreateDiffusePureColor(configs.GREY)]
    return TriangleMesh(v.reshape(-1, 3), np.arange(3 * n, dtype=np.uint32).reshape(-1, 3), np.zeros(n, np.int32), mats)


def _grid_mesh(m, seed):
    """An m x m vertex sheet over the unit square, and its triangles."""
    rng = np.random.default_rng(seed)
    x = np.linspace(0.0, 1.0, m)
    a, b, c, d = rng.uniform(2.0, 9.0, 4)
    y = 0.05 * (np.sin(a * x)[None, :] * np.cos(b * x)[:, None] + np.sin(c * x[None, :] + d * x[:, None]))
    v = np.stack([np.broadcast_to(x[None, :], (m, m)), y, np.broadcast_to(x[:, None], (m, m))], -1)
    j, i = np.mgrid[0:m - 1, 0:m - 1]
    p = (j * m + i).reshape(-1)
    idx = np.concatenate([np.stack([p, p + m, p + 1], 1), np.stack([p + 1, p + m, p + m + 1], 1)]).astype(np.uint32)
    mats = [configs.Material.CreateDiffusePureColor(configs.GREY)]
    return TriangleMesh(v.reshape(-1, 3).astype(np.float32), idx, np.zeros(len(idx), np.int32), mats)


def _moved(vertices, seed):
    """The sheet's vertices a moment later."""
    v = torch.as_tensor(vertices, device=DEV)
    phase = 0.1 + 0.01 * (seed % 97)
    out = v.clone()
    out[:, 1] += 0.02 * torch.sin(12.0 * v[:, 0] + phase) * torch.cos(7.0 * v[:, 2] - phase)
    return out


GUIDE_UNIT = 0.1


def _guide_probes(seed):
    """Probes as a guide has them after some frames: every voxel along the box's walls, every direction face, a few
    bright texels over a dim sphere; the coarser levels are the means of their children."""
    rng = np.random.default_rng(seed)
    x, y, z = np.mgrid[-5:5, -5:5, -5:5]
    wall = (np.minimum.reduce([x, y, z]) == -5) | (np.maximum.reduce([x, y, z]) == 4)
    vox = np.stack([x[wall], y[wall], z[wall]], 1)
    keys = np.concatenate([np.repeat(vox, 20, 0), np.tile(np.arange(20), len(vox))[:, None]], 1).astype(np.int32)
    n = len(keys)
    level = rng.gamma(0.3, 1.0, (n, 8, 8, 1)) * rng.uniform(0.2, 1.0, (n, 1, 1, 4)) + 1e-3
    levels = [level.reshape(n, 64, 4)]
    for res in (4, 2, 1):
        level = level.reshape(n, res, 2, res, 2, 4).mean((2, 4))
        levels.append(level.reshape(n, res * res, 4))
    texels = np.concatenate(levels + [np.zeros((n, 1, 4))], 1).astype(np.float32)
    return keys, texels, rng.integers(16, 4096, n).astype(np.uint64)


def _denoise_records(w, h, spp, seed):
    """A G-buffer and sample moments as a recorded render leaves them: a few flat surfaces, a sky strip without
    hits, noise that falls with the sample count."""
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:h, 0:w]
    region = ((x * 5) // max(1, w) + (y * 4) // max(1, h)) % 6
    g, s = np.zeros((h, w), DENOISE_GBUF_DTYPE), np.zeros((h, w), DENOISE_STAT_DTYPE)
    albedo = rng.uniform(0.1, 0.9, (6, 3))[region] + rng.normal(0.0, 0.01, (h, w, 3))
    normal = rng.normal(0.0, 1.0, (6, 3))[region] + rng.normal(0.0, 0.02, (h, w, 3))
    normal /= np.linalg.norm(normal, axis=-1, keepdims=True)
    hit = y >= h // 8
    half = np.zeros((h, w, 14))
    half[..., 0:3], half[..., 3:6] = albedo, normal
    half[..., 6], half[..., 7] = rng.choice([0.0, 1.0], 6)[region], rng.uniform(0.05, 1.0, 6)[region]
    half[..., 8 + 3] = 1.0
    half[~hit] = 0.0
    half[~hit, 8 + 4] = 1.0
    g["h"] = half.astype(np.float16).view(np.uint16)
    g["depth"] = np.where(hit, 1.0 + 0.5 * x / w + rng.normal(0.0, 1e-3, (h, w)), 0.0)
    g["valid"], g["frames"] = np.where(hit, spp, 0), spp
    level = rng.uniform(0.05, 2.0, (6, 1))[region] * np.array([0.95, 1.0, 1.05])
    sigma = 0.3 * level
    mean = 2.0 * (np.sqrt(level) - 1.0)
    s["num"] = spp
    s["mean"] = mean + rng.normal(0.0, 1.0, (h, w, 3)) * sigma / math.sqrt(spp)
    s["m2n"] = sigma ** 2 * rng.gamma(max(1.0, (spp - 1) / 2.0), 2.0 / max(1, spp - 1), (h, w, 3)) + 1e-6
    s["m3n"] = sigma ** 3 * rng.normal(0.0, 0.3, (h, w, 3))
    return g, s


# ------------------------------------------------------------------ state
def prepare(case, seed):
    k = case["kind"]
    st = {"case": dict(case)}
    if k in ("frame", "file", "render", "guided"):
        st["r"], st["cam"], st["kw"] = _renderer(case["scene"], seed, case.get("res", 0))
        shape = (case["height"], case["width"])
        if k == "frame":
            st["hdr"] = torch.zeros(*shape, 3, device=DEV)
            st["ldr"] = torch.zeros(*shape, dtype=torch.int32, device=DEV)
            st["frame"] = 0
        elif k == "guided":
            st["probes"] = _guide_probes(seed)
        elif k == "render":
            st["img"] = torch.empty(*shape, 3, dtype=torch.float64, device=DEV)
    elif k == "texture":
        a = configs.cornell_textures(case["res"], seed=seed)
        objs, mesh, tex = configs.textured_cornell(a)
        st["r"] = SceneRenderer(objs, mesh=mesh, textures=tex)
        st["r"].build()
        g = torch.Generator(device=DEV).manual_seed(seed)
        st["texels"] = torch.as_tensor(a, device=DEV).reshape(-1).requires_grad_()
        st["target"] = 0.2 * torch.rand(case["height"], case["width"], 3, generator=g, device=DEV, dtype=torch.float64)
    elif k == "rays":
        st["r"] = SceneRenderer([], mesh=_triangle_mesh(case["tris"], seed))
        st["r"].build()
        st["rays"] = _rays(case["rays"], seed, [0.0] * 3, [1.0] * 3, case["any"])
    elif k == "refit":
        mesh = _grid_mesh(case["grid"], seed)
        st["r"] = SceneRenderer([], mesh=mesh)
        st["r"].build()
        st["v"] = _moved(mesh.vertices, seed)
        st["rays"] = _rays(case["rays"], seed, [0.0, 0.0, 0.0], [1.0, 0.3, 1.0], False)
    elif k == "rebuild":
        st["r"] = SceneRenderer([], mesh=_triangle_mesh(case["tris"], seed))
        st["r"].set_build_mode("gpu")
        st["r"].build()
        st["mesh"] = _triangle_mesh(case["tris"], seed + 1000003)
        st["rays"] = _rays(case["rays"], seed, [0.0] * 3, [1.0] * 3, False)
    else:
        st["r"], _, _ = _renderer("cornell", seed)
        g, s = _denoise_records(case["width"], case["height"], case["spp"], seed)
        st["r"].set_denoise_records(g, s)
        x = np.maximum((1.0 + s["mean"] / 2.0), 0.0) ** 2
        st["xyz"] = torch.as_tensor(x.astype(np.float64), device=DEV)
        st["records"] = (g, s)
    return st


def run(st):
    c, r = st["case"], st["r"]
    k = c["kind"]
    if k in ("frame", "file", "render", "guided"):
        cam, kw = st["cam"], st["kw"]
        size = (c["width"], c["height"])
        common = dict(fov=cam["fov"], max_depth=c["depth"], **kw)
        if k == "frame":
            r.RenderFrame(st["hdr"], st["ldr"], size, cam["origin"], cam["direction"], st["frame"], 2,
                          denoise=c["denoise"], **common)
            st["frame"] += 1
            return {"hdr": st["hdr"], "ldr": st["ldr"]}
        if k == "file":
            img = r.Render(size, cam["origin"], cam["direction"], c["spp"], **common)
            return {"xyz": img, "rgba": r.tonemap(img)}
        if k == "render":
            r.render_into(st["img"], size, cam["origin"], cam["direction"], c["spp"], **common)
            return st["img"]
        r.set_guide_probes(*st["probes"], unit=GUIDE_UNIT)
        return r.Render(size, cam["origin"], cam["direction"], c["spp"], first_frame=64, guide=1,
                        guide_unit=GUIDE_UNIT, guide_frames=c["spp"], **common)
    if k == "texture":
        cam = configs.CORNELL_CAMERA
        st["texels"].grad = None
        img = render_textures(st["texels"], r, (c["width"], c["height"]), cam["origin"], cam["direction"], c["spp"],
                              fov=cam["fov"], max_depth=c["depth"])
        ((img - st["target"]) ** 2).sum().backward()
        return {"image": img.detach(), "grad": st["texels"].grad}
    if k == "refit":
        r.refit_mesh(st["v"])
    elif k == "rebuild":
        r.mesh = st["mesh"]
        r.MarkAsDirty()
        r.build()
    elif k == "denoise":
        return r.denoise(st["xyz"])
    if c.get("any"):
        return r.trace_any(st["rays"])
    ids, t = r.trace_closest(st["rays"])
    return {"ids": ids, "t": t}


# ------------------------------------------------------------------ work
def _scene_tris(case):
    res = case.get("res", 0)
    return {"terrain": 2 * res * res, "combined": 2 * res * res}.get(case.get("scene"), 40)


def work(case):
    """Bytes: scene and image once.  Flops: per ray about log2(triangles) box tests of 20 and three triangle tests
    of 50, per path vertex 400 of shading; per pixel pair of the denoiser 60."""
    k = case["kind"]
    if k in ("frame", "file", "render", "guided", "texture"):
        scene = case.get("scene", "textured")
        px = case["width"] * case["height"]
        tris = _scene_tris(case) if k != "texture" else 36
        rays = px * case.get("spp", 1) * RAYS_PER_SAMPLE[scene] * min(1.0, case["depth"] / 4.0)
        flops = rays * (20 * math.log2(tris) + 150 + 200)
        out = px * (16 if k == "frame" else 28 if k == "file" else 24)
        b = 36 * tris + out + (px * 12 if k == "frame" else 0)
        if k == "texture":
            flops, b = 3 * flops, b + 8 * case["res"] ** 2 * 3 * 4 * 2 + px * 24
        if k == "guided":
            b += 9760 * 1376
        if case.get("denoise"):
            flops, b = flops + px * 225 * 60, b + px * 160
        return {"bytes": float(b), "flops": float(flops)}
    if k == "denoise":
        px = case["width"] * case["height"]
        return {"bytes": float(px * (24 + 24 + 40 + 40)), "flops": float(px * 225 * 60)}
    tris = 2 * (case["grid"] - 1) ** 2 if k == "refit" else case["tris"]
    rays = case["rays"]
    b, flops = 36 * tris + rays * (32 + (4 if case.get("any") else 8)), rays * (20 * math.log2(max(2, tris)) + 150)
    if k == "refit":
        b += 36 * tris + 12 * case["grid"] ** 2
    elif k == "rebuild":
        b += 36 * tris * 2
    return {"bytes": float(b), "flops": float(flops)}


# ------------------------------------------------------------------ 64-bit values
def _nearest(rays, v):
    """Distance along each ray to the nearest triangle (v: (n, 3, 3)), -1 where it meets none: every pair, in
    64 bits, as products of the rays' Pluecker coordinates with the triangles'."""
    v = v.to(torch.float64)
    o, d = rays[:, 0:3].double(), rays[:, 4:7].double()
    tmin, tmax = rays[:, 3].double(), rays[:, 7].double()
    v0, e1, e2 = v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    n = torch.linalg.cross(e1, e2)
    line = torch.cat([torch.linalg.cross(o, d), d], 1)
    cu = torch.cat([e2, -torch.linalg.cross(e2, v0)], 1)
    cv = torch.cat([-e1, -torch.linalg.cross(v0, e1)], 1)
    nv0 = (n * v0).sum(1)
    out = torch.empty(len(rays), dtype=torch.float64, device=rays.device)
    step = max(1, (1 << 26) // max(1, len(v)))
    for a in range(0, len(rays), step):
        s = slice(a, a + step)
        inv = 1.0 / -(d[s] @ n.T)
        u, w = (line[s] @ cu.T) * inv, (line[s] @ cv.T) * inv
        t = (o[s] @ n.T - nv0) * inv
        ok = (u >= 0) & (w >= 0) & (u + w <= 1) & (t > 0) & (t >= tmin[s, None]) & (t < tmax[s, None])
        t = torch.where(ok, t, math.inf).amin(1)
        out[s] = torch.where(torch.isinf(t), -1.0, t)
    return out


def _t_quantiles(n, tail):
    """The t distribution's upper quantile at `tail` for 1..n degrees of freedom: t = sqrt(n) tan(a) turns the
    density into cos(a)^(n-1), integrated by Gauss-Legendre and inverted by bisection."""
    x, w = np.polynomial.legendre.leggauss(96)
    df = np.arange(1, n + 1, dtype=np.float64)[:, None]

    def above(a):  # integral from a to where cos(a)^(n-1) has died out, relative to the half range
        top = np.minimum(np.pi / 2, np.arccos(np.exp(-50.0 / np.maximum(df - 1, 1e-9))))
        mid, half = 0.5 * (top + a), 0.5 * (top - a)
        z = np.clip(mid + half * x, 0.0, np.pi / 2)
        return (half * (np.cos(z) ** (df - 1) * w).sum(1, keepdims=True))

    whole = 2.0 * above(np.zeros_like(df))
    lo, hi = np.zeros_like(df), np.full_like(df, np.pi / 2)
    for _ in range(60):
        a = 0.5 * (lo + hi)
        more = above(np.minimum(a, np.arccos(np.exp(-50.0 / np.maximum(df - 1, 1e-9))))) > tail * whole
        lo, hi = np.where(more, a, lo), np.where(more, hi, a)
    return (np.sqrt(df) * np.tan(lo))[:, 0]


def _bilateral(st):
    """The denoiser's filter in 64 bits: radius 7, a Welch t-test on the sample moments, G-buffer weights."""
    (g, s), xyz = st["records"], st["xyz"]

    def dev(a):
        return torch.as_tensor(np.ascontiguousarray(a).astype(np.float64), device=DEV)

    half = dev(g["h"].view(np.float16))
    alb, nrm, mr, model = half[..., 0:3], half[..., 3:6], half[..., 6:8], half[..., 8:13]
    nrm = nrm / nrm.norm(dim=-1, keepdim=True).clamp(min=1e-10)
    depth, num = dev(g["depth"]), dev(s["num"])[..., None]
    var = dev(s["m2n"]) * num / (num - 1).clamp(min=1)
    vth, theta = var / num, dev(s["mean"]) + dev(s["m3n"]) / 6 / var
    lo = vth ** 2 / (num - 1).clamp(min=1)
    col = torch.log1p(xyz)
    tq = torch.as_tensor(_t_quantiles(1024, 0.0025), device=DEV)
    h, w = depth.shape
    acc, wsum = col * 1e-6, torch.full_like(depth, 1e-6)
    for dj in range(-7, 8):
        for di in range(-7, 8):
            y = (torch.arange(h, device=DEV) + dj).clamp(0, h - 1)[:, None]
            x = (torch.arange(w, device=DEV) + di).clamp(0, w - 1)[None, :]
            t2 = (theta - theta[y, x]) ** 2
            ratio = (t2 + vth[y, x]) / (t2 + vth + vth[y, x]).clamp(min=1e-6)
            stat = torch.sqrt(0.5 / (1 - ratio) - 1)
            nu = (vth + vth[y, x]) ** 2 / (lo + lo[y, x])
            q = tq[(torch.nan_to_num(nu, nan=0.0).floor().clamp(1, 1024) - 1).long()]
            keep = (stat < q).all(-1)
            b = depth[y, x]
            term = ((alb - alb[y, x]) ** 2).sum(-1) * SIGMA["albedo"]
            term = term + (1 - (nrm * nrm[y, x]).sum(-1)) ** 2 * SIGMA["normal"]
            term = term + ((depth - b) / torch.maximum(depth, b).clamp(min=1e-6)) ** 2 * SIGMA["depth"]
            term = term + (mr[..., 0] - mr[y, x][..., 0]) ** 2 * SIGMA["metallic"]
            term = term + (mr[..., 1] - mr[y, x][..., 1]) ** 2 * SIGMA["rough"]
            term = term + (0.5 * (model - model[y, x]).abs().sum(-1)) ** 2 * SIGMA["model"]
            wt = torch.exp(-term - (di * di + dj * dj) * SIGMA["spatial"])
            wt = torch.where(keep, wt, 0.0)
            acc, wsum = acc + col[y, x] * wt[..., None], wsum + wt
    return torch.expm1(acc / wsum[..., None]).clamp(min=0)


def exact(case, seed):
    """Hit distances and the filtered image in 64 bits; path-traced images have no closed value."""
    k = case["kind"]
    if k == "denoise":
        return _bilateral(prepare(case, seed))
    if k not in ("rays", "refit", "rebuild") or case.get("any"):
        return None
    tris = 2 * (case["grid"] - 1) ** 2 if k == "refit" else case["tris"]
    if tris * case["rays"] > 4e10:
        return None
    if k == "refit":
        mesh = _grid_mesh(case["grid"], seed)
        v = _moved(mesh.vertices, seed)[torch.as_tensor(mesh.indices.astype(np.int64), device=DEV)]
        rays = _rays(case["rays"], seed, [0.0, 0.0, 0.0], [1.0, 0.3, 1.0], False)
    else:
        mesh = _triangle_mesh(case["tris"], seed + (1000003 if k == "rebuild" else 0))
        v = torch.as_tensor(mesh.vertices, device=DEV).reshape(-1, 3, 3)
        rays = _rays(case["rays"], seed, [0.0] * 3, [1.0] * 3, False)
    return {"ids": None, "t": _nearest(rays, v)}
