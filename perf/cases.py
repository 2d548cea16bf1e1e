"""The work this renderer is used for, as cases that can be timed and compared.

Every case goes through the package's public entry points, the way a program
that uses the renderer calls them: ray queries (``CudaIntegrator.intersect``
and the C ABI's device arrays), renders into host and device films, the
viewer's progressive passes, batches of views, the forward/backward pair and
the GPU BVH build. A program keeps one ``CudaIntegrator`` and the scenes it
uploaded; so does this file.

Scenes are the package's own presets. Meshes are fixed assets, generated once
per process; the seed draws what changes from call to call: materials, ray
sets, sample ranges, images.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

from pyre_gb300 import CudaIntegrator, PathIntegrator
from pyre_gb300 import native as N
from pyre_gb300 import presets as P
from pyre_gb300.scene import DisneyBsdf, Film, HdriEnvironmentLight, Lambertian, Scene

MAX_RAYS = 1 << 24               # the ray microbenchmark
MAX_SAMPLES = 1920 * 1080 * 64   # the headline frame


def listed():
    return [
        # picking and collision queries of a host program: a few rays at a time, host arrays in and out
        {"name": "query-cornell-4k", "kind": "query", "scene": "cornell_box", "level": 0, "rays": 4096, "any": False,
         "host": True},
        # visibility tests of a baking tool: any hit, device arrays, a mid-sized mesh, a ragged count
        {"name": "query-any-3m", "kind": "query", "scene": "mesh", "level": 7, "rays": 3_000_017, "any": True,
         "host": False},
        # the ray microbenchmark: 16.8 M incoherent rays against 1.3 M triangles, device arrays
        {"name": "query-closest-16m", "kind": "query", "scene": "mesh", "level": 8, "rays": 1 << 24, "any": False,
         "host": False},
        # a thumbnail: the smallest render, bound by launches
        {"name": "render-cornell-64", "kind": "render", "scene": "cornell_box", "width": 64, "height": 64, "spp": 4,
         "depth": 8, "cdf": False, "sort": 0, "crop": False, "host": True},
        # one refresh of the interactive viewer at the command line's default size
        {"name": "viewer-pass-800x600", "kind": "progressive", "scene": "studio_ref", "width": 800, "height": 600,
         "passes": 1, "depth": 8, "cdf": False},
        # the plain Cornell box of the benchmark plan, film to the host
        {"name": "render-cornell-256", "kind": "render", "scene": "cornell_box", "width": 256, "height": 256,
         "spp": 16, "depth": 8, "cdf": False, "sort": 0, "crop": False, "host": True},
        # one tile of a tiled preview: a ragged crop of an odd-sized image, the reference's own environment sampling
        {"name": "render-studio-tile", "kind": "render", "scene": "studio", "width": 959, "height": 541, "spp": 9,
         "depth": 5, "cdf": True, "sort": 0, "crop": True, "host": False},
        # the command line's default preset at its default size and sample count
        {"name": "render-cornellref-800x600", "kind": "render", "scene": "cornell_ref", "width": 800, "height": 600,
         "spp": 16, "depth": 8, "cdf": False, "sort": 0, "crop": False, "host": True},
        # the headline frame: 1080p, 64 spp, thin lens, motion blur, 2.1 M triangles, HDRI
        {"name": "render-studio-1080p", "kind": "render", "scene": "studio", "width": 1920, "height": 1080, "spp": 64,
         "depth": 8, "cdf": False, "sort": 1, "crop": False, "host": False},
        # a batch of views of uneven size, for data generation, films to the host
        {"name": "batch-40-views", "kind": "batch", "jobs": 40, "plan": 11, "res_max": 1024, "spp_max": 64},
        # one step of an inverse-rendering loop: forward, loss, path-replay adjoint
        {"name": "adjoint-512", "kind": "adjoint", "width": 512, "height": 512, "spp": 32, "depth": 8},
        # rebuilding a mesh's BVH on the GPU after it was deformed, host arrays in and out
        {"name": "bvh-build-300k", "kind": "bvh", "triangles": 300_007},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["query", "query", "render", "render", "render", "progressive", "batch", "adjoint", "bvh"])
    if kind == "query":
        mesh = rng.random() < 0.75
        rays = _log_uniform(rng, 4096, MAX_RAYS)
        return {"kind": kind, "scene": "mesh" if mesh else "cornell_box", "level": rng.randint(4, 8) if mesh else 0,
                "rays": rays, "any": rng.random() < 0.4, "host": rays < 100_000 and rng.random() < 0.5}
    if kind == "bvh":
        return {"kind": kind, "triangles": _log_uniform(rng, 1000, 20 * 4 ** 8)}
    if kind == "batch":
        return {"kind": kind, "jobs": rng.randint(3, 24), "plan": rng.randint(12, 10_000),
                "res_max": rng.choice([256, 512]), "spp_max": rng.choice([16, 64])}
    if kind == "adjoint":
        return {"kind": kind, "width": _log_uniform(rng, 48, 512), "height": _log_uniform(rng, 48, 512),
                "spp": _log_uniform(rng, 4, 32), "depth": rng.randint(4, 8)}
    if kind == "progressive":
        return {"kind": kind, "scene": rng.choice(["cornell_box", "cornell_ref", "studio_ref", "studio"]),
                "width": _log_uniform(rng, 64, 1920), "height": _log_uniform(rng, 48, 1080),
                "passes": rng.randint(1, 8), "depth": 8, "cdf": rng.random() < 0.5}
    scene = rng.choice(["cornell_box", "cornell_ref", "studio_ref", "studio", "studio"])
    return {"kind": "render", "scene": scene, "width": _log_uniform(rng, 32, 1920), "height": _log_uniform(rng, 32, 1080),
            "spp": _log_uniform(rng, 1, 64), "depth": rng.randint(4, 12), "cdf": rng.random() < 0.3,
            "sort": rng.choice([0, 1]), "crop": rng.random() < 0.25, "host": rng.random() < 0.5}


# ------------------------------------------------------------------ scenes --
@functools.lru_cache(maxsize=1)
def _ctx() -> CudaIntegrator:
    return CudaIntegrator(0)


@functools.lru_cache(maxsize=4)
def _preset(name: str, level: int = 0) -> Scene:
    if name == "mesh":
        return P.microbench_scene(level)
    if name == "studio":
        return P.studio_procedural()
    if name == "adjoint":
        return P.studio_procedural(hdri_size=(512, 256))
    return {"cornell_box": P.cornell_box, "cornell_ref": lambda: P.cornell_ref(True),
            "studio_ref": lambda: P.studio_ref(True)}[name]()


def _camera(name: str, width: int, height: int):
    if name in ("studio", "adjoint"):
        return P.studio_procedural_camera(width, height)
    if name == "studio_ref":
        return P.studio_ref_camera(width, height, aperture=0.05)
    return P.cornell_ref_camera(width, height) if name == "cornell_ref" else P.cornell_box_camera(width, height)


def _materials(materials, rng):
    """The scene's materials with colors (and Disney parameters) drawn from rng."""
    out = []
    for m in materials:
        if isinstance(m, Lambertian):
            out.append(Lambertian(np.clip(m.albedo * rng.uniform(0.85, 1.15, 3), 0, 0.95)))
        else:
            out.append(DisneyBsdf(rng.random(3), 1.0 if rng.random() < 0.3 else 0.0, 0.05 + 0.95 * rng.random(), 0.5))
    return out


def _seeded(base: Scene, seed: int) -> Scene:
    return Scene(list(base.primitives), _materials(base.materials, np.random.default_rng(seed)), list(base.lights),
                 base.env)


def _spp_begin(seed: int) -> int:
    return int(np.random.default_rng([seed, 1]).integers(1 << 20))


def _crop(case):
    """A quarter of the image, off its centre."""
    w, h = case["width"], case["height"]
    return (w // 5, h // 4, w // 5 + (w + 1) // 2, h // 4 + (h + 1) // 2) if case.get("crop") else None


def _crop_size(case):
    c = _crop(case) or (0, 0, case["width"], case["height"])
    return c[2] - c[0], c[3] - c[1]


def _rays(case, seed):
    base = _preset(case["scene"], case["level"])
    n = case["rays"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    if case["scene"] == "mesh":  # origins in the 1.5x bounds, as presets.random_rays draws them
        pos = base.primitives[0].instance.mesh.positions
        lo, hi = pos.min(0), pos.max(0)
        centre, half = torch.tensor((lo + hi) / 2).cuda(), torch.tensor((hi - lo) / 2 * 1.5).cuda()
    else:  # inside the box
        centre, half = torch.zeros(3, device="cuda"), torch.full((3,), 0.9, device="cuda")
    org = centre + (torch.rand(n, 3, device="cuda", generator=g) * 2 - 1) * half
    d = torch.randn(n, 3, device="cuda", generator=g)
    d = d / d.norm(dim=1, keepdim=True)
    tmin = torch.full((n,), 1e-4, device="cuda")
    tmax = torch.full((n,), math.inf, device="cuda")
    if case["any"]:  # visibility between points: segments of finite length
        tmax = torch.rand(n, device="cuda", generator=g) * 2 + 0.1
    return org.contiguous(), d.contiguous(), tmin, tmax


def _batch_plan(case):
    return _batch_plan_of(case["jobs"], case["plan"], case["res_max"], case["spp_max"])


@functools.lru_cache(maxsize=2)
def _batch_plan_of(jobs, plan, res_max, spp_max):
    res = tuple(r for r in (128, 256, 512, 1024) if r <= res_max)
    spp = tuple(s for s in (4, 16, 64) if s <= spp_max)
    return P.batch_jobs(jobs, seed=plan, resolutions=res, spps=spp)


# ----------------------------------------------------------------- prepare --
def prepare(case, seed):
    ctx = _ctx()
    st = {"ctx": ctx, "case": case}
    kind = case["kind"]
    rng = np.random.default_rng([seed, 2])
    if kind == "query":
        ctx.set_bvh_builder("device")
        st["scene"] = ctx.upload(_preset(case["scene"], case["level"]))
        ctx.set_bvh_builder("host")
        rays = _rays(case, seed)
        n = case["rays"]
        if case["host"]:
            st["rays"] = [r.cpu().numpy() for r in rays]
            return st
        st["rays"] = rays
        st["desc"] = N.Rays(*[N.dptr(r) for r in rays], None)
        if case["any"]:
            st["occ"] = torch.empty(n, dtype=torch.uint8, device="cuda")
        else:
            out = {k: torch.empty(n, dtype=torch.int32, device="cuda") for k in ("kind", "instance", "triangle")}
            out.update({k: torch.empty(n, dtype=torch.float32, device="cuda") for k in ("t", "u", "v")})
            st["out"] = out
            st["hits"] = N.Hits(*[N.dptr(out[k], C.c_int32) for k in ("kind", "instance", "triangle")],
                                *[N.dptr(out[k]) for k in ("t", "u", "v")])
        return st
    if kind == "bvh":
        level = next(k for k in range(9) if 20 * 4 ** k >= case["triangles"])
        mesh = P.icosphere_displaced(level, 0.1, seed=int(rng.integers(1 << 16)))
        n = case["triangles"]
        st["positions"], st["indices"] = mesh.positions, np.ascontiguousarray(mesh.indices[:3 * n])
        st["nodes"], st["prim"] = np.zeros(2 * n, N.BVH2_DTYPE), np.zeros(n, np.uint32)
        return st
    if kind == "batch":
        plan = _batch_plan(case)
        scenes, jobs = [], []
        for k, j in enumerate(plan):
            scenes.append(_seeded(j["scene"], seed * 1000 + k))
            jobs.append({"part": k, "camera": j["camera"], "width": j["width"], "height": j["height"], "spp": j["spp"],
                         "spp_begin": _spp_begin(seed), "integrator": j["integrator"]})
        ctx.set_bvh_builder("device")
        st["scene"] = ctx.upload_batch(scenes)
        ctx.set_bvh_builder("host")
        st["jobs"] = jobs
        st["films"] = [Film(j["width"], j["height"]) for j in plan]
        return st
    name = "adjoint" if kind == "adjoint" else case["scene"]
    sc = _seeded(_preset(name), seed)
    if kind == "adjoint":  # the environment is a parameter too
        env = sc.env
        px = (env.pixels * rng.uniform(0.5, 2.0, env.pixels.shape)).astype(np.float32)
        sc.env = HdriEnvironmentLight(env.width, env.height, px, env.intensity)
    w, h = case["width"], case["height"]
    st["it"] = PathIntegrator(case["depth"], 3)
    st["cam"] = _camera(name, w, h)
    st["spp_begin"] = _spp_begin(seed)
    ctx.set_bvh_builder("device")
    st["scene"] = ctx.upload(sc)
    ctx.set_bvh_builder("host")
    cw, ch = _crop_size(case)
    if kind == "adjoint":  # the target image: the scene with other materials
        ctx.set_materials(st["scene"], _materials(sc.materials, rng))
        st["target"] = ctx.render(st["scene"], st["cam"], st["it"], w, h, 4, spp_begin=1 << 22).radiance
        ctx.set_materials(st["scene"], sc.materials)
    elif kind == "progressive":
        if case["cdf"]:
            st["env_sampling"] = N.PYRE_ENV_CDF
        st["mean"] = rng.random((h, w, 3), dtype=np.float32)  # what the passes before left
    elif not case["host"]:
        film = {"radiance": torch.empty((ch, cw, 3), device="cuda"), "albedo": torch.empty((ch, cw, 3), device="cuda"),
                "normal": torch.empty((ch, cw, 3), device="cuda"), "depth": torch.empty((ch, cw), device="cuda")}
        st["film"] = film
        st["film_desc"] = N.Film(*[N.dptr(film[k]) for k in ("radiance", "albedo", "normal", "depth")],
                                 N.PYRE_MEM_DEVICE)
        st["params"] = ctx.params(w, h, st["spp_begin"], st["spp_begin"] + case["spp"], st["it"], crop=_crop(case),
                                  env_sampling=N.PYRE_ENV_CDF if case["cdf"] else N.PYRE_ENV_ALIAS,
                                  sort_by_material=case["sort"])
    return st


# --------------------------------------------------------------------- run --
def run(st):
    ctx, case = st["ctx"], st["case"]
    kind = case["kind"]
    if kind == "query":
        if case["host"]:
            r = ctx.intersect(st["scene"], *st["rays"], any_hit=case["any"])
            return {"occluded": r} if case["any"] else r
        if case["any"]:
            ctx.check(ctx.lib.pyre_intersect_any(ctx.handle, st["scene"].handle, C.byref(st["desc"]), case["rays"],
                                                 N.dptr(st["occ"], C.c_uint8), N.PYRE_MEM_DEVICE))
            return {"occluded": st["occ"]}
        ctx.check(ctx.lib.pyre_intersect_closest(ctx.handle, st["scene"].handle, C.byref(st["desc"]), case["rays"],
                                                 C.byref(st["hits"]), N.PYRE_MEM_DEVICE))
        return st["out"]
    if kind == "bvh":
        nodes, prim, count = st["nodes"], st["prim"], C.c_uint32()
        ctx.check(ctx.lib.pyre_bvh_build_device(ctx.handle, N.fptr(st["positions"]), len(st["positions"]),
                                                N.u32ptr(st["indices"]), case["triangles"],
                                                nodes.ctypes.data_as(C.POINTER(N.Bvh2Node)), N.u32ptr(prim),
                                                C.byref(count)))
        return {"bounds_min": nodes["bounds_min"], "bounds_max": nodes["bounds_max"],
                "offset": nodes["offset"].view(np.int32), "count": nodes["n_primitives"].view(np.int16),
                "axis": nodes["axis"], "primitives": prim.view(np.int32), "nodes": count.value}
    if kind == "batch":
        films = ctx.render_batch(st["scene"], st["jobs"], films=st["films"])
        return {"radiance": [f.radiance for f in films][:24], "depth": [f.depth for f in films][:24]}
    w, h = case["width"], case["height"]
    if kind == "adjoint":
        img = ctx.forward(st["scene"], st["cam"], st["it"], w, h, case["spp"], spp_begin=st["spp_begin"]).radiance
        dl = (2.0 / img.size) * (img - st["target"])
        mat, env = ctx.backward(st["scene"], st["cam"], st["it"], w, h, case["spp"], dl, spp_begin=st["spp_begin"])
        return {"image": img, "materials": mat, "env": env}
    if kind == "progressive":
        first = 1 + st["spp_begin"] % 1000
        mean = ctx.render_progressive(st["scene"], st["cam"], st["it"], w, h, case["passes"], mean=st["mean"].copy(),
                                      pass_begin=first, env_sampling=st.get("env_sampling", N.PYRE_ENV_ALIAS))
        return {"mean": mean}
    if case["host"]:
        f = ctx.render(st["scene"], st["cam"], st["it"], w, h, case["spp"], spp_begin=st["spp_begin"], crop=_crop(case),
                       env_sampling=N.PYRE_ENV_CDF if case["cdf"] else N.PYRE_ENV_ALIAS, sort_by_material=case["sort"])
        return {"radiance": f.radiance, "albedo": f.albedo, "normal": f.normal, "depth": f.depth}
    ctx.render_into(st["scene"], st["cam"], st["params"], st["film_desc"])
    return st["film"]


# -------------------------------------------------------------------- work --
def _triangles(name, level=0):
    if name == "mesh":
        return 20 * 4 ** level
    return {"cornell_box": 34, "cornell_ref": 2 * 2 * 48 * 23 + 34, "studio_ref": 2 * 2 * 64 * 31 + 2,
            "studio": 64 * 32768 + 2, "adjoint": 64 * 32768 + 2}[name]


def _ray_flops(triangles):
    """Two child boxes of 18 operations per level of a binary tree, and two triangle tests of 45."""
    return 36 * max(1.0, math.log2(triangles)) + 90


def _sample_flops(name):
    """Path vertices per sample (Russian roulette from depth 3), each with a closest-hit ray, a shadow ray and
    about 300 operations of shading."""
    vertices = 2.4 if name in ("studio", "adjoint") else 2.0 if name == "studio_ref" else 4.0
    return vertices * (2 * _ray_flops(_triangles(name)) + 300)


def work(case):
    kind = case["kind"]
    if kind == "query":
        t = _triangles(case["scene"], case["level"])
        n = case["rays"]
        return {"bytes": n * (32 + (1 if case["any"] else 24)) + 36 * t, "flops": n * _ray_flops(t)}
    if kind == "bvh":
        t = case["triangles"]
        # positions and indices in; two nodes of 32 B per leaf and the order out; each primitive binned per level
        return {"bytes": t * (6 + 12 + 40 + 4), "flops": t * 40 * math.log2(t)}
    if kind == "batch":
        plan = _batch_plan(case)
        pix = sum(j["width"] * j["height"] for j in plan)
        fl = sum(j["width"] * j["height"] * j["spp"] * 4.0 * (2 * _ray_flops(j["scene"].triangle_count()) + 300)
                 for j in plan)
        return {"bytes": pix * 40 + 36 * sum(j["scene"].triangle_count() for j in plan), "flops": fl}
    cw, ch = _crop_size(case)
    pix = cw * ch
    if kind == "progressive":
        return {"bytes": pix * 24 + 36 * _triangles(case["scene"]),
                "flops": pix * case["passes"] * _sample_flops(case["scene"])}
    if kind == "adjoint":
        env = 512 * 256 * 12
        # the adjoint replays the forward's paths and evaluates the BSDF's derivatives at each vertex
        return {"bytes": pix * (12 + 12 + 12) + 36 * _triangles("adjoint") + 2 * env,
                "flops": pix * case["spp"] * 2.5 * _sample_flops("adjoint")}
    return {"bytes": pix * 40 + 36 * _triangles(case["scene"]), "flops": pix * case["spp"] * _sample_flops(case["scene"])}


# ------------------------------------------------------------------- exact --
# The same results in 64 bits: brute-force ray queries, and a path tracer for
# the Lambertian Cornell box that consumes the sampler's own stream.
F64 = torch.float64


def _t64(a):
    return torch.as_tensor(np.asarray(a, np.float64), device="cuda")


def _cross(a, b):
    return torch.linalg.cross(a, b, dim=-1)


def _dot(a, b):
    return (a * b).sum(-1)


class _Soup:
    """Every triangle of a scene without motion, and its quad lights."""

    def __init__(self, sc: Scene):
        v, nrm, mat = [], [], []
        for p in sc.primitives:
            m = p.instance.mesh
            tri = m.indices.reshape(-1, 3)
            v.append(m.positions[tri])
            nrm.append(m.normals[tri] if m.normals is not None else np.zeros((len(tri), 3, 3), np.float32))
            mat += [p.material_id] * len(tri)
        v = _t64(np.concatenate(v))
        self.v0, self.e1, self.e2 = v[:, 0], v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
        self.normals, self.mat = _t64(np.concatenate(nrm)), torch.tensor(mat, device="cuda")
        self.lights = [{k: _t64(getattr(q, k)) for k in ("p0", "edge_u", "edge_v", "emission")} for q in sc.lights]
        for q in self.lights:
            q["crs"] = _cross(q["edge_u"], q["edge_v"])
            q["area"] = q["crs"].norm()
            q["normal"] = q["crs"] / q["area"]

    def closest(self, o, d, tmin, tmax, chunk=1 << 25):
        """(t, u, v, triangle) of the closest hit per ray; t = inf where there is none."""
        n, out = o.shape[0], []
        step = max(1, chunk // self.v0.shape[0])
        for a in range(0, n, step):
            oo, dd = o[a:a + step, None], d[a:a + step, None]
            h = _cross(dd.expand(-1, self.e2.shape[0], -1), self.e2[None].expand(oo.shape[0], -1, -1))
            det = _dot(self.e1[None], h)
            f = 1.0 / torch.where(det.abs() < 1e-8, math.inf, det)
            s = oo - self.v0[None]
            u = f * _dot(s, h)
            q = _cross(s, self.e1[None].expand(s.shape[0], -1, -1))
            v = f * _dot(dd, q)
            t = f * _dot(self.e2[None], q)
            ok = (det.abs() >= 1e-8) & (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1)
            ok &= (t > tmin[a:a + step, None]) & (t < tmax[a:a + step, None])
            t, k = torch.where(ok, t, math.inf).min(1)
            pick = lambda x: x.gather(1, k[:, None])[:, 0]  # noqa: E731
            out.append((t, pick(u), pick(v), k))
        return [torch.cat(x) for x in zip(*out)]

    def light(self, q, o, d, tmin, tmax):
        """Distance to quad light q, inf where the ray misses it."""
        den = _dot(d, q["normal"])
        t = _dot(q["p0"] - o, q["normal"]) / torch.where(den.abs() < 1e-9, math.inf, den)
        r = o + t[:, None] * d - q["p0"]
        c2 = _dot(q["crs"], q["crs"])
        al = _dot(_cross(r, q["edge_v"].expand_as(r)), q["crs"]) / c2
        be = _dot(_cross(q["edge_u"].expand_as(r), r), q["crs"]) / c2
        ok = (den.abs() >= 1e-9) & (t >= tmin) & (t <= tmax) & (al >= 0) & (al <= 1) & (be >= 0) & (be <= 1)
        return torch.where(ok, t, math.inf)


def _shr(x, k):
    return (x >> k) & ((1 << (64 - k)) - 1)


def _signed(x):
    return x - (1 << 64) if x >= 1 << 63 else x


class _Stream:
    """pixel_seed and Xoshiro256++ (sampler.rs:15-49) for many paths at once, in wrapping 64-bit integers."""

    def __init__(self, x, y, s):
        mul = lambda a, k: a * _signed(k)  # noqa: E731
        h = (x << 32) | y
        h = h ^ mul(s, 0x9E3779B97F4A7C15)
        h = mul(h ^ _shr(h, 30), 0xBF58476D1CE4E5B9)
        h = mul(h ^ _shr(h, 27), 0x94D049BB133111EB)
        seed = h ^ _shr(h, 31)
        self.s = []
        for _ in range(4):
            seed = seed + _signed(0x9E3779B97F4A7C15)
            z = mul(seed ^ _shr(seed, 30), 0xBF58476D1CE4E5B9)
            z = mul(z ^ _shr(z, 27), 0x94D049BB133111EB)
            self.s.append(z ^ _shr(z, 31))

    def draw(self):
        rotl = lambda v, k: (v << k) | _shr(v, 64 - k)  # noqa: E731
        a, b, c, d = self.s
        out = rotl(a + d, 23) + a
        t = b << 17
        c, d = c ^ a, d ^ b
        b, a = b ^ c, a ^ d
        self.s = [a, b, c ^ t, rotl(d, 45)]
        return _shr(out, 40).to(F64) / 16777216.0


def _exact_cornell(case, seed):
    """The Lambertian Cornell box, path by path (camera.rs:65-73, integrator.rs:57-240), in 64 bits."""
    sc = _seeded(_preset("cornell_box"), seed)
    soup, cam = _Soup(sc), _camera("cornell_box", case["width"], case["height"])
    albedo = _t64([m.albedo for m in sc.materials])
    w, h, spp, first = case["width"], case["height"], case["spp"], _spp_begin(seed)
    c = _crop(case) or (0, 0, w, h)
    org, tgt, up = _t64(cam.origin), _t64(cam.target), _t64(cam.up)
    unit = lambda a: a / a.norm(dim=-1, keepdim=True)  # noqa: E731
    fwd = unit(tgt - org)
    right = unit(_cross(fwd, up))
    vup = _cross(right, fwd)
    hh = math.tan(math.radians(cam.vfov_deg) / 2)
    hw = cam.aspect * hh
    ys, xs = torch.meshgrid(torch.arange(c[1], c[3], device="cuda"), torch.arange(c[0], c[2], device="cuda"),
                            indexing="ij")
    total = {"radiance": 0, "albedo": 0, "normal": 0, "depth": 0}
    x, y = xs.reshape(-1), ys.reshape(-1)
    for s in range(first, first + spp):
        g = _Stream(x, y, torch.full_like(x, s))
        jx, jy = g.draw(), g.draw()
        for _ in range(3):  # lens and time
            g.draw()
        nx, ny = 2 * (x + jx) / w - 1, 1 - 2 * (y + jy) / h
        d = unit(fwd + nx[:, None] * hw * right + ny[:, None] * hh * vup)
        o = org.expand_as(d)
        n = x.numel()
        rad, beta = torch.zeros(n, 3, device="cuda", dtype=F64), torch.ones(n, 3, device="cuda", dtype=F64)
        aov_a, aov_n, aov_d = torch.zeros_like(rad), torch.zeros_like(rad), torch.zeros(n, device="cuda", dtype=F64)
        live = torch.ones(n, device="cuda", dtype=torch.bool)
        last = torch.zeros_like(aov_d)
        lo, inf = torch.full_like(last, 1e-4), torch.full_like(last, math.inf)
        q = soup.lights[0]
        power = lambda a, b: a * a / (a * a + b * b)  # noqa: E731
        for depth in range(case["depth"]):
            t, u, v, k = soup.closest(o, d, lo, inf)
            tl = soup.light(q, o, d, 1e-4, t)
            at_light = live & (tl < t)
            cos_l = -_dot(d, q["normal"])
            le = torch.where((cos_l > 0)[:, None], q["emission"], 0.0)
            wt = torch.ones_like(last) if depth == 0 else power(last, torch.where(
                cos_l > 0, tl * tl / (cos_l * q["area"]), 0.0))
            rad = torch.where(at_light[:, None], rad + beta * le * wt[:, None], rad)
            surf = live & ~at_light & t.isfinite()
            t = torch.where(surf, t, 1.0)
            p = o + d * t[:, None]
            nn = soup.normals[k]
            ns = unit((1 - u - v)[:, None] * nn[:, 0] + u[:, None] * nn[:, 1] + v[:, None] * nn[:, 2])
            alb = albedo[soup.mat[k]]
            if depth == 0:
                aov_a = torch.where(surf[:, None], alb, torch.where(at_light[:, None], 1.0, 0.0))
                aov_n = torch.where(surf[:, None], ns, torch.where(at_light[:, None], q["normal"], 0.0))
                aov_d = torch.where(surf, t, torch.where(at_light, tl, 0.0))
            helper = torch.where((ns[:, :1].abs() > 0.9), _t64([0, 1, 0]), _t64([1, 0, 0]))
            ft = unit(_cross(helper, ns))
            fb = _cross(ns, ft)
            live = surf & (-_dot(d, ns) > 0)
            po = p + 1e-3 * ns
            u0, u1 = g.draw(), g.draw()  # the quad light
            lp = q["p0"] + u0[:, None] * q["edge_u"] + u1[:, None] * q["edge_v"]
            dist2 = _dot(lp - p, lp - p)
            wi = (lp - p) / dist2.sqrt()[:, None]
            cl, cs = -_dot(wi, q["normal"]), _dot(wi, ns)
            lpdf = dist2 / (cl * q["area"])
            to = (lp - 1e-3 * wi) - po
            dist = to.norm(dim=-1)
            nee = live & (cl > 0) & (cs > 0)
            st = soup.closest(po, to / dist[:, None], torch.full_like(last, 1e-3), dist - 1e-3)[0]
            nee &= ~st.isfinite()
            con = beta * alb / math.pi * q["emission"] * (cs * power(lpdf, cs / math.pi) / lpdf)[:, None]
            rad = torch.where(nee[:, None], rad + con, rad)
            u0, u1 = g.draw(), g.draw()  # the BSDF
            r, phi = u0.sqrt(), 2 * math.pi * u1
            cz = (1 - u0).sqrt()
            d = (r * phi.cos())[:, None] * ft + (r * phi.sin())[:, None] * fb + cz[:, None] * ns
            live = live & (cz > 0)
            last = cz / math.pi
            beta = beta * alb
            if depth >= 3:  # Russian roulette
                stop = (1 - beta.max(1).values).clamp(0.05, 0.95)
                live = live & (g.draw() >= stop)
                beta = beta / (1 - stop)[:, None]
            o = po
        total = {k: total[k] + a for k, a in (("radiance", rad), ("albedo", aov_a), ("normal", aov_n), ("depth", aov_d))}
    shape = (c[3] - c[1], c[2] - c[0])
    return {k: (a / spp).reshape(shape + a.shape[1:]) for k, a in total.items()}


def exact(case, seed):
    if case["kind"] == "query" and not case["any"]:
        sc = _preset(case["scene"], case["level"])
        if case["rays"] * sc.triangle_count() > 4e9:
            return None
        soup = _Soup(sc)
        org, d, tmin, tmax = [r.to(F64) for r in _rays(case, seed)]
        t, u, v, _ = soup.closest(org, d, tmin, tmax)
        hit = t.isfinite()
        for q in soup.lights:
            tl = soup.light(q, org, d, tmin, t)
            hit &= ~(tl < t)
            t = torch.minimum(t, tl)
        out = {"kind": None, "instance": None, "triangle": None, "t": t, "u": None, "v": None}
        if case["scene"] == "mesh":  # the Cornell boxes stand on the floor: two faces at one distance
            out.update(u=torch.where(hit, u, 0.0), v=torch.where(hit, v, 0.0))
        return out
    if case["kind"] == "render" and case["scene"] == "cornell_box":
        cw, ch = _crop_size(case)
        if cw * ch * case["spp"] <= 1 << 22 and case["depth"] <= 12:
            return _exact_cornell(case, seed)
    return None
