"""What this framework's users have it do, as cases that can be timed and compared.

Every case goes through the package's public entry points (Scene, SceneBatch, the schedulers,
DifferentiableRender). Sizes are those of the repository's benchmark configurations and tests, or generic.

  hits      closest hits of a batch of device rays (Scene.intersect_device)
  visible   any-hit visibility of a batch of device segments (Scene.occluded_device)
  host      closest hits of a host array of rays (Scene.intersect_host)
  render    one scene through the "mt" scheduler into a host film (pt, pt.direct, pt.mis)
  frame     one scene through SceneBatch.render_device into a device film
  batch     several scenes of different sizes through SceneBatch.render_device
  adjoint   forward image and gradients (DifferentiableRender)
"""
import math
import warnings

import numpy as np
import torch

from lightmetrica_b200 import scenes, workloads
from lightmetrica_b200.batch import SceneBatch
from lightmetrica_b200.diff import DifferentiableRender, light_emission, triangle_albedo
from lightmetrica_b200.render import create_renderer, create_scheduler
from lightmetrica_b200.scene import create_scene, soup_primitives

warnings.filterwarnings("ignore", category=RuntimeWarning)
DEV = "cuda"


# ---------------------------------------------------------------- the cases ----

def listed():
    return [
        # An interactive pick or a few probe rays: latency and launch count.
        {"name": "hits_tiny", "kind": "hits", "impl": "bvh", "tris": 4096, "rays": 512},
        # An ordinary query of a baking tool: odd sizes, the 4-wide scene type.
        {"name": "hits_ragged", "kind": "hits", "impl": "qbvh", "tris": 65537, "rays": 300007},
        # The ray-intersection benchmark's soup, incoherent rays; half its rays per call.
        {"name": "hits_soup", "kind": "hits", "impl": "bvh", "tris": 1048576, "rays": 1 << 23},
        # Visibility segments between points inside a scene (ambient occlusion, light baking).
        {"name": "visible", "kind": "visible", "impl": "bvh", "tris": 262144, "rays": 2000003},
        # A host program's query: pageable host arrays in and out.
        {"name": "host_rays", "kind": "host", "impl": "bvh", "tris": 30011, "rays": 1000003},
        # The Cornell box benchmark configuration, whole scheduler call.
        {"name": "cornell", "kind": "render", "scene": "classic", "tech": "pt.mis", "w": 256, "h": 256, "spp": 16,
         "max_pv": 9, "rr": 3, "sampling": "stratified", "fp64": False},
        # A preview: tiny film, mirrors and an environment, unbounded depth, uniform raster, double film.
        {"name": "preview_pt", "kind": "render", "scene": "mixed", "tech": "pt", "w": 67, "h": 45, "spp": 8,
         "max_pv": -1, "rr": 1, "sampling": "uniform", "fp64": True},
        # Direct lighting of a terrain with objects through the scheduler.
        {"name": "terrain_direct", "kind": "render", "scene": "terrain", "grid": 256, "spheres": 24, "ico": 3,
         "tech": "pt.direct", "w": 641, "h": 359, "spp": 8, "max_pv": 6, "rr": 3, "sampling": "stratified", "fp64": False},
        # The headline frame's scene type, camera and film; fewer triangles and samples, so that it builds quickly.
        {"name": "frame_1080p", "kind": "frame", "grid": 512, "spheres": 64, "ico": 4, "w": 1920, "h": 1080, "spp": 8,
         "max_pv": 17, "rr": 5, "layout": "bvh"},
        # Scenes of the 64-scene benchmark set rendered together (soups and heightfields, half mirror).
        {"name": "batch_6", "kind": "batch", "count": 6, "first": 10, "mode": "waves", "layout": "bvh", "spp_max": 16},
        # The differentiable benchmark configuration: forward image and gradients.
        {"name": "adjoint", "kind": "adjoint", "levels": 5, "tech": "pt.mis", "w": 512, "h": 512, "spp": 32,
         "max_pv": 9, "rr": 3},
        # A gradient step of an optimisation loop on a small image.
        {"name": "adjoint_small", "kind": "adjoint", "levels": 1, "tech": "pt.direct", "w": 65, "h": 49, "spp": 4,
         "max_pv": 6, "rr": 3},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["hits", "visible", "host", "render", "render", "frame", "batch", "adjoint"])
    if kind in ("hits", "visible", "host"):
        top = {"hits": 1 << 23, "visible": 1 << 22, "host": 1 << 20}[kind]
        return {"kind": kind, "impl": rng.choice(["bvh", "bvh", "qbvh"]), "tris": _log_int(rng, 1000, 1 << 20),
                "rays": _log_int(rng, 256, top)}
    tech = rng.choice(["pt", "pt.direct", "pt.mis"])
    w = _log_int(rng, 32, 700)
    h = max(16, int(w * rng.uniform(0.5, 1.0)))
    depth = rng.randint(3, 17)
    rr = rng.randint(1, 5)
    spp = rng.randint(1, 16)
    if kind == "render":
        c = {"kind": kind, "scene": rng.choice(["classic", "mixed", "terrain"]), "tech": tech, "w": w, "h": h, "spp": spp,
             "max_pv": rng.choice([depth, depth, -1]), "rr": rr, "sampling": rng.choice(["stratified", "uniform"]),
             "fp64": rng.random() < 0.25}
        if c["scene"] == "terrain":
            c.update(grid=_log_int(rng, 32, 512), spheres=rng.randint(1, 64), ico=rng.randint(1, 4))
        return c
    if kind == "frame":
        return {"kind": kind, "grid": _log_int(rng, 64, 512), "spheres": rng.randint(4, 64), "ico": rng.randint(2, 4),
                "w": 2 * w, "h": 2 * h, "spp": rng.randint(1, 8), "max_pv": depth, "rr": rr,
                "layout": rng.choice(["bvh", "qbvh", "bvh_q16", "bvh_qshadow"])}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(2, 8), "first": rng.randint(0, 56),
                "mode": rng.choice(["waves", "overlap", "stream"]), "layout": rng.choice(["bvh", "bvh_qshadow"]),
                "spp_max": rng.randint(2, 8)}
    return {"kind": kind, "levels": rng.randint(0, 5), "tech": tech, "w": min(w, 512), "h": min(h, 512), "spp": spp,
            "max_pv": min(depth, 9), "rr": rr}


# ------------------------------------------------------------------ inputs ----

def _torch_gen(seed):
    return torch.Generator(device=DEV).manual_seed(1000003 * int(seed) + 17)


def _soup(case, seed):
    return workloads.random_soup(case["tris"], seed=7919 * int(seed) + 1, sigma=0.01 * math.sqrt((1 << 20) / case["tris"]) ** 0.75)


def _device_rays(case, seed):
    """SoA rays: origins in [-2, 2]^3 and directions on the sphere, or segments between points of the scene's box."""
    n, g = case["rays"], _torch_gen(seed)
    if case["kind"] == "visible":
        a, b = (torch.rand((3, n), generator=g, device=DEV) * 2.0 - 1.0 for _ in range(2))
        d = b - a
        length = d.norm(dim=0)
        d = d / length
        tmin, tmax = torch.full((n,), 1e-4, device=DEV), length * (1.0 - 1e-4)
    else:
        a = torch.rand((3, n), generator=g, device=DEV) * 4.0 - 2.0
        z = 1.0 - 2.0 * torch.rand(n, generator=g, device=DEV)
        phi = 2.0 * math.pi * torch.rand(n, generator=g, device=DEV)
        r = torch.sqrt(torch.clamp(1.0 - z * z, min=0.0))
        d = torch.stack([r * torch.cos(phi), r * torch.sin(phi), z])
        tmin, tmax = torch.zeros(n, device=DEV), torch.full((n,), workloads.FLT_MAX, device=DEV)
    return {"ox": a[0].contiguous(), "oy": a[1].contiguous(), "oz": a[2].contiguous(), "dx": d[0].contiguous(),
            "dy": d[1].contiguous(), "dz": d[2].contiguous(), "tmin": tmin, "tmax": tmax}


def _scene_prims(case, seed):
    """The scene's primitives and sizes; the seed moves the terrain and the objects."""
    if case["kind"] == "adjoint":
        return scenes.cornell_refined(case["levels"], case["w"], case["h"])
    if case["kind"] == "frame" or case["scene"] == "terrain":
        return scenes.terrain_spheres(case["w"], case["h"], grid=case["grid"], spheres=case["spheres"],
                                      ico_level=case["ico"], seed=100 + int(seed))
    return scenes.cornell_box(case["w"], case["h"], variant=case["scene"])


def _built(prims, impl="bvh"):
    sc = create_scene(impl)
    sc.load(prims)
    sc.configure({})
    sc.build()
    return sc


def _renderer(tech, rr, max_pv, seed, sampling="stratified"):
    r = create_renderer(tech)
    r.configure({"rr_depth": rr, "max_path_vertices": max_pv, "sampler": {"rng_seed": int(seed) + 11, "sampling": sampling}})
    return r


def _batch_items(case):
    return [scenes.batch_scene(case["first"] + i) for i in range(case["count"])]


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("hits", "visible", "host"):
        pos, faces = _soup(case, seed)
        st = {"kind": kind, "scene": _built(soup_primitives(pos, faces), case["impl"]), "n": case["rays"]}
        rays = _device_rays(case, seed)
        if kind == "host":
            st["rays"] = torch.stack([rays[k] for k in ("ox", "oy", "oz", "dx", "dy", "dz", "tmin", "tmax")], 1).cpu().numpy()
            return st
        st["keep"] = rays
        st["rays"] = {k: v.data_ptr() for k, v in rays.items()}
        n = case["rays"]
        if kind == "visible":
            st["out"] = torch.zeros(n, dtype=torch.uint8, device=DEV)
        else:
            st["out"] = {"tri_id": torch.zeros(n, dtype=torch.int32, device=DEV), **{k: torch.zeros(n, device=DEV) for k in "tuv"}}
            st["hits"] = {k: v.data_ptr() for k, v in st["out"].items()}
        return st
    if kind == "render":
        sched = create_scheduler("mt")
        sched.configure({"num_samples": case["w"] * case["h"] * case["spp"], "film_fp64": case["fp64"]})
        return {"kind": kind, "scene": _built(_scene_prims(case, seed)), "sched": sched,
                "renderer": _renderer(case["tech"], case["rr"], case["max_pv"], seed, case["sampling"])}
    if kind == "frame":
        sc = _built(_scene_prims(case, seed))
        b = SceneBatch([sc])
        b.configure(layout=case["layout"])
        return {"kind": kind, "scenes": [sc], "batch": b, "samples": [case["w"] * case["h"] * case["spp"]],
                "renderers": [_renderer("pt.mis", case["rr"], case["max_pv"], seed)],
                "films": [torch.zeros(case["h"] * case["w"] * 3, device=DEV)]}
    if kind == "batch":
        items = _batch_items(case)
        scs = [_built(it["prims"]) for it in items]
        b = SceneBatch(scs)
        b.configure(layout=case["layout"], mode=case["mode"])
        films = [it["prims"].camera.film for it in items]
        return {"kind": kind, "scenes": scs, "batch": b,
                "samples": [f.width * f.height * min(it["spp"], case["spp_max"]) for f, it in zip(films, items)],
                "renderers": [_renderer("pt.mis", 5, it["max_path_vertices"], seed + 31 * i) for i, it in enumerate(items)],
                "films": [torch.zeros(f.width * f.height * 3, device=DEV) for f in films]}
    prims = _scene_prims(case, seed)
    sc = _built(prims)
    albedo, emission, target = _diff_inputs(prims, case, seed)
    return {"kind": kind, "scene": sc, "albedo": albedo, "emission": emission, "dL": target,
            "diff": DifferentiableRender(sc, _renderer(case["tech"], case["rr"], case["max_pv"], seed),
                                         case["w"] * case["h"] * case["spp"])}


def _diff_inputs(prims, case, seed):
    """Per-triangle albedo around the scene's own, light emission, and the loss gradient of an image."""
    g = _torch_gen(seed)
    albedo = torch.from_numpy(triangle_albedo(prims)).to(DEV)
    albedo = (albedo * (0.8 + 0.4 * torch.rand(albedo.shape, generator=g, device=DEV))).clamp(max=0.95)
    emission = torch.from_numpy(light_emission(prims)).to(DEV)
    dL = torch.randn((case["h"], case["w"], 3), generator=g, device=DEV) / (case["h"] * case["w"]) + 1.0 / (case["h"] * case["w"])
    return albedo, emission, dL


# -------------------------------------------------------------------- runs ----

def run(state):
    kind = state["kind"]
    if kind == "hits":
        state["scene"].intersect_device(state["rays"], state["hits"], state["n"], torch.cuda.current_stream().cuda_stream)
        return state["out"]
    if kind == "visible":
        state["scene"].occluded_device(state["rays"], state["out"].data_ptr(), state["n"], torch.cuda.current_stream().cuda_stream)
        return state["out"]
    if kind == "host":
        return state["scene"].intersect_host(state["rays"])
    if kind == "render":
        return state["sched"].render(state["renderer"], state["scene"])
    if kind in ("frame", "batch"):
        for f in state["films"]:
            f.zero_()
        return state["batch"].render_device(state["renderers"], state["samples"], state["films"])
    image = state["diff"].forward(state["albedo"], state["emission"])
    d_albedo, d_emission = state["diff"].backward(state["albedo"], state["emission"], state["dL"])
    return {"image": image, "d_albedo": d_albedo, "d_emission": d_emission}


# ------------------------------------------------------ work and tolerance ----

def _ray_flops(tris):
    """One ray: a balanced binary tree's two box tests per level (6 multiply-adds and the comparisons) and a triangle test."""
    return 2 * 20 * max(1.0, math.log2(max(2, tris))) + 40


def _render_work(samples, tris, pixels, max_pv, rr, shadow, passes=1):
    """A sample's rays: the camera's, one a bounce until Russian roulette ends the path (survival at most a half), and a
    shadow ray per vertex where the technique casts them; 300 operations of shading a vertex."""
    depth = 64 if max_pv == -1 else max_pv - 1
    verts = sum(0.5 ** max(0, k - max(1, rr) + 1) * 0.8 ** (k - 1) for k in range(1, depth + 1))
    rays = samples * verts * (2 if shadow else 1)
    return {"bytes": passes * (48.0 * tris + 12.0 * pixels), "flops": passes * (rays * _ray_flops(tris) + samples * verts * 300.0)}


def work(case):
    kind = case["kind"]
    if kind in ("hits", "host", "visible"):
        out = 1 if kind == "visible" else 16
        return {"bytes": case["rays"] * (32.0 + out) + 48.0 * case["tris"], "flops": case["rays"] * _ray_flops(case["tris"])}
    if kind == "batch":
        parts = []
        for it in _batch_items(case):
            px = it["prims"].camera.film.width * it["prims"].camera.film.height
            parts.append(_render_work(px * min(it["spp"], case["spp_max"]), it["triangles"], px, it["max_path_vertices"], 5, True))
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    px = case["w"] * case["h"]
    if kind == "adjoint":
        return _render_work(px * case["spp"], 36 * 4 ** case["levels"], px, case["max_pv"], case["rr"], case["tech"] != "pt", 2)
    if kind == "frame" or case["scene"] == "terrain":
        tris = 2 * (case["grid"] - 1) ** 2 + case["spheres"] * 20 * 4 ** case["ico"] + 320
    else:
        tris = 36
    return _render_work(px * case["spp"], tris, px, case["max_pv"], case["rr"], kind == "frame" or case["tech"] != "pt")


def tolerance(case):
    # Closest hits and visibility are the reference's, bit for bit, in every layout.
    if case["kind"] in ("hits", "host", "visible"):
        return "exact"
    # Renders compare sample by sample (same random numbers). The device code compiled with fused multiply-adds, another
    # correct implementation at the same precision, differs by up to 2.4e-3: a ray within rounding of an edge takes
    # another path. Order of the film's float atomics: 5e-7. Another tree or node layout: up to 3.4e-4.
    return {"rel": 1e-2}


# ------------------------------------------------------------ 64-bit results ----

def exact(case, seed):
    kind = case["kind"]
    if kind in ("hits", "visible", "host"):
        if case["rays"] * case["tris"] > 4e10:
            return None
        return _exact_hits(case, seed)
    if kind == "render" and case["scene"] in ("classic", "mixed"):
        prims = _scene_prims(case, seed)
        image, _ = _PathTracer(prims, case["tech"], case["rr"], case["max_pv"], case["sampling"] == "stratified",
                               int(seed) + 11).film(case["w"] * case["h"] * case["spp"])
        return image.cpu().numpy()
    if kind == "adjoint" and case["levels"] <= 2 and case["w"] * case["h"] * case["spp"] * 4 ** case["levels"] <= 1 << 20:
        prims = _scene_prims(case, seed)
        albedo, emission, dL = _diff_inputs(prims, case, seed)
        pt = _PathTracer(prims, case["tech"], case["rr"], case["max_pv"], True, int(seed) + 11,
                         albedo.double().requires_grad_(), emission.double().requires_grad_())
        image, (albedo, emission) = pt.film(case["w"] * case["h"] * case["spp"])
        da, de = torch.autograd.grad((image * dL.double()).sum(), (albedo, emission))
        return {"image": image.detach(), "d_albedo": da, "d_emission": de}
    return None


def _nearest(p1, e1, e2, o, d, tmin, tmax, any_hit=False):
    """Brute force over all triangles in 64 bits: (index or -1, t, u, v) per ray, or whether any is hit."""
    T, n = p1.shape[0], o.shape[0]
    idx = torch.full((n,), -1, dtype=torch.int64, device=o.device)
    best = tmax.clone()
    u_, v_ = torch.zeros_like(best), torch.zeros_like(best)
    step = max(1, (1 << 25) // T)
    for a in range(0, n, step):
        s = slice(a, min(n, a + step))
        ro, rd = [o[s, k, None] for k in range(3)], [d[s, k, None] for k in range(3)]
        A, B, P = ([m[None, :, k] for k in range(3)] for m in (e1, e2, p1))
        pv = [rd[1] * B[2] - rd[2] * B[1], rd[2] * B[0] - rd[0] * B[2], rd[0] * B[1] - rd[1] * B[0]]
        inv = 1.0 / (A[0] * pv[0] + A[1] * pv[1] + A[2] * pv[2])
        tv = [ro[k] - P[k] for k in range(3)]
        u = (tv[0] * pv[0] + tv[1] * pv[1] + tv[2] * pv[2]) * inv
        del pv
        qv = [tv[1] * A[2] - tv[2] * A[1], tv[2] * A[0] - tv[0] * A[2], tv[0] * A[1] - tv[1] * A[0]]
        v = (rd[0] * qv[0] + rd[1] * qv[1] + rd[2] * qv[2]) * inv
        t = (B[0] * qv[0] + B[1] * qv[1] + B[2] * qv[2]) * inv
        ok = (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= tmin[s, None]) & (t <= tmax[s, None])
        t, j = torch.where(ok, t, math.inf).min(1)
        hit = torch.isfinite(t)
        idx[s] = torch.where(hit, j, -1)
        best[s] = torch.where(hit, t, best[s])
        u_[s] = torch.where(hit, u.gather(1, j[:, None])[:, 0], 0.0)
        v_[s] = torch.where(hit, v.gather(1, j[:, None])[:, 0], 0.0)
    return (idx >= 0) if any_hit else (idx, best, u_, v_)


def _exact_hits(case, seed):
    pos, faces = _soup(case, seed)
    p = torch.from_numpy(pos[faces.astype(np.int64)]).to(DEV).double()
    r = {k: v.double() for k, v in _device_rays(case, seed).items()}
    o, d = torch.stack([r["ox"], r["oy"], r["oz"]], 1), torch.stack([r["dx"], r["dy"], r["dz"]], 1)
    tri = (p[:, 0], p[:, 1] - p[:, 0], p[:, 2] - p[:, 0])
    if case["kind"] == "visible":
        return _nearest(*tri, o, d, r["tmin"], r["tmax"], any_hit=True).to(torch.uint8)
    idx, t, u, v = _nearest(*tri, o, d, r["tmin"], r["tmax"])
    out = {"tri_id": idx.to(torch.int32), "t": torch.where(idx >= 0, t, 0.0), "u": u, "v": v}
    return {k: x.cpu().numpy() for k, x in out.items()} if case["kind"] == "host" else out


_GOLDEN = 0x9E3779B97F4A7C15


def _i64(x):
    x &= (1 << 64) - 1
    return x - (1 << 64) if x >> 63 else x


def _mix(x):
    """The SplitMix64 finaliser on int64 tensors (wrapping products, logical shifts)."""
    for shift, mul in ((30, 0xBF58476D1CE4E5B9), (27, 0x94D049BB133111EB), (31, None)):
        x = x ^ ((x >> shift) & ((1 << (64 - shift)) - 1))
        if mul is not None:
            x = x * _i64(mul)
    return x


def _dot(a, b):
    return (a * b).sum(-1, keepdim=True)


def _unit(a):
    return a / a.norm(dim=-1, keepdim=True)


class _PathTracer:
    """The path tracers in 64-bit torch over all triangles (no acceleration structure): one wave of all samples, each
    sample's random numbers a hash of (seed, sample, dimension). Diffuse albedos per triangle and light emissions may be
    differentiable tensors; Russian roulette and MIS weights are held at their values."""

    EPS, EPS_LARGE = 1e-4, 1e-3

    def __init__(self, prims, tech, rr, max_pv, stratified, seed, albedo=None, emission=None):
        self.tech, self.rr, self.max_pv, self.stratified, self.seed = tech, rr, max_pv, stratified, seed
        P, Nn, kind, R, light, lights = [], [], [], [], [], []
        for pr in prims.primitives:
            f = pr.mesh.faces.astype(np.int64)
            P.append(pr.mesh.positions[f])
            Nn.append(pr.mesh.normals[f])
            kind.append(np.full(len(f), pr.bsdf.kind))
            R.append(np.tile(np.asarray(pr.bsdf.reflectance, np.float32), (len(f), 1)))
            if pr.light is not None and pr.light not in lights:
                lights.append(pr.light)
            light.append(np.full(len(f), lights.index(pr.light) if pr.light is not None else -1))

        def dev(x):
            return torch.from_numpy(np.concatenate(x)).to(DEV)
        p, self.n = dev(P).double(), dev(Nn).double()
        self.p1, self.e1, self.e2 = p[:, 0].contiguous(), p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
        c = torch.cross(self.e1, self.e2, dim=1)
        self.gn, area = _unit(c), 0.5 * c.norm(dim=1)
        self.kind, self.light = dev(kind), dev(light)
        self.R = albedo if albedo is not None else dev(R).double()
        self.Le = emission if emission is not None else torch.tensor([l.luminance for l in lights], device=DEV, dtype=torch.float64)
        self.grad = (albedo, emission)
        self.tables = []
        for li in range(len(lights)):
            ids = (self.light == li).nonzero()[:, 0]
            cdf = torch.cat([torch.zeros(1, device=DEV, dtype=torch.float64), area[ids].cumsum(0)])
            self.tables.append((ids, cdf / cdf[-1], float(cdf[-1])))
        self.light_area = torch.tensor([t[2] for t in self.tables] + [math.inf], device=DEV, dtype=torch.float64)
        cam = prims.camera
        self.w, self.h = cam.film.width, cam.film.height
        eye, ctr, up = (torch.tensor(np.asarray(v, np.float32), device=DEV).double() for v in (cam.eye, cam.center, cam.up))
        self.eye, self.f = eye, _unit(ctr - eye)
        self.s = _unit(torch.linalg.cross(self.f, _unit(up)))
        self.u = torch.linalg.cross(self.s, self.f)
        self.ty = math.tan(math.radians(float(np.float32(cam.fovy))) / 2)
        self.tx = self.ty * self.w / self.h
        self.env = prims.environment_light is not None
        if self.env:
            lo = torch.minimum(p.reshape(-1, 3).amin(0), eye)
            hi = torch.maximum(p.reshape(-1, 3).amax(0), eye)
            self.env_c = (lo + hi) / 2
            self.env_r = float((self.env_c - hi).norm())
            self.env_Le = torch.tensor(prims.environment_light.luminance, device=DEV, dtype=torch.float64)
            self.env_area = 4 * math.pi * self.env_r ** 2
        self.num_lights = len(lights) + (1 if self.env else 0)

    # ---- pieces
    def rnd(self, key, dim):
        x = _mix(key ^ _i64((dim + 1) * _GOLDEN))
        return ((x >> 40) & 0xFFFFFF).double() / 16777216.0

    def importance(self, cos):
        c = torch.where((cos - 1).abs() < self.EPS_LARGE, 1.0, cos)
        return torch.where(cos > 0, 1.0 / (4 * self.tx * self.ty) / c ** 3, 0.0)

    def pixel(self, rx, ry):
        x = (rx * self.w).long().clamp(0, self.w - 1)
        y = (ry * self.h).long().clamp(0, self.h - 1)
        return y * self.w + x

    def env_hit(self, o, d, tmin, tmax):
        oc = o - self.env_c
        a, b, c = _dot(d, d)[:, 0], 2 * _dot(oc, d)[:, 0], _dot(oc, oc)[:, 0] - self.env_r ** 2
        det = b * b - 4 * a * c
        e = det.clamp(min=0).sqrt()
        t0, t1 = (-b - e) / (2 * a), (-b + e) / (2 * a)
        ok = (det >= 0) & (t0 <= tmax) & (t1 >= tmin)
        t = torch.where(t0 < tmin, t1, t0)
        return ok & (t <= tmax), t

    def visible(self, a, b):
        d = b - a
        length = d.norm(dim=1)
        d = d / length[:, None]
        tmin, tmax = torch.full_like(length, self.EPS), length * (1 - self.EPS)
        hit = _nearest(self.p1, self.e1, self.e2, a, d, tmin, tmax, any_hit=True)
        if self.env:
            hit = hit | self.env_hit(a, d, tmin, tmax)[0]
        return ~hit

    def sample_light(self, u0, u1):
        """Position, normal, area pdf (times the selection's) and light index of each sample."""
        nl = self.num_lights
        li = (u0 * nl).long().clamp(max=nl - 1)
        u0 = u0 * nl - li
        p = torch.zeros((len(u0), 3), device=DEV, dtype=torch.float64)
        nrm, pdf = torch.zeros_like(p), torch.zeros_like(u0)
        for k, (ids, cdf, area) in enumerate(self.tables):
            m = li == k
            if not m.any():
                continue
            j = (torch.searchsorted(cdf, u1[m], right=True) - 1).clamp(0, len(ids) - 1)
            v = (u1[m] - cdf[j]) / (cdf[j + 1] - cdf[j])
            sq = u0[m].clamp(min=0).sqrt()
            b0, b1 = 1 - sq, v * sq
            t = ids[j]
            p[m] = self.p1[t] + self.e1[t] * b0[:, None] + self.e2[t] * b1[:, None]
            nrm[m] = self.gn[t]
            pdf[m] = 1.0 / (area * nl)
        if self.env:
            m = li == nl - 1
            z = 1 - 2 * u0[m]
            r = (1 - z * z).clamp(min=0).sqrt()
            phi = 2 * math.pi * u1[m]
            d = torch.stack([r * phi.cos(), r * phi.sin(), z], 1)
            p[m] = self.env_c + d * self.env_r
            nrm[m] = -d
            pdf[m] = 1.0 / (self.env_area * nl)
        return p, nrm, pdf, li

    def emission(self, li):
        Le = torch.cat([self.Le, self.env_Le[None]]) if self.env else self.Le
        return Le[li]

    def geometry(self, p1, n1, deg1, p2, n2):
        d = p2 - p1
        l2 = _dot(d, d)[:, 0]
        d = d / l2.sqrt()[:, None]
        num = torch.where(deg1, 1.0, _dot(n1, d)[:, 0].abs()) * _dot(n2, d)[:, 0].abs()
        return torch.where(l2.sqrt() < self.EPS, 0.0, num / l2)

    def splat(self, film, pixel, c):
        return film.index_add(0, pixel, c)

    @staticmethod
    def hemisphere(u0, u1):
        a, b = 2 * u0 - 1, 2 * u1 - 1
        q = math.pi / 4
        r = torch.where(a > -b, torch.where(a > b, a, b), torch.where(a < b, -a, -b))
        th = torch.where(a > -b, torch.where(a > b, q * b / a, q * (2 - a / b)),
                         torch.where(a < b, q * (4 + b / a), q * (6 - a / b)))
        th = torch.where((a == 0) & (b == 0), 0.0, th)
        x, y = r * th.cos(), r * th.sin()
        return x, y, (1 - x * x - y * y).clamp(min=0).sqrt()

    # ---- the path loop
    def film(self, count):
        N = count
        sample = torch.arange(N, device=DEV, dtype=torch.int64)
        key = _mix(_mix(torch.tensor(_i64(self.seed + _GOLDEN), device=DEV)) ^ (sample * _i64(0xD1B54A32D192ED03)))
        rx, ry = self.rnd(key, 0), self.rnd(key, 1)
        if self.stratified:
            pix = sample % (self.w * self.h)
            rx, ry = (pix % self.w + rx) / self.w, (pix // self.w + ry) / self.h
        pixel = self.pixel(rx, ry)
        local = _unit(torch.stack([(2 * rx - 1) * self.tx, (2 * ry - 1) * self.ty, -torch.ones_like(rx)], 1))
        dirs = local[:, :1] * self.s + local[:, 1:2] * self.u - local[:, 2:] * self.f
        film = torch.zeros((self.w * self.h, 3), device=DEV, dtype=torch.float64)
        thr = torch.ones((N, 3), device=DEV, dtype=torch.float64)
        o, d = self.eye.expand(N, 3), _unit(dirs)
        pdf = self.importance(-local[:, 2])
        prev_n = torch.tensor([0.0, 0, 1], device=DEV, dtype=torch.float64).expand(N, 3)
        deg = torch.ones(N, dtype=torch.bool, device=DEV)
        spec = torch.zeros_like(deg)
        tmin = torch.full((N,), 0.0 if self.tech == "pt" else self.EPS, device=DEV, dtype=torch.float64)
        lum = torch.tensor([0.212671, 0.715160, 0.072169], device=DEV, dtype=torch.float64)

        def roulette(thr, v):
            p = (thr.detach() @ lum).clamp(max=0.5)
            return self.rnd(key, 8 * v + 2) <= p, thr / p[:, None]

        if self.max_pv != -1 and self.max_pv <= 1:
            N = 0
        elif self.tech != "pt":
            film = self.camera_light(film, key)
            if self.rr != -1 and self.rr <= 1:
                ok, thr = roulette(thr, 1)
                key, pixel, o, d, thr, pdf, prev_n, deg, spec, tmin = (x[ok] for x in (key, pixel, o, d, thr, pdf, prev_n, deg, spec, tmin))
        k = 1
        while len(key) and N and (self.max_pv == -1 or k < self.max_pv):
            tri, t, b0, b1 = _nearest(self.p1, self.e1, self.e2, o, d, tmin, torch.full_like(tmin, math.inf))
            wi = -d
            # emission at the hit
            surf = tri >= 0
            tj = tri.clamp(min=0)
            p = o + d * torch.where(surf, t, 0.0)[:, None]
            n = _unit((self.n[tj] * torch.stack([1 - b0 - b1, b0, b1], 1)[:, :, None]).sum(1))
            gn = self.gn[tj]
            li = torch.where(surf, self.light[tj], -1)
            larea = self.light_area[li]
            if self.env:
                eh, et = self.env_hit(o, d, tmin, torch.full_like(tmin, math.inf))
                eh = eh & ~surf
                p = torch.where(eh[:, None], o + d * et[:, None], p)
                n = torch.where(eh[:, None], _unit(self.env_c - p), n)
                li = torch.where(eh, self.num_lights - 1, li)
                larea = torch.where(eh, self.env_area, larea)
            lit = (li >= 0) & (_dot(n, wi)[:, 0] > 0)
            w = torch.ones_like(t)
            if self.tech == "pt.mis":
                G = self.geometry(o, prev_n, deg, p, n)
                pdl = torch.where(G == 0, 0.0, 1.0 / (larea * self.num_lights * G))
                w = torch.where(spec, 1.0, pdf / (pdf + pdl))
            elif self.tech == "pt.direct":
                w = spec.double()
            m = lit.nonzero()[:, 0]
            if len(m):
                film = self.splat(film, pixel[m], thr[m] * self.emission(li[m]) * w[m][:, None])
            v = k + 1
            keep = surf
            if self.tech != "pt" and self.max_pv != -1 and v >= self.max_pv:
                break
            key, pixel, thr, wi, p, n, gn, tj = (x[keep] for x in (key, pixel, thr, wi, p, n, gn, tj))
            if not len(key):
                break
            kind, R = self.kind[tj], self.R[tj]
            a = torch.where((n[:, 0].abs() > n[:, 1].abs())[:, None], torch.stack([n[:, 2], torch.zeros_like(n[:, 0]), -n[:, 0]], 1),
                            torch.stack([torch.zeros_like(n[:, 0]), n[:, 2], -n[:, 1]], 1))
            st = _unit(a)
            ss = _unit(torch.cross(st, n, dim=1))
            wiz = _dot(n, wi)[:, 0]
            front = _dot(gn, wi)[:, 0] * wiz > 0
            half = torch.where(kind == 2, 0.5, 1.0)
            if self.tech != "pt":
                lp, ln, lpdf, lli = self.sample_light(self.rnd(key, 8 * v), self.rnd(key, 8 * v + 1))
                wl = _unit(lp - p)
                lz = _dot(n, wl)[:, 0]
                G = self.geometry(p, n, torch.zeros(len(p), dtype=torch.bool, device=DEV), lp, ln)
                ok = ((kind == 0) | (kind == 2)) & (wiz > 0) & (lz > 0) & front & (_dot(gn, wl)[:, 0] * lz > 0) & (G != 0)
                ok = ok & (_dot(ln, -wl)[:, 0] > 0)
                m = ok.nonzero()[:, 0]
                if len(m):
                    m = m[self.visible(p[m], lp[m])]
                if len(m):
                    w = 1.0
                    if self.tech == "pt.mis":
                        pdl = lpdf[m] / G[m]
                        w = pdl / (pdl + half[m] / math.pi)
                    film = self.splat(film, pixel[m], thr[m] * R[m] * self.emission(lli[m]) * (w * G[m] / lpdf[m] * half[m] / math.pi)[:, None])
            kv = k if self.tech == "pt" else v
            alive = torch.ones(len(key), dtype=torch.bool, device=DEV)
            if self.tech != "pt" and self.rr != -1 and kv >= self.rr:
                alive, thr = roulette(thr, kv)
            x, y, z = self.hemisphere(self.rnd(key, 8 * kv + 3), self.rnd(key, 8 * kv + 4))
            diffuse = (kind == 0) | ((kind == 2) & (self.rnd(key, 8 * kv + 5) < 0.5))
            lx, ly = _dot(ss, wi)[:, 0], _dot(st, wi)[:, 0]
            wo = torch.stack([torch.where(diffuse, x, -lx), torch.where(diffuse, y, -ly), torch.where(diffuse, z, wiz)], 1)
            pdf = torch.where(diffuse, half / math.pi, half / wo[:, 2])
            dn = ss * wo[:, :1] + st * wo[:, 1:2] + n * wo[:, 2:]
            alive = alive & (kind != 3) & (wiz > 0) & front & (_dot(gn, dn)[:, 0] * wo[:, 2] > 0) & (R.detach() != 0).any(1)
            thr = thr * R
            if self.tech == "pt" and self.rr != -1 and k >= self.rr:
                ok, thr = roulette(thr, k)
                alive = alive & ok
            if self.tech == "pt" and self.max_pv != -1 and k + 1 >= self.max_pv:
                break
            spec, deg = ~diffuse, torch.zeros_like(diffuse)
            key, pixel, o, d, thr, pdf, prev_n, deg, spec = (x[alive] for x in (key, pixel, p, dn, thr, pdf, n, deg, spec))
            tmin = torch.full((len(key),), self.EPS, device=DEV, dtype=torch.float64)
            k += 1
        scale = self.w * self.h / count
        return film.reshape(self.h, self.w, 3) * scale, self.grad

    def camera_light(self, film, key):
        """The camera vertex's light sample, at its own raster position."""
        lp, ln, lpdf, li = self.sample_light(self.rnd(key, 8), self.rnd(key, 9))
        d = _unit(lp - self.eye)
        cx, cy, cz = (d @ self.s), (d @ self.u), -(d @ self.f)
        rx, ry = (cx / self.tx / -cz + 1) / 2, (cy / self.ty / -cz + 1) / 2
        We = self.importance(-cz)
        G = self.geometry(self.eye.expand_as(lp), ln, torch.ones(len(lp), dtype=torch.bool, device=DEV), lp, ln)
        ok = (rx >= 0) & (rx <= 1) & (ry >= 0) & (ry <= 1) & (We > 0) & (G != 0) & (_dot(ln, -d)[:, 0] > 0)
        m = ok.nonzero()[:, 0]
        if len(m):
            m = m[self.visible(self.eye.expand(len(m), 3).contiguous(), lp[m])]
        if not len(m):
            return film
        w = 1.0
        if self.tech == "pt.mis":
            pdl = lpdf[m] / G[m]
            w = pdl / (pdl + We[m])
        c = self.emission(li[m]) * (w * We[m] * G[m] / lpdf[m])[:, None]
        return self.splat(film, self.pixel(rx[m], ry[m]), c)
