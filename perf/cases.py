"""The library's performance cases: what its users have it do, over the range of sizes they do it at.

A case is a dict of plain values; ``op`` names the entry point:

* ``closest`` / ``any`` / ``closest_d`` / ``any_d`` -- ray queries on a triangle accelerator (float or double rays),
  device buffers in and out;
* ``build`` -- making an accelerator from host meshes and reading its tree back;
* ``knn`` -- filtered photon lookups;
* ``direct`` -- one direct-lighting frame (diffuse and glossy box, the sphere scene, a glass sphere with its specular
  recursion, or a participating medium);
* ``batch`` -- many views of one scene as one launch;
* ``adjoint`` -- a frame and its albedo / emission gradients through torch.autograd;
* ``photon`` -- shooting photons, building the maps and rendering a frame with them.

``listed`` gives the named cases, ``draw`` further ones of the same ranges, ``prepare`` what a program holds before
the call, ``run`` the call, ``work`` the bytes it cannot do without and ``exact`` the answer in 64 bits by brute force
where that is affordable.
"""
from __future__ import annotations

import dataclasses
import functools
import math

import numpy as np
import torch

from skwarka_gb300 import scenes
from skwarka_gb300.accel import Primitive, TriangleAccelerator, TriangleMesh
from skwarka_gb300.adjoint import DirectLighting
from skwarka_gb300.kdtree import PhotonKDTree, compress_directions
from skwarka_gb300.photon import PhotonMap, render_photon
from skwarka_gb300.render import (LD, METAL, PLASTIC, STRATIFIED, TRANSPARENT, Camera, Material, Medium, PointLight,
                                  RenderBatch, RenderPrimitive, RenderScene)

RAY_OPS = ("closest", "any", "closest_d", "any_d")
RAY_BYTES, HIT_BYTES = {"closest": 32, "any": 32, "closest_d": 64, "any_d": 64}, \
    {"closest": 16, "any": 1, "closest_d": 16, "any_d": 1}


def listed():
    return [
        # A picking / probing program: a thousand rays at a time on a scene of some 18,000 triangles.  Latency counts.
        {"name": "closest small", "op": "closest", "level": 6, "scatter": 2000, "rays": 1000},
        # The ray-query benchmark: 4M incoherent rays on the 1.1M-triangle scene.
        {"name": "closest large", "op": "closest", "level": 9, "scatter": 50000, "rays": 4194304},
        # Shadow / visibility queries on the same scene, a ragged count.
        {"name": "any hit", "op": "any", "level": 9, "scatter": 50000, "rays": 2000003},
        # The reference's own integrators over the drop-in accelerator: batches of double rays, exact t.
        {"name": "closest double", "op": "closest_d", "level": 9, "scatter": 50000, "rays": 200001},
        # Loading a scene: the 1.1M-triangle accelerator from host meshes.
        {"name": "accelerator build", "op": "build", "level": 9, "scatter": 50000},
        # Photon-map lookups at the primary hits of a 512 x 512 frame at 4 samples a pixel.
        {"name": "photon lookup", "op": "knn", "photons": 275764, "side": 512, "spp": 4, "k": 100, "radius": 0.05,
         "filter": True},
        # The plain direct-lighting frame of the GUI's preview: 256 x 256, 2 x 2 strata, 20,480 triangles.
        {"name": "direct frame", "op": "direct", "scene": "box", "width": 256, "height": 256, "spp_x": 2, "spp_y": 2,
         "sampler": STRATIFIED},
        # A glass object: specular trees of depth 6, an uneven film, the GUI's LD sampler.
        {"name": "glass frame", "op": "direct", "scene": "glass", "width": 301, "height": 211, "spp_x": 2, "spp_y": 2,
         "sampler": LD},
        # Fog: the ray march through a homogeneous medium in the 200k-triangle scene.
        {"name": "medium frame", "op": "direct", "scene": "medium", "width": 200, "height": 150, "spp_x": 2,
         "spp_y": 2, "sampler": STRATIFIED},
        # Data-set rendering: views of uneven size of the 200k-triangle scene in one launch, 8 samples a pixel.
        {"name": "view batch", "op": "batch", "views": 16, "lo": 64, "hi": 1024, "spp_x": 4, "spp_y": 2},
        # Inverse rendering: a 512 x 512 frame at 16 samples a pixel and its gradients.
        {"name": "adjoint", "op": "adjoint", "width": 512, "height": 512, "spp_x": 4, "spp_y": 4},
        # Photon mapping on the 1.1M-triangle scene: 2M paths, the maps, a 512 x 512 frame with final gathering.
        {"name": "photon mapping", "op": "photon", "level": 9, "scatter": 50000, "paths": 2000000, "width": 512,
         "height": 512, "spp_x": 2, "spp_y": 2, "gather": 16},
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    op = rng.choice(("closest", "any", "closest_d", "any_d", "build", "knn", "box", "spheres", "glass", "medium", "batch",
                     "adjoint", "photon"))
    if op in RAY_OPS:
        most = 4000000 if op in ("closest", "any") else 200000
        return {"op": op, "level": rng.randint(4, 9), "scatter": _log(rng, 100, 50000), "rays": _log(rng, 500, most)}
    if op == "build":
        return {"op": op, "level": rng.randint(5, 9), "scatter": _log(rng, 100, 50000)}
    if op == "knn":
        return {"op": op, "photons": _log(rng, 2000, 275000), "side": _log(rng, 32, 512), "spp": rng.randint(1, 4),
                "k": _log(rng, 8, 200), "radius": round(rng.uniform(0.03, 0.1), 4), "filter": rng.random() < 0.8}
    if op in ("box", "spheres", "glass", "medium"):
        hi = {"box": 640, "spheres": 640, "glass": 320, "medium": 200}[op]
        return {"op": "direct", "scene": op, "width": _log(rng, 24, hi), "height": _log(rng, 24, hi),
                "spp_x": rng.randint(1, 3), "spp_y": rng.randint(1, 2), "sampler": rng.choice((STRATIFIED, LD))}
    if op == "batch":
        return {"op": op, "views": rng.randint(2, 16), "lo": 64, "hi": _log(rng, 128, 1024), "spp_x": rng.randint(1, 4),
                "spp_y": rng.randint(1, 2)}
    if op == "adjoint":
        return {"op": op, "width": _log(rng, 32, 512), "height": _log(rng, 32, 512), "spp_x": rng.randint(1, 4),
                "spp_y": rng.randint(1, 4)}
    return {"op": op, "level": rng.randint(5, 9), "scatter": _log(rng, 100, 50000), "paths": _log(rng, 50000, 2000000),
            "width": _log(rng, 64, 512), "height": _log(rng, 64, 512), "spp_x": rng.randint(1, 2),
            "spp_y": rng.randint(1, 2), "gather": rng.choice((4, 9, 16))}


# ---------------------------------------------------------------- inputs --

@functools.lru_cache(maxsize=None)
def _unit_sphere(level):
    v, t = scenes.sphere_mesh(level)
    return v, t


class _Surface:
    """A unit sphere pushed in and out along its radius by a seeded sum of waves (up to 5 %)."""

    def __init__(self, seed):
        rng = np.random.default_rng([seed, 1])
        self.wave = torch.as_tensor(rng.normal(size=(12, 3)) * 5.0, device="cuda")
        self.phase = torch.as_tensor(rng.uniform(0.0, 2.0 * np.pi, size=12), device="cuda")
        self.height = 0.05 / 12 ** 0.5

    def radius(self, d):
        return 1.0 + self.height * torch.sin(d @ self.wave.T + self.phase).sum(1)

    def points(self, d):
        return d * self.radius(d)[:, None]

    def normals(self, d):
        # of the level set |x| - r(x / |x|)
        g = self.height * torch.cos(d @ self.wave.T + self.phase) @ self.wave
        g = (g - (g * d).sum(1, keepdim=True) * d) / self.radius(d)[:, None]
        n = d - g
        return n / n.norm(dim=1, keepdim=True)


def _meshes(case, seed):
    v, t = _unit_sphere(case["level"])
    p = _Surface(seed).points(torch.as_tensor(v, device="cuda")).float().cpu().numpy()
    return [(p, t), scenes.random_triangles(case["scatter"], 0.01, 0.0, 1.0, seed)]


def _uniform_rays(case, meshes, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    lo, hi = (torch.as_tensor(b, device="cuda") for b in scenes.scene_bounds(meshes))
    n = case["rays"]
    r = torch.zeros((n, 8), dtype=torch.float64, device="cuda")
    r[:, 0:3] = lo + (hi - lo) * torch.rand((n, 3), generator=g, dtype=torch.float64, device="cuda")
    d = torch.randn((n, 3), generator=g, dtype=torch.float64, device="cuda")
    r[:, 3:6] = d / d.norm(dim=1, keepdim=True)
    if case["op"].startswith("any"):
        r[:, 7] = 2.0 * torch.rand(n, generator=g, dtype=torch.float64, device="cuda")
    else:
        r[:, 7] = float("inf")
    return r if case["op"].endswith("_d") else r.float()


def _frame(axis):
    """Two directions that make an orthonormal frame with `axis`."""
    a = np.asarray(axis, np.float64)
    a = a / np.linalg.norm(a)
    u = np.cross(a, (0.0, 0.0, 1.0) if abs(a[2]) < 0.9 else (1.0, 0.0, 0.0))
    u /= np.linalg.norm(u)
    return torch.as_tensor(np.stack([u, np.cross(a, u), a]), device="cuda")


def _lift(uv, frame):
    """Points of the unit disc to directions of the hemisphere around frame[2] (parallel projection)."""
    z = torch.sqrt(torch.clamp(1.0 - (uv * uv).sum(1), min=0.0))
    return torch.cat([uv, z[:, None]], 1) @ frame


def _photon_inputs(case, seed):
    """Photons a distant light leaves on the waved sphere, and a camera's primary hits in pixel order."""
    rng = np.random.default_rng([seed, 2])
    g = torch.Generator(device="cuda").manual_seed(seed)
    s = _Surface(seed)
    cam = rng.normal(size=3)
    light = cam / np.linalg.norm(cam) + 0.7 * rng.normal(size=3)
    n = case["photons"]
    r = torch.sqrt(torch.rand(n, generator=g, dtype=torch.float64, device="cuda"))
    a = 2.0 * math.pi * torch.rand(n, generator=g, dtype=torch.float64, device="cuda")
    d = _lift(torch.stack([r * torch.cos(a), r * torch.sin(a)], 1), _frame(light))
    pos = s.points(d).float().cpu().numpy()
    nid = compress_directions(s.normals(d).cpu().numpy())
    side, spp = case["side"], case["spp"]
    y, x, j = torch.meshgrid(torch.arange(side, device="cuda"), torch.arange(side, device="cuda"),
                             torch.arange(spp, device="cuda"), indexing="ij")
    pixel = 2.2 / side
    corner = torch.stack([x.reshape(-1), y.reshape(-1)], 1).double() * pixel - 1.1
    corner = corner[(corner + 0.5 * pixel).norm(dim=1) + 0.71 * pixel < 0.995]  # pixels that lie on the sphere
    qd = _lift(corner + pixel * torch.rand(corner.shape, generator=g, dtype=torch.float64, device="cuda"), _frame(cam))
    return pos, nid, s.points(qd).contiguous(), s.normals(qd).contiguous()


def _sphere_scene(seed):
    """A box with 32 spheres of mixed materials (201,742 triangles) and a quad light."""
    rng = np.random.default_rng([seed, 3])
    bv, bt = scenes._box_inward()
    wall = rng.uniform(0.2, 0.8, size=(6, 3)).astype(np.float32)
    mats = [Material(kd=(0.5, 0.5, 0.5)), Material(kd=(0.0, 0.0, 0.0)), Material(kd=(0.7, 0.5, 0.3)),
            Material(kind=PLASTIC, kd=(0.3, 0.4, 0.6), ks=(0.4, 0.4, 0.4), roughness=0.15),
            Material(kind=METAL, eta=(0.2, 0.9, 1.1), k=(3.9, 2.4, 2.2), roughness=0.2)]
    prims = [RenderPrimitive(TriangleMesh(bv, bt), 0, triangle_albedo=np.repeat(wall, 2, axis=0))]
    for level in (6,) * 12 + (3,) * 20:
        v, t = _unit_sphere(level)
        r = rng.uniform(0.05, 0.2) * (1.0 + rng.uniform(-0.01, 0.01, size=(len(v), 1)))
        p = (v * r + rng.uniform(-0.75, 0.75, size=3)).astype(np.float32)
        prims.append(RenderPrimitive(TriangleMesh(p, t), int(rng.integers(2, 5)), vertex_normals=v.astype(np.float32)))
    lv = np.array([[-0.3, 0.98, -0.3], [0.3, 0.98, -0.3], [0.3, 0.98, 0.3], [-0.3, 0.98, 0.3]], np.float32)
    prims.append(RenderPrimitive(TriangleMesh(lv, np.array([[0, 1, 2], [0, 2, 3]], np.int32)), 1,
                                 emission=(10.0, 10.0, 10.0)))
    return prims, mats


def _inside_camera(width, height):
    return Camera.look_at((0.0, 0.3, -0.9), (0.0, -0.4, 0.6), (0, 1, 0), math.radians(70.0), width, height)


def _direct_scene(case, seed):
    w, h = case["width"], case["height"]
    rng = np.random.default_rng([seed, 4])
    if case["scene"] == "box":
        prims, mats, camera = scenes.direct_lighting_box(seed % (1 << 31))
        return RenderScene(prims, mats), camera(w, h)
    if case["scene"] == "glass":
        tint = tuple(float(x) for x in rng.uniform(0.8, 1.0, size=3))
        glass = Material(kind=TRANSPARENT, kd=(1.0, 1.0, 1.0), ks=tint, refractive_index=1.5)
        prims, mats, lights, camera = scenes.glass_sphere_scene(glass, "area", (w, h))
        scene = RenderScene(prims, mats, lights)
        scene.set_max_specular_depth(6)
        return scene, camera
    scene = RenderScene(*_sphere_scene(seed))
    if case["scene"] == "medium":
        scene.set_medium(Medium(sigma_a=(0.05,) * 3, sigma_s=(0.2,) * 3, g=0.3, step=0.05))
    return scene, _inside_camera(w, h)


def prepare(case, seed):
    op = case["op"]
    state = {"op": op, "case": case, "seed": seed}
    if op in RAY_OPS or op == "build":
        meshes = _meshes(case, seed)
        prims = [Primitive(TriangleMesh(v, t)) for v, t in meshes]
        if op == "build":
            # the tree's size depends on the input: room for it, the rest stays zero
            return {**state, "prims": prims, "nodes": np.zeros((_triangles(case), 8), np.int32)}
        return {**state, "accel": TriangleAccelerator(prims), "rays": _uniform_rays(case, meshes, seed)}
    if op == "knn":
        pos, nid, q, qn = _photon_inputs(case, seed)
        return {**state, "tree": PhotonKDTree(pos, nid), "q": q, "qn": qn if case["filter"] else None}
    if op == "direct":
        scene, camera = _direct_scene(case, seed)
        return {**state, "scene": scene, "camera": camera}
    if op == "batch":
        scene = RenderScene(*_sphere_scene(seed))
        sides = [c.width for c in scenes.batching_views(case["views"], 5, case["lo"], case["hi"])]
        cameras = [dataclasses.replace(c, width=n, height=n)
                   for c, n in zip(scenes.batching_views(case["views"], seed % (1 << 31)), sides)]
        batch = RenderBatch(scene, cameras, case["spp_x"], case["spp_y"], 1, seed)
        return {**state, "batch": batch, "films": batch.new_films()}
    if op == "adjoint":
        scene = RenderScene(*_sphere_scene(seed))
        w, h = case["width"], case["height"]
        render = DirectLighting(scene, _inside_camera(w, h), case["spp_x"], case["spp_y"], 1, seed)
        g = torch.Generator(device="cuda").manual_seed(seed)
        albedo = 0.1 + 0.8 * torch.rand((scene.n_triangles, 3), generator=g, device="cuda")
        return {**state, "render": render, "albedo": albedo.requires_grad_(),
                "scale": torch.ones((), device="cuda", requires_grad=True),
                "target": torch.rand((h, w, 3), generator=g, device="cuda")}
    rng = np.random.default_rng([seed, 5])
    prims = [RenderPrimitive(TriangleMesh(v, t), 0) for v, t in _meshes(case, seed)]
    light = PointLight(tuple(float(x) for x in np.array((1.2, 0.9, 0.7)) + rng.uniform(-0.1, 0.1, size=3)), (50.0,) * 3)
    camera = Camera.look_at((2.2, 1.8, 1.6), (0.0, 0.0, 0.0), (0.0, 0.0, 1.0), math.radians(38.0), case["width"],
                            case["height"])
    return {**state, "scene": RenderScene(prims, [Material(kd=(0.6, 0.6, 0.6))], [light]), "camera": camera}


# ------------------------------------------------------------------ calls --

def run(state):
    op, case = state["op"], state["case"]
    if op == "closest":
        hits = state["accel"].intersect(state["rays"])
        return {"t": hits[:, 0].view(torch.float32), "prim": hits[:, 1], "tri": hits[:, 2], "flags": hits[:, 3]}
    if op == "closest_d":
        hits = state["accel"].intersect_d(state["rays"])
        ids = hits.view(torch.int32)
        return {"t": hits[:, 0], "prim": ids[:, 2], "tri": ids[:, 3]}
    if op == "any":
        return {"occluded": state["accel"].intersect_test(state["rays"])}
    if op == "any_d":
        return {"occluded": state["accel"].intersect_test_d(state["rays"])}
    if op == "build":
        nodes, prim, tri = TriangleAccelerator(state["prims"]).export()
        state["nodes"][:len(nodes)] = nodes.view(np.int32)
        return {"nodes": state["nodes"], "prim": prim, "tri": tri}
    if op == "knn":
        cos = math.cos(math.radians(30.0)) if case["filter"] else -1.0
        return state["tree"].get_nearest_points(state["q"], state["qn"], case["k"], case["radius"], cos)
    if op == "direct":
        return {"film": state["scene"].render_direct(state["camera"], case["spp_x"], case["spp_y"], 1, state["seed"],
                                                     sampler=case["sampler"])}
    if op == "batch":
        return {"films": state["batch"].run(state["films"])}
    if op == "adjoint":
        image = state["render"](state["albedo"], state["scale"])
        loss = ((image - state["target"]) ** 2).sum()
        g_albedo, g_scale = torch.autograd.grad(loss, (state["albedo"], state["scale"]))
        return {"image": image.detach(), "g_albedo": g_albedo, "g_scale": g_scale}
    maps = PhotonMap.shoot(state["scene"], case["paths"], max_bounces=8, rr_probability=0.7, seed=state["seed"])
    info = maps.info()
    film = render_photon(state["scene"], maps, state["camera"], case["spp_x"], case["spp_y"],
                         gather_samples=case["gather"], seed=state["seed"])
    return {"film": film, "direct": info["n_direct"], "indirect": info["n_indirect"],
            "irradiance": info["n_irradiance"]}


def _triangles(case):
    return 4 * 4 ** case["level"] + case["scatter"]


def work(case):
    """Inputs read once and outputs written once.  A triangle is 9 floats (36 bytes); a render's inputs are its
    triangles, its output the film (and the gradients).  No operations are counted: how many boxes and triangles a ray
    has to be tested against depends on the tree."""
    op = case["op"]
    if op in RAY_OPS:
        return {"bytes": 36 * _triangles(case) + case["rays"] * (RAY_BYTES[op] + HIT_BYTES[op]), "flops": 0}
    if op == "build":
        # 12 bytes of indices and about half a vertex per triangle in; 32-byte nodes and 8 bytes of ids out
        return {"bytes": _triangles(case) * (12 + 6 + 32 * 0.57 + 8), "flops": 0}
    if op == "knn":
        queries = case["side"] ** 2 * case["spp"] * math.pi / 4.84
        return {"bytes": 18 * case["photons"] + queries * (24 + (24 if case["filter"] else 0) + 4 + 12 * case["k"]),
                "flops": 0}
    tris = {"box": 20494, "glass": 1028}.get(case.get("scene"), 201742)
    if op == "direct":
        return {"bytes": 36 * tris + 12 * case["width"] * case["height"], "flops": 0}
    if op == "batch":
        lo, hi = case["lo"], case["hi"]
        pixels = case["views"] * (hi * hi - lo * lo) / (2.0 * math.log(hi / lo))
        return {"bytes": 36 * tris + 12 * pixels, "flops": 0}
    if op == "adjoint":
        # albedo and its gradient, the image, its target and dL/dI
        return {"bytes": (36 + 24) * tris + 36 * case["width"] * case["height"], "flops": 0}
    return {"bytes": 36 * _triangles(case) + 28 * 0.17 * case["paths"] + 12 * case["width"] * case["height"], "flops": 0}


# ------------------------------------------------------- 64-bit answers --

def _closest_exact(case, seed):
    """Closest-hit t of every ray by brute force (Moller-Trumbore over all triangles in double)."""
    meshes = _meshes(case, seed)
    rays = _uniform_rays(case, meshes, seed).double()
    o, d, tmax = rays[:, 0:3], rays[:, 3:6], rays[:, 7]
    corners = torch.cat([torch.as_tensor(v[t.reshape(-1)], device="cuda").double().reshape(-1, 3, 3)
                         for v, t in meshes])
    best = torch.full((len(rays),), float("inf"), dtype=torch.float64, device="cuda")
    step = max(1, (1 << 26) // len(rays))
    for i in range(0, len(corners), step):
        v0, v1, v2 = corners[i:i + step].unbind(1)
        e1, e2 = v1 - v0, v2 - v0
        s1 = torch.linalg.cross(d[:, None], e2[None], dim=2)
        inv = 1.0 / (s1 * e1).sum(2)
        to = o[:, None] - v0
        b1 = (to * s1).sum(2) * inv
        s2 = torch.linalg.cross(to, e1[None].expand_as(to), dim=2)
        b2 = (d[:, None] * s2).sum(2) * inv
        t = (e2 * s2).sum(2) * inv
        eps = 2.220446049250313e-16
        hit = (b1 > -eps) & (b2 > -eps) & (b1 + b2 < 1.0 + eps) & (t >= 0.0) & (t <= tmax[:, None])
        best = torch.minimum(best, torch.where(hit, t, float("inf")).amin(1))
    return best


def exact(case, seed):
    if case["op"] in ("closest", "closest_d") and _triangles(case) * case["rays"] <= 4e9:
        return {"t": _closest_exact(case, seed), "prim": None, "tri": None, "flags": None}
    # any-hit and build answers are whole numbers, a lookup's distances lie in its heap's order, and a render's film
    # is a sum over the renderer's own random samples
    return None
