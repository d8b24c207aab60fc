"""The work a program has this renderer do, as measurable cases.

A case is a dict of plain values; ``prepare`` makes what a program holds before the call
(scene on the GPU, ray and film buffers), ``run`` makes one pass through the public entry
points (``GpuScene``, ``GpuBatch``, ``film``), and ``work`` says what that pass cannot do
without.  Kinds of cases:

  trace     ray queries (``GpuScene.trace`` / ``trace_device``): picking and ambient-occlusion
            or light-map baking, closest hit and occlusion
  frame     one frame of a resident scene (``GpuScene.render``): path tracer, Whitted ray
            tracer, BDPT
  oneshot   a scene that changed: upload, BVH build, one frame, 8-bit image
  batch     many scenes as one frame (``GpuBatch.render``), replayed
  optimise  one step of inverse rendering: parameter update, forward, backward

Scenes are the seeded builders of ``rumi_b200.scenes``.  The seed moves the mesh, its
colours, the rays and the random numbers of a frame, never a size.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rumi-renderer_b200"))

import rumi_b200  # noqa: E402
from rumi_b200 import film as film_io  # noqa: E402
from rumi_b200 import scenes  # noqa: E402
from rumi_b200.scene import (Film, Matte, Model, PathTracer, BidirectionalPathTracer, RayTracer, Scene)  # noqa: E402


def listed():
    return [
        # a click in a viewport: a handful of camera rays from host memory
        dict(name="trace_pick", kind="trace", rays="camera", n=61, levels=0, anyhit=False, device=False),
        # ambient occlusion / light-map baking over a large mesh: incoherent closest hits
        dict(name="trace_bake", kind="trace", rays="diffuse", n=2000003, levels=9, anyhit=False, device=True),
        # visibility of a light from the points of a mid-size mesh
        dict(name="trace_shadow", kind="trace", rays="shadow", n=500009, levels=7, anyhit=True, device=True),
        # interactive preview: a small frame, few samples, short paths, film to the host
        dict(name="frame_preview", kind="frame", scene="cornell", levels=0, width=67, height=51, spp=4, depth=4,
             integrator="pt", device=False),
        # the reference's own case: analytic Cornell box, film to the host
        dict(name="frame_cornell", kind="frame", scene="cornell", levels=0, width=256, height=256, spp=16, depth=8,
             integrator="pt", device=False),
        # the largest frame: a million triangles, 64 spp, ten bounces
        dict(name="frame_mesh", kind="frame", scene="mesh", levels=9, width=1024, height=1024, spp=64, depth=10,
             integrator="pt", device=True),
        # participating medium, glass and a spot light
        dict(name="frame_medium", kind="frame", scene="caustic", levels=0, width=333, height=251, spp=25, depth=9,
             integrator="pt", device=True),
        # the ray tracer over mirror and coloured glass
        dict(name="frame_whitted", kind="frame", scene="glass", levels=0, width=640, height=480, spp=9, depth=10,
             integrator="whitted", device=False),
        # bidirectional path tracing of the volumetric caustic
        dict(name="frame_bdpt", kind="frame", scene="caustic", levels=0, width=256, height=255, spp=8, depth=6,
             integrator="bdpt", device=True),
        # a deforming mesh: every frame uploads it, builds its BVH, renders and tonemaps
        dict(name="oneshot_mesh", kind="oneshot", levels=8, width=512, height=384, spp=8, depth=5),
        # many uneven scenes in one frame (data generation), replayed from its graph
        dict(name="batch_uneven", kind="batch", scenes=24, tris=20000, res=128, spp=8, depth=8),
        # inverse rendering: one optimisation step over albedo and medium
        dict(name="optimise_step", kind="optimise", levels=7, width=256, height=256, spp=16, depth=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["trace", "trace", "frame", "frame", "frame", "oneshot", "batch", "optimise"])
    if kind == "trace":
        levels = rng.randint(0, 8)
        rays = rng.choice(["camera", "diffuse", "shadow"])
        device = rng.random() < 0.7
        return dict(kind=kind, rays=rays, n=_log(rng, 33, 2000000 if device else 60000), levels=levels,
                    anyhit=rays == "shadow", device=device)
    if kind == "frame":
        scene = rng.choice(["cornell", "mesh", "mesh", "caustic", "glass", "dof", "subsurface", "two_lights"])
        integrator = rng.choice(["pt", "pt", "pt", "whitted", "bdpt"])
        bdpt = integrator == "bdpt"
        depth = rng.randint(3, 6) if bdpt else rng.randint(2, 10)
        spp = rng.choice([1, 4, 7, 16]) if bdpt else rng.choice([1, 4, 9, 16, 23, 64])
        pixels = _log(rng, 2000, (500000 if bdpt else 16000000) // spp)
        width = max(16, int(math.sqrt(pixels * rng.uniform(0.6, 1.9))))
        return dict(kind=kind, scene=scene, levels=rng.randint(4, 8) if scene == "mesh" else 0, width=width,
                    height=max(16, pixels // width), spp=spp, depth=depth, integrator=integrator,
                    device=rng.random() < 0.5)
    if kind == "oneshot":
        return dict(kind=kind, levels=rng.randint(4, 8), width=_log(rng, 64, 600), height=_log(rng, 64, 600),
                    spp=rng.choice([1, 4, 9]), depth=rng.randint(2, 8))
    if kind == "batch":
        return dict(kind=kind, scenes=rng.randint(3, 30), tris=_log(rng, 1000, 30000), res=_log(rng, 32, 200),
                    spp=rng.choice([2, 4, 8]), depth=rng.randint(3, 8))
    return dict(kind=kind, levels=rng.randint(3, 7), width=_log(rng, 48, 400), height=_log(rng, 48, 400),
                spp=rng.choice([4, 9, 16]), depth=rng.randint(3, 8))


# ------------------------------------------------------------------------------ scenes
@functools.lru_cache(maxsize=2)
def _topology(levels):
    return scenes.subdivided_tetrahedron(levels)


def _mesh(levels, seed):
    """``scenes.displaced_sphere`` in the box, its connectivity made once per process."""
    verts, faces = _topology(levels)
    disp = scenes.fbm((verts * np.float32(4.0)).astype(np.float32), seed % 100003)
    r = np.float32(0.25) + np.float32(0.05) * disp
    pos = (verts * r[:, None] + np.array([0.5, 0.35, 0.5], np.float32)).astype(np.float32)
    return np.ascontiguousarray(pos[faces])


def _mesh_scene(levels, seed, width, height, spp, depth):
    """The Cornell box holding the displaced sphere, a colour per triangle."""
    sc = Scene()
    scenes.add_cornell_box(sc)
    tris = _mesh(levels, seed)
    sc.add(Model(tris, albedo=scenes.random_albedo(tris.shape[0], seed + 1)), Matte(1.0, scenes.WHITE))
    sc.camera = scenes.cornell_camera()
    sc.image = Film(width, height, spp)
    sc.tracer = PathTracer(depth)
    return sc


def _frame_scene(c, seed):
    w, h, spp, depth = c["width"], c["height"], c["spp"], c["depth"]
    name = c["scene"]
    if name == "mesh":
        sc = _mesh_scene(c["levels"], seed, w, h, spp, depth)
    elif name == "cornell":
        sc = scenes.cornell_pt(w, h, spp, depth)
    elif name == "dof":
        sc = scenes.cornell_dof_pt(w, h, spp, depth)
    elif name == "glass":
        sc = scenes.absorbing_glass_cornell(w, h, spp, depth)
    elif name == "subsurface":
        sc = scenes.subsurface_cornell(w, h, spp, depth)
    elif name == "two_lights":
        sc = scenes.cornell_two_lights_pt(w, h, spp, depth)
    else:
        sc = scenes.volumetric_caustic(w, h, spp, 6, 7)
    if c["integrator"] == "pt":
        sc.tracer = PathTracer(depth)
    elif c["integrator"] == "whitted":
        sc.tracer = RayTracer(depth)
    else:
        sc.tracer = BidirectionalPathTracer(depth, depth + 1)
    return sc


def _trace_scene(c, seed):
    if c["levels"] == 0:
        return scenes.cornell_pt(64, 64, 1, 1)
    return _mesh_scene(c["levels"], seed, 64, 64, 1, 1)


def _rays(c, flat, seed):
    """(n, 7) float32 o, d, tmax on the host: through the pixels of the camera, or from
    points of the scene's triangles in their order, cosine-distributed about the normal
    (diffuse) or toward points of the light (shadow)."""
    rng = np.random.Generator(np.random.PCG64(seed))
    n = c["n"]
    r = np.empty((n, 7), np.float32)
    if c["rays"] == "camera":
        side = max(1, int(math.sqrt(n)))
        k = np.arange(n)
        x = (k % side + rng.random(n)) / side
        y = ((k // side) % side + rng.random(n)) / side
        f = 2.0 * math.tan(math.radians(20.0))
        d = np.stack([(x - 0.5) * f, (y - 0.5) * f, np.ones(n)], 1)
        r[:, 0:3] = np.array([0.5, 0.5, -1.4])
        r[:, 3:6] = d / np.linalg.norm(d, axis=1)[:, None]
        r[:, 6] = 3.4e38
        return r
    tri = flat.tri_vertices
    pick = np.sort(rng.integers(0, tri.shape[0], n))
    v = tri[pick].astype(np.float64)
    e1, e2 = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    nrm = np.cross(e1, e2)
    nrm /= np.maximum(np.linalg.norm(nrm, axis=1), 1e-30)[:, None]
    su = np.sqrt(rng.random(n))
    b = rng.random(n) * su
    p = v[:, 0] + (1.0 - su)[:, None] * e1 + b[:, None] * e2
    centre = np.where(pick < 10, 0, 1)[:, None] * np.array([0.0, -0.15, 0.0]) + 0.5  # walls face the box, the mesh outward
    out = np.where(pick < 10, 1.0, -1.0) * np.einsum("ij,ij->i", centre - p, nrm)
    nrm *= np.where(out < 0.0, -1.0, 1.0)[:, None]
    r[:, 0:3] = p + 2e-4 * nrm
    if c["rays"] == "diffuse":
        d = rng.standard_normal((n, 3))
        d = d / np.linalg.norm(d, axis=1)[:, None] + nrm
        r[:, 3:6] = d / np.maximum(np.linalg.norm(d, axis=1), 1e-30)[:, None]
        r[:, 6] = 3.4e38
    else:
        to = np.array([0.375, 0.999, 0.375]) + rng.random((n, 3)) * np.array([0.25, 0.0, 0.25]) - r[:, 0:3]
        dist = np.linalg.norm(to, axis=1)
        r[:, 3:6] = to / dist[:, None]
        r[:, 6] = dist
    return r


# --------------------------------------------------------------------------- the passes
def prepare(case, seed):
    c, kind = dict(case), case["kind"]
    st = {"case": c, "seed": seed + 1}
    if kind == "trace":
        st["gpu"] = rumi_b200.GpuScene(_trace_scene(c, seed))
        rays = _rays(c, st["gpu"].flat, seed)
        if c["device"]:
            packed = np.zeros((c["n"], 8), np.float32)
            packed[:, 0:3], packed[:, 4:8] = rays[:, 0:3], rays[:, 3:7]
            st["rays"] = torch.from_numpy(packed).cuda()
            st["t"] = torch.zeros(c["n"], dtype=torch.float32, device="cuda")
            st["prim"] = torch.zeros(c["n"], dtype=torch.int32, device="cuda")
        else:
            st["rays"] = rays
    elif kind == "frame":
        st["gpu"] = rumi_b200.GpuScene(_frame_scene(c, seed))
        if c["device"]:
            st["film"] = torch.zeros((c["height"], c["width"], 3), dtype=torch.float32, device="cuda")
    elif kind == "oneshot":
        # the mesh of this frame, flattened as a program with its own scene graph holds it
        st["flat"] = _mesh_scene(c["levels"], seed, c["width"], c["height"], c["spp"], c["depth"]).flatten()
    elif kind == "batch":
        gpu = []
        for i in range(c["scenes"]):  # sizes go by the place in the batch, the content by the seed
            up = 2.0 ** ((i * 5) % 7 - 3)
            gpu.append(rumi_b200.GpuScene(scenes.batch_scene(
                (seed + 131 * i) % 1000003, max_depth=c["depth"], res=max(16, int(c["res"] * math.sqrt(up))),
                spp=c["spp"] * (1 + i % 3), n_tris=max(200, int(c["tris"] * up)))))
        st["batch"] = rumi_b200.GpuBatch(gpu)
        st["spp"] = [c["spp"] * (1 + i % 3) for i in range(c["scenes"])]
        st["seeds"] = [seed + 7 * i + 1 for i in range(c["scenes"])]
        st["films"] = torch.zeros(st["batch"].n_floats, dtype=torch.float32, device="cuda")
    else:
        sc = scenes.inverse_rendering(c["width"], c["height"], c["spp"], c["depth"], levels=c["levels"],
                                      albedo_seed=seed % 100003, medium=scenes.INVERSE_START_MEDIUM)
        st["gpu"] = rumi_b200.GpuScene(sc)
        rng = np.random.Generator(np.random.PCG64(seed))
        n = st["gpu"].flat.tri_vertices.shape[0]
        st["albedo"] = torch.from_numpy((0.2 + 0.6 * rng.random((n, 3))).astype(np.float32)).cuda()
        st["d_film"] = torch.from_numpy(
            (rng.standard_normal((c["height"], c["width"], 3)) * 1e-3).astype(np.float32)).cuda()
        st["film"] = torch.zeros((c["height"], c["width"], 3), dtype=torch.float32, device="cuda")
        st["g_albedo"] = torch.zeros((n, 3), dtype=torch.float32, device="cuda")
        st["g_volume"] = torch.zeros(7, dtype=torch.float32, device="cuda")
    return st


def run(state):
    c, kind = state["case"], state["case"]["kind"]
    if kind == "trace":
        # node and primitive counts are left out: they describe the tree, not the hits; so is
        # an occlusion query's distance, which is that of any of the occluders
        if c["device"]:
            state["gpu"].trace_device(c["n"], state["rays"].data_ptr(), state["t"].data_ptr(),
                                      state["prim"].data_ptr(), anyhit=c["anyhit"], count=False)
            t, prim = state["t"], state["prim"]
        else:
            t, prim = state["gpu"].trace(state["rays"], anyhit=c["anyhit"])[:2]
        return {"prim": prim} if c["anyhit"] else {"t": t, "prim": prim}
    if kind == "frame":
        if c["device"]:
            _, st = state["gpu"].render(seed=state["seed"], film_device_ptr=state["film"].data_ptr())
            film = state["film"]
        else:
            film, st = state["gpu"].render(seed=state["seed"])
        return {"film": film, "nan": st["nan_samples"]}
    if kind == "oneshot":
        film, _ = rumi_b200.render(state["flat"], seed=state["seed"])
        return {"film": film, "image": film_io.tonemap(film, c["spp"])}
    if kind == "batch":
        state["batch"].render(state["spp"], state["seeds"], c["depth"], graph=True,
                              films_device_ptr=state["films"].data_ptr())
        return {"films": state["films"]}
    g = state["gpu"]
    g.set_albedo(device_ptr=state["albedo"].data_ptr())
    g.set_volume((0.31, 0.3, 0.29), (0.05, 0.06, 0.05), 0.12)
    g.forward(seed=state["seed"], film_device_ptr=state["film"].data_ptr())
    g.backward_device(state["d_film"].data_ptr(), state["g_albedo"].data_ptr(), state["g_volume"].data_ptr(),
                      seed=state["seed"] + 1)
    return {"film": state["film"], "g_albedo": state["g_albedo"], "g_volume": state["g_volume"]}


# ------------------------------------------------------------------------------- bounds
def _scene_size(levels, extra=13):
    return 4 ** (levels + 1) + extra if levels else extra


def _ray_flops(n_prims):
    """One ray against a tree of n primitives: two boxes per level, one primitive."""
    return 40.0 * max(1.0, math.log2(n_prims)) + 60.0


def work(case):
    """Bytes: the scene's records once (36 B of geometry, 36 B of normals, 12 B of colour, 4 B of
    index per triangle, as the path uses them), rays in and hits out, films out.  Operations:
    per ray what a balanced tree needs; a path has one closest-hit and one shadow ray per
    vertex and about 200 operations of shading."""
    c, kind = case, case["kind"]
    if kind == "trace":
        n = _scene_size(c["levels"])
        return {"bytes": c["n"] * (28 + 8) + n * 36, "flops": c["n"] * _ray_flops(n)}
    if kind == "batch":
        paths = geometry = pixels = 0
        for i in range(c["scenes"]):
            up = 2.0 ** ((i * 5) % 7 - 3)
            res = max(16, int(c["res"] * math.sqrt(up)))
            pixels += res * res
            paths += res * res * c["spp"] * (1 + i % 3)
            geometry += max(200, int(c["tris"] * up))
        per = c["depth"] * (2 * _ray_flops(geometry / c["scenes"]) + 200.0)
        return {"bytes": geometry * 88 + pixels * 12, "flops": paths * per}
    n = _scene_size(c["levels"])
    pixels = c["width"] * c["height"]
    paths = pixels * c["spp"]
    per = c["depth"] * (2 * _ray_flops(n) + 200.0)
    if kind == "optimise":
        return {"bytes": n * (88 + 24) + pixels * 24, "flops": 3.0 * paths * per}
    if kind == "oneshot":
        # the build reads every triangle's bounds once per level of the tree
        return {"bytes": n * 88 + pixels * 15, "flops": paths * per + n * 20.0 * math.log2(n)}
    if c["integrator"] == "bdpt":  # two subpaths and a shadow ray per pair of their vertices
        per = (2 * c["depth"] + 1) * (_ray_flops(n) + 200.0) + c["depth"] * (c["depth"] + 1) * (_ray_flops(n) + 200.0) / 4
    elif c["integrator"] == "whitted":  # most chains end at the first diffuse surface
        per = 1.3 * (2 * _ray_flops(n) + 200.0)
    return {"bytes": n * 88 + pixels * 12, "flops": paths * per}


# -------------------------------------------------------------------------------- exact
def exact(case, seed):
    """Hit distances of small closest-hit queries in 64 bits: every ray against every
    primitive.  Frames, gradients and large queries have no such value: a frame is a sum over
    paths whose scattering decisions are made in 32 bits."""
    c = case
    if c["kind"] != "trace" or c["anyhit"] or c["n"] * _scene_size(c["levels"]) > 40000000:
        return None
    flat = _trace_scene(c, seed).flatten()
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f64 = functools.partial(torch.as_tensor, dtype=torch.float64, device=dev)
    rays = f64(_rays(c, flat, seed).astype(np.float64))
    tri, rect, sph = (f64(a.astype(np.float64)) for a in (flat.tri_vertices, flat.rects, flat.spheres))
    eps = 1e-4
    best = []
    for r in rays.split(max(1, 4000000 // max(1, tri.shape[0]))):
        o, d, tmax = r[:, None, 0:3], r[:, None, 3:6], r[:, None, 6]
        cand = []
        v0, e1, e2 = tri[None, :, 0], (tri[:, 1] - tri[:, 0])[None], (tri[:, 2] - tri[:, 0])[None]
        p = torch.linalg.cross(d.expand(-1, tri.shape[0], -1), e2.expand(r.shape[0], -1, -1))
        det = (p * e1).sum(-1)
        tv = o - v0
        q = torch.linalg.cross(tv, e1.expand(r.shape[0], -1, -1))
        u, v, t = (p * tv).sum(-1) / det, (q * d).sum(-1) / det, (q * e2).sum(-1) / det
        cand.append((t, (det.abs() >= 1e-8) & (u >= 0) & (v >= 0) & (u + v <= 1)))
        if rect.shape[0]:  # the light: two-sided
            p0, l, w = rect[None, :, 0:3], rect[None, :, 3:6], rect[None, :, 6:9]
            nrm = torch.linalg.cross(l, w)
            t = ((p0 - o) * nrm).sum(-1) / (d * nrm).sum(-1)
            at = o + d * t[..., None] - p0
            a, b = (at * l).sum(-1) / (l * l).sum(-1), (at * w).sum(-1) / (w * w).sum(-1)
            cand.append((t, (a >= 0) & (a <= 1) & (b >= 0) & (b <= 1)))
        if sph.shape[0]:
            oc = o - sph[None, :, 0:3]
            half = (d * oc).sum(-1)
            disc = half * half - (oc * oc).sum(-1) + sph[None, :, 3] ** 2
            cand.append((-half - disc.clamp(min=0).sqrt(), disc >= 0))
        t = torch.cat([x for x, _ in cand], 1)
        ok = torch.cat([y for _, y in cand], 1) & (t >= eps) & (tmax - t >= eps)
        t = torch.where(ok, t, torch.full_like(t, math.inf)).min(1).values
        best.append(torch.where(torch.isinf(t), torch.zeros_like(t), t))
    return {"t": torch.cat(best), "prim": None}
