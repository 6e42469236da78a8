"""The work that users of this framework have it do, as timed cases.

A case is a dict of plain values: what is rendered or computed ("kind"), on
which scene, at which size. ``listed()`` names the standing ones, ``draw(rng)``
gives further ones of the same ranges, ``prepare`` builds what a user's program
holds before the call (a loaded scenario with its renderer and parameters set),
``run`` is one pass through the public entry points, up to the image (or the
gradient, or the hits) in host memory, where the C API delivers it.

Kinds:
  pt      "Pathtracer": reset, ``spp`` iterations, image read-back
  targets "Pathtracer" with all eight targets and their variances
  lt      "Lighttracer"; bpt "Bidirectional Pathtracer"; vcm "Vertex Connection
          and Merging": reset, ``spp`` iterations, image read-back
  albedo  forward render and gradient of an albedo texture through torch.autograd
  batch   render_batch over several scenes, one image per job
  reload  an edited scene: an instance moved, the scenario loaded again (upload,
          BVH and light builds), ``spp`` iterations, image read-back
  rays    closest hits of a caller's own rays (baking, picking, sensors)
"""
from __future__ import annotations

import dataclasses
import functools
import math

import numpy as np
import torch

from mufflon_b200 import adjoint, bindings, scenes

# Rays (extension and shadow) that one sample of one pixel takes, measured once
# per scene; they only scale work(), the least work a pass can do.
RAYS_PER_SAMPLE = {"cornell": 8.0, "icosphere": 1.85, "instanced": 4.7, "plane": 3.0, "cutouts": 7.0}


def listed():
    return [
        # an interactive preview of a small scene: launches and latency count
        dict(name="cornell_64", kind="pt", scene="cornell", detail=0, width=64, height=64, spp=1, depth=8, nee=1),
        # the box scene at its usual size
        dict(name="cornell_256", kind="pt", scene="cornell", detail=0, width=256, height=256, spp=4, depth=8, nee=1),
        # the headline workload: a 1.31 M-triangle mesh at full HD
        dict(name="icosphere_1080p", kind="pt", scene="icosphere", detail=8, width=1920, height=1080, spp=16, depth=10,
             nee=1),
        # 4 096 instances of ten meshes plus 20 000 spheres, long paths
        dict(name="instanced_720p", kind="pt", scene="instanced", detail=4096, width=1280, height=720, spp=4, depth=12,
             nee=1),
        # denoiser and compositing input: every target with its variance, cut-out surfaces, two
        # next-event samples, a ragged image size
        dict(name="targets_cutouts", kind="targets", scene="cutouts", detail=0, width=613, height=457, spp=4, depth=8,
             nee=2),
        # the other renderers on the large mesh
        dict(name="lt_1080p", kind="lt", scene="icosphere", detail=8, width=1920, height=1080, spp=4, depth=10, nee=1),
        dict(name="bpt_720p", kind="bpt", scene="icosphere", detail=8, width=1280, height=720, spp=2, depth=10, nee=1),
        dict(name="vcm_ragged", kind="vcm", scene="icosphere", detail=7, width=1001, height=701, spp=2, depth=10, nee=1),
        # inverse rendering: one gradient step on a 512 x 512 texture
        dict(name="albedo_512", kind="albedo", scene="textured", detail=512, width=512, height=512, spp=16, depth=6, nee=1),
        # a render service: jobs of uneven size over four scenes
        dict(name="batch_16", kind="batch", scene="mixed", detail=16, width=384, height=384, spp=8, depth=12, nee=1),
        # an animation frame: an instance moved, everything built again, one sample per pixel
        dict(name="reload_540p", kind="reload", scene="icosphere", detail=8, width=960, height=540, spp=1, depth=10, nee=1),
        # a caller's rays against a mid-size mesh
        dict(name="rays_64k", kind="rays", scene="icosphere", detail=5, width=65536, height=1, spp=1, depth=1, nee=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pt", "pt", "pt", "targets", "lt", "bpt", "vcm", "albedo", "batch", "reload", "rays"])
    scene = {"pt": rng.choice(["cornell", "icosphere", "instanced", "plane", "cutouts"]),
             "targets": rng.choice(["cutouts", "icosphere", "cornell"]), "albedo": "textured", "batch": "mixed",
             "reload": rng.choice(["icosphere", "plane", "instanced"]),
             "rays": rng.choice(["icosphere", "plane"])}.get(kind, rng.choice(["icosphere", "cornell", "plane"]))
    detail = {"icosphere": rng.randint(4, 8), "plane": _log(rng, 40, 400), "instanced": _log(rng, 200, 4096),
              "textured": _log(rng, 64, 512), "mixed": rng.randint(2, 16)}.get(scene, 0)
    if kind == "rays":
        return dict(kind=kind, scene=scene, detail=min(detail, 8 if scene == "icosphere" else 224),
                    width=_log(rng, 1000, 1_000_000), height=1, spp=1, depth=1, nee=1)
    # pixels over their logarithm, the aspect ratio around 16:9, odd sizes as they come
    most = {"pt": 2_000_000, "targets": 500_000, "lt": 2_000_000, "bpt": 900_000, "vcm": 700_000, "albedo": 260_000,
            "batch": 150_000, "reload": 1_000_000}[kind]
    pixels = _log(rng, 4096, most)
    aspect = rng.uniform(1.0, 2.0)
    height = max(16, int(round(math.sqrt(pixels / aspect))))
    width = max(16, int(round(pixels / height)))
    budget = {"pt": 8_000_000 if scene != "instanced" else 3_500_000, "targets": 1_200_000, "lt": 8_000_000,
              "bpt": 1_800_000, "vcm": 1_400_000, "albedo": 4_000_000, "batch": 1_200_000, "reload": 1_000_000}[kind]
    spp = rng.randint(1, max(1, min(16, budget // (width * height))))
    depth = rng.randint(4, 6) if kind == "albedo" else rng.randint(4, 12)
    nee = rng.choice([1, 1, 2, 3]) if kind in ("pt", "targets") else 1
    return dict(kind=kind, scene=scene, detail=detail, width=width, height=height, spp=spp, depth=depth, nee=nee)


# ------------------------------------------------------------------ scenes
@functools.lru_cache(maxsize=None)
def _base(scene, detail):
    if scene == "icosphere":
        return scenes.displaced_icosphere(0, subdiv=detail)
    if scene == "instanced":
        return scenes.instanced_scene(0, num_instances=detail)
    if scene == "plane":
        return scenes.displaced_plane(0, n=detail)
    raise ValueError(scene)


def _spec(scene, detail, width, height, seed):
    """The scene of a seed: other shapes, materials and camera for every seed."""
    if scene == "cornell":
        return scenes.cornell_box(seed, width, height)
    if scene == "cutouts":
        return scenes.alpha_cutouts(seed, width, height)
    if scene == "textured":
        return scenes.cornell_box_textured(seed, width, height, texture_size=detail)
    base = _base(scene, detail)
    rng = np.random.default_rng(seed)
    lods = list(base.lods)
    for k, lod in enumerate(lods):
        if len(lod.vertices) > 8:  # a smooth bump field over the mesh, another one for every seed
            f, ph = rng.uniform(1.5, 4.0, 3), rng.uniform(0.0, 2.0 * math.pi, 3)
            v = lod.vertices
            bump = np.sin(v[:, 0] * np.float32(f[0]) + np.float32(ph[0])) * np.sin(v[:, 1] * np.float32(f[1]) + np.float32(ph[1]))
            bump = bump * np.sin(v[:, 2] * np.float32(f[2]) + np.float32(ph[2])) * np.float32(0.02)
            lods[k] = dataclasses.replace(lod, vertices=np.ascontiguousarray(v * (np.float32(1.0) + bump)[:, None]))
    mats = [dataclasses.replace(m, albedo=tuple(float(x) for x in rng.uniform(0.2, 0.8, 3)),
                                **({"roughness": (r, r)} if (r := float(rng.uniform(0.1, 0.5))) and m.type == scenes.MAT_TORRANCE
                                   else {})) for m in base.materials]
    cam = tuple(float(c + d) for c, d in zip(base.cam_pos, rng.uniform(-0.1, 0.1, 3)))
    return dataclasses.replace(base, lods=lods, materials=mats, cam_pos=cam, width=width, height=height)


def _world(spec):
    dll = bindings.DllInterface()
    bindings.load_scene_spec(dll, spec)
    return dll


def _renderer(dll, name, case, seed):
    for i in range(dll.render_get_renderer_count()):
        if dll.render_get_renderer_short_name(i) == name:
            dll.render_enable_renderer(i, 0)
    params = {"Seed": seed & 0x7FFFFFFF, "Max. path length": case["depth"]}
    if name == "PT":
        params["NEE count"] = case["nee"]
        if case["scene"] == "instanced":
            params["RR start depth"] = 3
    for key, value in params.items():
        if not dll.renderer_set_parameter_int(key, value):
            raise RuntimeError(dll.core_get_dll_error())


TARGETS = ["Radiance", "Position", "Depth", "Normal", "UV", "Albedo", "Lightness", "Hit ID"]


def prepare(case, seed):
    kind, scene = case["kind"], case["scene"]
    w, h = case["width"], case["height"]
    if kind == "batch":
        worlds = [_world(_spec(s, d, w, h, seed + k)) for k, (s, d) in enumerate(
            [("cornell", 0), ("icosphere", 7), ("instanced", 500), ("plane", 224)])]
        for dll in worlds:
            _renderer(dll, "PT", case, seed)
        rng = np.random.default_rng(case["detail"])  # the jobs' sizes are the case's, their scenes and samples the seed's
        jobs = []
        for j in range(case["detail"]):  # sides and samples spread about the case's own
            s = math.exp(rng.uniform(-0.9, 0.0)) if j else 1.0
            jobs.append(dict(instance=worlds[j % 4], width=max(16, int(w * s)), height=max(16, int(h * s)),
                             spp=int(rng.integers(1, case["spp"] + 1)) if j else case["spp"], seed=seed % 10007 + j,
                             max_path=4 + (case["depth"] - 4) * (j % 4) // 3, rr_start=0, nee=case["nee"]))
        return dict(kind=kind, worlds=worlds, jobs=jobs)
    spec = _spec(scene, case["detail"], 64 if kind == "rays" else w, 64 if kind == "rays" else h, seed)
    dll = _world(spec)
    state = dict(kind=kind, dll=dll, spp=case["spp"])
    if kind == "rays":
        state["rays"] = _rays(spec, w, seed)
        return state
    _renderer(dll, {"lt": "LT", "bpt": "BPT", "vcm": "VCM"}.get(kind, "PT"), case, seed)
    if kind == "targets":
        for t in TARGETS:
            dll.render_enable_render_target(t, True)
    else:
        dll.render_enable_render_target("Radiance", False)
    if kind == "albedo":
        n = case["detail"]
        g = torch.Generator().manual_seed(seed)
        state["texels"] = (torch.rand((n, n, 3), generator=g) * 0.6 + 0.2).cuda()
        state["target"] = torch.rand((h, w, 3), generator=g).cuda()
        state["renderer"] = adjoint.AlbedoRenderer(dll, dll.textures[0], (n, n), spp=case["spp"], seed=seed & 0x7FFFFFFF,
                                                   max_path=case["depth"], nee=case["nee"])
    if kind == "reload":
        state["moving"] = _moving(dll, spec, seed)
    return state


def _moving(dll, spec, seed):
    """The instance that the animation moves, a small copy of the scene's first object, and its pose."""
    core = dll.core
    handle = core.world_create_instance(dll.muffInst, core.world_get_object(dll.muffInst, spec.lods[0].name.encode()), 0)
    rng = np.random.default_rng(seed + 77)
    yaw, scale, pos = rng.uniform(0.0, 2.0 * math.pi), rng.uniform(0.2, 0.4), rng.uniform(-1.0, 1.0, 3)
    rot = np.array([[math.cos(yaw), 0.0, math.sin(yaw)], [0.0, 1.0, 0.0], [-math.sin(yaw), 0.0, math.cos(yaw)]])
    m = bindings.Mat3x4()
    m.v[:] = [float(x) for x in np.concatenate([rot.T / scale, (-rot.T / scale @ pos)[:, None]], axis=1).reshape(-1)]
    return handle, m


def _rays(spec, n, seed):
    """Rays towards the mesh, from around it (a plane: from above it); they hit, since a miss reports
    the largest distance, next to which an error of the hits would not show."""
    rng = np.random.default_rng(seed + 5)
    v = spec.lods[0].vertices
    ctr, ext = v.mean(0), float(np.abs(v - v.mean(0)).max())
    if spec.name == "displaced_plane":
        o = rng.uniform(-0.95, 0.95, (n, 3)) * ext
        o[:, 1] = rng.uniform(0.2, 2.0, n) * ext
        t = rng.uniform(-0.95, 0.95, (n, 3)) * ext
        t[:, 1] = -0.5 * ext
    else:
        o = rng.normal(size=(n, 3))
        o = o / np.linalg.norm(o, axis=1, keepdims=True) * rng.uniform(1.6, 3.0, (n, 1)) * ext
        t = rng.uniform(-0.5, 0.5, (n, 3)) * ext
    d = t - o
    d = d / np.linalg.norm(d, axis=1, keepdims=True)
    return np.ascontiguousarray(np.concatenate([o + ctr, d], 1), np.float32)


# ------------------------------------------------------------------ one pass
def _frame(dll, spp):
    dll.render_reset()
    for _ in range(spp):
        dll.render_iterate()


def run(state):
    kind = state["kind"]
    if kind == "batch":
        return bindings.render_batch(state["jobs"])[0]
    dll = state["dll"]
    if kind == "rays":
        t, inst, prim, sp = dll.trace_rays(state["rays"])
        return dict(t=t, instance=inst, primitive=prim, surface=sp)
    if kind == "albedo":
        tex = state["texels"].clone().requires_grad_(True)
        image = adjoint.render_albedo(tex, state["renderer"])
        loss = ((image - state["target"]) ** 2).sum()
        loss.backward()
        return dict(image=image.detach(), gradient=tex.grad)
    if kind == "reload":
        _move(dll, *state["moving"])
    _frame(dll, state["spp"])
    if kind == "targets":
        return {t + v: dll.get_target_image(t, variance=bool(v)) for t in TARGETS for v in ("", " variance")}
    # the library's own read-back buffer, as the C API hands it out; the image keeps its library open
    image = dll.get_target_image("Radiance", copy=False).view(_Image)
    image.owner = dll
    return image


class _Image(np.ndarray):
    owner = None


def _move(dll, handle, matrix):
    if not dll.instance_set_transformation_matrix(handle, matrix, True):
        raise RuntimeError(dll.core_get_dll_error())
    if not dll.world_load_scenario(dll.world_get_current_scenario()):
        raise RuntimeError(dll.core_get_dll_error())


# ------------------------------------------------------------------ what a pass cannot do without
def _triangles(scene, detail):
    return {"icosphere": 20 * 4 ** detail, "plane": 2 * detail * detail, "instanced": 760_000, "mixed": 1_200_000}.get(scene, 34)


def work(case):
    """Bytes: the scene read once, the image (or gradient, or hits) written once. Operations: per ray
    one descent through an 8-wide hierarchy (eight boxes of 18 operations a level) and two
    triangle tests of 60, per sample the shading of its vertices (300 each)."""
    tris = _triangles(case["scene"], case["detail"])
    scene_bytes = tris * 30.0
    pixels = float(case["width"] * case["height"])
    channels = 3.0
    if case["kind"] == "targets":
        channels = 2.0 * (3 + 3 + 1 + 3 + 2 + 3 + 1 + 2)
    elif case["kind"] == "batch":
        pixels *= 1.0 + (case["detail"] - 1) * 0.46
    elif case["kind"] == "rays":
        channels = 5.0 + 6.0
    samples = pixels * case["spp"]
    if case["kind"] == "batch":
        samples *= 0.56
    per = RAYS_PER_SAMPLE.get({"textured": "cornell", "mixed": "instanced"}.get(case["scene"], case["scene"]), 2.0)
    if case["kind"] == "rays":
        per = 1.0
    elif case["kind"] in ("bpt", "vcm"):
        per *= 2.5
    elif case["kind"] == "albedo":
        per *= 2.0  # the samples are replayed for the gradient
    levels = max(1.0, math.log(tris, 8.0))
    flops = samples * per * (levels * 8.0 * 18.0 + 120.0 + 300.0)
    extra = {"albedo": 2.0 * case["detail"] ** 2 * 12.0 + pixels * 12.0}.get(case["kind"], 0.0)
    if case["kind"] == "reload":
        scene_bytes += tris * (30.0 + 64.0)  # uploaded, and the hierarchy written
        flops += tris * 200.0
    return {"bytes": scene_bytes + pixels * channels * 4.0 + extra, "flops": flops}


def tolerance(case):
    """The path tracer's images and the hits are defined bit for bit: every random decision of a path
    is a comparison of 32-bit values whose operations and order are fixed, and the running mean adds the
    samples in order. The renderers below add splats (or texel gradients) with 32-bit atomics in any
    order: the sums of a pixel or texel differ in their last bits from pass to pass."""
    if case["kind"] in ("lt", "bpt", "vcm", "albedo"):
        return {"rel": 1e-6, "max": 4e-5}
    return "exact"


def exact(case, seed):
    """Closest hits in 64 bits by testing every triangle; None for the Monte Carlo images, which have no
    value of their own in 64 bits: a path's random decisions are comparisons of 32-bit values."""
    if case["kind"] != "rays":
        return None
    spec = _spec(case["scene"], case["detail"], 64, 64, seed)
    if case["width"] * _triangles(case["scene"], case["detail"]) > 4e9:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    rays = torch.from_numpy(_rays(spec, case["width"], seed)).to(dev, torch.float64)
    lod = spec.lods[0]
    v = torch.from_numpy(lod.vertices).to(dev, torch.float64)
    tri = v[torch.from_numpy(lod.triangles.astype(np.int64)).to(dev)]
    if len(spec.lods) > 1:  # the ground quad is planar: two triangles
        g = torch.from_numpy(spec.lods[1].vertices).to(dev, torch.float64)
        tri = torch.cat([tri, torch.stack([torch.stack([g[0], g[1], g[2]]), torch.stack([g[0], g[2], g[3]])])])
    a, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    # Moeller-Trumbore as matrix products: det = d.(e1 x e2) and so on, with o and d apart
    n = torch.linalg.cross(e1, e2)
    out_t = torch.full((case["width"],), -1.0, dtype=torch.float64, device=dev)
    step = max(1, int(4e7) // len(tri))
    for i in range(0, case["width"], step):
        o, d = rays[i:i + step, :3], rays[i:i + step, 3:]
        od = torch.linalg.cross(o, d)
        det = -(d @ n.T)
        t = ((o @ n.T) - (a * n).sum(1)) / det
        # u = e2 . ((o - a) x d) / det, v = -e1 . ((o - a) x d) / det
        ae2, ae1 = torch.linalg.cross(e2, a), torch.linalg.cross(e1, a)
        u = (od @ e2.T - d @ ae2.T) / det
        w = -(od @ e1.T - d @ ae1.T) / det
        hit = (u >= 0) & (w >= 0) & (u + w <= 1) & (t > 0)
        t = torch.where(hit, t, torch.inf)
        best = t.min(1).values
        out_t[i:i + step] = torch.where(torch.isfinite(best), best, float(MISS))
    return dict(t=out_t.cpu().numpy(), instance=None, primitive=None, surface=None)


MISS = 1048576.0  # the distance reported for a miss: the queries' default maximum
