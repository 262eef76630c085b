"""The work a user of this library has it do, as cases that can be timed.

Every case goes through the package's public entry points:

  frames    `RayTracingRenderer.render_to_device`: an app that keeps its scene
            on the GPU and moves the camera (implicit, textured and mesh
            scenes; 1 to 8 bounces; plain and 2x2 supersampled canvases)
  animated  `RayTracingRenderer.render`: the drop-in call of an app that moves
            its objects too -- host scene BVH, per-frame uploads, the frame,
            and the canvas in ordinary host arrays
  batch     `BatchRenderer`: a batch of requests arrives, each with a scene,
            a camera and a canvas of its own
  query     `RadianceCache.query` on device samples
  train     `RadianceCache.train`, one Adam step, and its gradients

The scenes are the package's own generators (`scenes.config1`, `config2`,
`config3`, `batch_request`).  The library holds one scene at a time, as the
reference does, so the scene belongs to the case (a program uploads it once)
and the seed makes what changes from frame to frame: the camera, the moved
objects, the requests, the samples.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from slimtracincpp_b200 import layout as L
from slimtracincpp_b200 import scenes
from slimtracincpp_b200.batch import BatchRenderer
from slimtracincpp_b200.native import set_render_options
from slimtracincpp_b200.radiance_cache import RadianceCache
from slimtracincpp_b200.renderer import RayTracingRenderer, Viewport
from slimtracincpp_b200.scene import Camera, MeshAsset


def listed():
    return [
        # a thumbnail or preview pane of a simple scene: launch latency
        {"name": "preview_180p", "kind": "implicit", "width": 320, "height": 180, "depth": 1, "ssaa": False, "layout": 0},
        # the same scene supersampled on an odd canvas: the ordinary viewport of an editor
        {"name": "implicit_ssaa_361p", "kind": "implicit", "width": 641, "height": 361, "depth": 1, "ssaa": True,
         "layout": 0},
        # glass, mirrors, textures and sky in a small odd window, mips by per-pixel cones
        {"name": "textured_241p", "kind": "textured", "width": 427, "height": 241, "depth": 8, "ssaa": False,
         "layout": 0, "cones": True},
        # the same scene full screen
        {"name": "textured_1080p", "kind": "textured", "width": 1920, "height": 1080, "depth": 8, "ssaa": False,
         "layout": 0, "cones": False},
        # light meshes (5,120 and 7,938 triangles) in a ragged window, a few bounces
        {"name": "mesh_359p", "kind": "mesh", "width": 637, "height": 359, "depth": 4, "ssaa": False, "layout": 0,
         "subdivisions": 4, "grid": 64},
        # the headline frame: 81,920- and 130,050-triangle meshes, depth 2
        {"name": "mesh_1080p", "kind": "mesh", "width": 1920, "height": 1080, "depth": 2, "ssaa": False, "layout": 0,
         "subdivisions": 6, "grid": 256},
        # the same scene with the reference's full bounce depth
        {"name": "mesh_1080p_deep", "kind": "mesh", "width": 1920, "height": 1080, "depth": 8, "ssaa": False,
         "layout": 0, "subdivisions": 6, "grid": 256},
        # the largest canvas the batched workload uses
        {"name": "mesh_2160p", "kind": "mesh", "width": 3840, "height": 2160, "depth": 2, "ssaa": False, "layout": 0,
         "subdivisions": 6, "grid": 256},
        # an app's whole frame with moving objects, into host arrays
        {"name": "animated_720p", "kind": "animated", "width": 1280, "height": 720, "depth": 2, "ssaa": False,
         "layout": 0, "subdivisions": 6, "grid": 256},
        # a server's batch: small and large canvases, shallow and deep paths together
        {"name": "batch_8", "kind": "batch", "requests": 8, "subdivisions": 6, "grid": 256},
        # the radiance cache answering half a 1080p frame
        {"name": "query_1m", "kind": "query", "count": 1036801},
        # one training step of the default size
        {"name": "train_16k", "kind": "train", "count": 16384},
    ]


def draw(rng):
    kind = rng.choice(["implicit", "implicit", "textured", "textured", "mesh", "mesh", "mesh", "animated", "batch",
                       "query", "train"])
    if kind == "query":
        return {"kind": kind, "count": int(math.exp(rng.uniform(math.log(1000), math.log(2073600))))}
    if kind == "train":
        return {"kind": kind, "count": int(math.exp(rng.uniform(math.log(1000), math.log(65536))))}
    meshes = {"subdivisions": rng.randint(3, 6), "grid": rng.randint(48, 256)}
    if kind == "batch":
        return {"kind": kind, "requests": rng.randint(2, 8), **meshes}
    case = {"kind": kind, "layout": rng.randint(0, 999)}
    if kind == "implicit":
        case["depth"], largest = rng.randint(1, 3), 3840 * 2160
    elif kind == "textured":
        case["depth"], largest = rng.randint(1, 8), 1920 * 1080
        case["cones"] = rng.random() < 0.5
    elif kind == "mesh":
        case["depth"] = rng.randint(1, 8)
        largest = 2560 * 1440 if case["depth"] <= 2 else 1600 * 900
    else:
        case["depth"], largest = rng.randint(1, 4), 1920 * 1080
    if kind in ("mesh", "animated"):
        case.update(meshes)
    samples = math.exp(rng.uniform(math.log(320 * 180), math.log(largest)))
    case["ssaa"] = kind != "animated" and rng.random() < 0.25
    pixels = samples / 4 if case["ssaa"] else samples
    aspect = rng.choice([16 / 9, 16 / 9, 4 / 3, 1.0, 21 / 9, 9 / 16])
    case["width"] = max(16, int(math.sqrt(pixels * aspect)))
    case["height"] = max(16, int(pixels / case["width"]))
    return case


# ---- assets and scenes of a case -------------------------------------------------

_assets = {}
_workloads = {}
_uploaded = {"key": None, "handle": None}


def _meshes(case):
    """The icosphere and the heightfield of the mesh scenes at the case's detail."""
    out = []
    for key, build in ((("sphere", case["subdivisions"]), lambda: scenes.icosphere(case["subdivisions"])),
                       (("field", case["grid"]), lambda: scenes.heightfield(np.random.default_rng(7), case["grid"], 0.3))):
        if key not in _assets:
            positions, indices, normals = build()
            _assets[key] = MeshAsset.build(positions, indices, normals=normals, normal_indices=indices)
        out.append(_assets[key])
    return out


def _scene_key(case):
    return tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "width", "height", "ssaa")))


def _workload(case):
    key = _scene_key(case)
    if key not in _workloads:
        w, h, layout = case["width"], case["height"], case["layout"]
        if case["kind"] == "implicit":
            work = scenes.config1(layout, w, h)
        elif case["kind"] == "textured":
            work = scenes.config3(layout, w, h, tex_size=512, cube_size=256)
        else:
            work = scenes.config2(layout, w, h, meshes=_meshes(case))
        _workloads.clear()
        _workloads[key] = work
    return _workloads[key]


def _upload(key, build):
    """The program's one-time upload: again only when another scene took its place."""
    if _uploaded["key"] != key:
        _uploaded["key"] = None
        _uploaded["handle"] = build()
        _uploaded["key"] = key
    return _uploaded["handle"]


def _renderer(case):
    def build():
        scene, st = _workload(case).scene, _workload(case).settings
        set_render_options(engine=L.ENGINE_AUTO,
                           ray_cones=L.CONES_PER_PIXEL if case.get("cones") else L.CONES_REFERENCE)
        return RayTracingRenderer(scene, max_depth=case["depth"],
                                  skybox_color_texture_id=int(st["skybox_color_texture_id"]),
                                  skybox_radiance_texture_id=int(st["skybox_radiance_texture_id"]),
                                  skybox_irradiance_texture_id=int(st["skybox_irradiance_texture_id"]))
    return _upload(_scene_key(case), build)


def _viewport(case, rng):
    """The scene's own camera, moved and turned a little: the next frame of a walk."""
    eye = {"implicit": (0.0, 6.0, -14.0), "textured": (0.0, 5.0, -13.0)}.get(case["kind"], (0.0, 6.0, -11.0))
    eye = np.array(eye) + rng.uniform(-0.8, 0.8, 3)
    target = np.array((0.0, 1.0, 1.0)) + rng.uniform(-0.3, 0.3, 3)
    return Viewport(Camera.look_at(eye, target, 60.0), case["width"], case["height"],
                    L.AA_SSAA if case["ssaa"] else L.AA_NONE)


def _samples(rng, count, device="cuda"):
    """Cache samples as the tracer gathers them: position in the scene box and
    roughness, direction, shading normal, albedo."""
    f = np.zeros((count, 16), np.float32)
    f[:, 0:3] = rng.random((count, 3))
    f[:, 3] = rng.uniform(0.05, 1.0, count)
    for k in (4, 8):
        v = rng.standard_normal((count, 3))
        f[:, k:k + 3] = v / np.linalg.norm(v, axis=1, keepdims=True)
    f[:, 12:15] = rng.uniform(0.2, 1.0, (count, 3))
    return torch.from_numpy(f).to(device)


def _targets(rng, count, device="cuda"):
    """Radiance of path suffixes: log-normal, a tenth of them black."""
    y = np.zeros((count, 4), np.float32)
    y[:, :3] = np.exp(rng.normal(-1.0, 1.0, (count, 3))) * (rng.random((count, 1)) > 0.1)
    return torch.from_numpy(y).to(device)


def _cache_weights():
    """He-uniform weights, the output layer ten times smaller."""
    rng = np.random.default_rng(11)
    shapes = [(64, 96), (64, 64), (64, 64), (64, 64), (3, 64)]
    return np.concatenate([(rng.uniform(-1, 1, r * c) * math.sqrt(6.0 / c) * (0.1 if r == 3 else 1.0))
                           for r, c in shapes]).astype(np.float32)


# ---- the cases -------------------------------------------------------------------

def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind in ("query", "train"):
        def build():   # the cache lives beside a scene: the smallest one
            set_render_options(engine=L.ENGINE_AUTO)
            RayTracingRenderer(scenes.config1(0, 320, 180).scene, max_depth=1)
            return RadianceCache.configure()
        cache = _upload(("cache",), build)
        cache.weights = _cache_weights()
        state = {"cache": cache, "count": case["count"], "features": _samples(rng, case["count"])}
        if kind == "train":
            state["targets"] = _targets(rng, case["count"])
        else:
            state["radiance"] = torch.empty((case["count"], 4), device="cuda")
        return {"kind": kind, **state}
    if kind == "batch":
        meshes = _meshes(case)

        def build():
            set_render_options(engine=L.ENGINE_AUTO)
            return BatchRenderer(scenes.config2(0, 320, 180, meshes=meshes).scene)
        batch = _upload(_scene_key({**case, "requests": 0}), build)
        requests, outputs, tensors = [], [], []
        for i in range(case["requests"]):
            w, h = scenes.BATCH_RESOLUTIONS[i % 4]
            requests.append(scenes.batch_request(rng, meshes, w, h, 1 + (3 * i) % 8, L.CACHE_OFF, i))
            pixels, depths = torch.empty((w * h, 4), device="cuda"), torch.empty(w * h, device="cuda")
            tensors.append((pixels, depths))
            outputs.append((pixels.data_ptr(), depths.data_ptr()))
        return {"kind": kind, "batch": batch, "requests": requests, "outputs": outputs, "tensors": tensors}
    renderer = _renderer(case)
    viewport = _viewport(case, rng)
    state = {"kind": kind, "renderer": renderer, "viewport": viewport}
    if kind == "animated":
        geometries = _workload(case).scene.geometries
        if "rest" not in _uploaded or _uploaded["rest"][0] != _scene_key(case):
            _uploaded["rest"] = (_scene_key(case), geometries.copy())
        moved = _uploaded["rest"][1].copy()
        moved["position"][:8] += rng.uniform(-0.4, 0.4, (8, 3)).astype(np.float32)
        state["geometries"] = moved
        return state
    s = 4 if case["ssaa"] else 1
    count = case["width"] * case["height"] * s
    state["pixels"] = torch.empty((count, 4), device="cuda")
    state["depths"] = torch.empty(count, device="cuda")
    return state


def run(state):
    kind = state["kind"]
    if kind == "query":
        state["cache"].query(state["features"].data_ptr(), state["count"], state["radiance"].data_ptr())
        return state["radiance"]
    if kind == "train":
        state["cache"].train(state["features"].data_ptr(), state["targets"].data_ptr(), state["count"])
        return state["cache"].gradients()
    if kind == "batch":
        state["batch"].set_requests(state["requests"], state["outputs"])
        state["batch"].render()
        return state["tensors"]
    renderer = state["renderer"]
    if kind == "animated":
        renderer.scene.geometries[:] = state["geometries"]   # the app's objects have moved
        return renderer.render(state["viewport"])
    renderer.render_to_device(state["viewport"], state["pixels"].data_ptr(), state["depths"].data_ptr())
    return state["pixels"], state["depths"]


def work(case):
    kind = case["kind"]
    macs = 96 * 64 + 3 * 64 * 64 + 64 * 3
    if kind == "query":
        return {"bytes": case["count"] * (64 + 16) + 2 * macs, "flops": 2 * macs * case["count"]}
    if kind == "train":
        # weights, both moments and the gradient beside the samples
        return {"bytes": case["count"] * (64 + 16) + 8 * 4 * macs, "flops": 3 * 2 * macs * case["count"]}
    # the canvas written once, the scene's records read once
    triangles = 20 * 4 ** case["subdivisions"] + 2 * (case["grid"] - 1) ** 2 if "grid" in case else 0
    scene = triangles * 128 + (2 * triangles - 1) * 32 if triangles else 0
    if kind == "textured":
        scene += 6 * (513 * 513 * 4 // 3) * 12
    if kind == "batch":
        sizes = [scenes.BATCH_RESOLUTIONS[i % 4] for i in range(case["requests"])]
        return {"bytes": scene + sum(w * h for w, h in sizes) * 20, "flops": 0}
    samples = case["width"] * case["height"] * (4 if case["ssaa"] else 1)
    return {"bytes": scene + samples * 20, "flops": 0}


# ---- the same in 64 bits ---------------------------------------------------------

def exact(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    if kind == "query":
        z = _network(_cache_weights(), _samples(rng, case["count"]))[0]
        y = torch.clamp(torch.exp(torch.clamp(z, max=15.0)) - 0.01, min=0.0)
        return torch.cat([y, torch.zeros_like(y[:, :1])], 1)
    if kind == "train":
        z, weights = _network(_cache_weights(), _samples(rng, case["count"]), grad=True)
        y = _targets(rng, case["count"])[:, :3].double()
        ((z - torch.log(y + 0.01)) ** 2).mean().backward()
        return torch.cat([w.grad.reshape(-1) for w in weights])
    if kind == "implicit":   # no mirrors, no glass: paths end at the first hit
        return _implicit_frame(case, _viewport(case, rng))
    # Paths through meshes or past the first hit: testing a ray against every
    # triangle in 64 bits takes minutes, and one ulp at an edge sends a
    # bounced path elsewhere.
    return None


def _network(params, features, grad=False):
    """The radiance cache's network: encoding, four ReLU layers, three outputs."""
    f = features.double()
    columns = []
    for axis in range(3):
        for octave in range(12):
            a = f[:, axis] * (2.0 ** octave) * math.pi
            columns += [torch.sin(a), torch.cos(a)]
    x, y, z = f[:, 4], f[:, 5], f[:, 6]
    c1, c2, c3 = math.sqrt(3 / (4 * math.pi)), math.sqrt(15 / (4 * math.pi)), math.sqrt(5 / (16 * math.pi))
    c4, c5, c6 = math.sqrt(35 / (32 * math.pi)), math.sqrt(105 / (4 * math.pi)), math.sqrt(21 / (32 * math.pi))
    columns += [torch.full_like(x, math.sqrt(1 / (4 * math.pi))), -c1 * y, c1 * z, -c1 * x,
                c2 * x * y, -c2 * y * z, c3 * (3 * z * z - 1), -c2 * x * z, c2 / 2 * (x * x - y * y),
                -c4 * y * (3 * x * x - y * y), c5 * x * y * z, c6 * y * (1 - 5 * z * z),
                math.sqrt(7 / (16 * math.pi)) * z * (5 * z * z - 3), c6 * x * (1 - 5 * z * z),
                c5 / 2 * z * (x * x - y * y), c4 * x * (3 * y * y - x * x)]
    columns += [f[:, 8], f[:, 9], f[:, 10], f[:, 3], f[:, 12], f[:, 13], f[:, 14], torch.ones_like(x)]
    h, weights, at = torch.stack(columns, 1), [], 0
    for rows, cols in [(64, 96), (64, 64), (64, 64), (64, 64), (3, 64)]:
        w = torch.from_numpy(params[at:at + rows * cols]).to(h.device).double().reshape(rows, cols).requires_grad_(grad)
        at += rows * cols
        weights.append(w)
        h = h @ w.T
        if rows == 64:
            h = torch.relu(h)
    return h, weights


def _cross(a, b):
    return torch.linalg.cross(a, b.expand_as(a) if b.dim() < a.dim() else b)


def _rotate(axis, w, v):
    axis = axis.expand_as(v)
    out = _cross(axis, v)
    return 2.0 * (w * out + _cross(axis, out)) + v


def _dot(a, b):
    return (a * b).sum(-1)


def _unit(a):
    return a / torch.sqrt(_dot(a, a))[..., None]


_TET = 0.57735025882720947       # float(1/sqrt 3) and half of it, as the layout stores them
_TET_HALF = 0.28867515921592712


def _hit(kind, o, d, any_hit=False):
    """Distance and local normal of the nearest accepted hit (inf: none) of a unit primitive."""
    inf = torch.full_like(o[:, 0], math.inf)
    zero = torch.zeros_like(o)
    if kind == L.GEOMETRY_QUAD:
        t = -o[:, 1] / d[:, 1]
        p = o + d * t[:, None]
        ok = (t > 0) & (p[:, 0].abs() <= 1) & (p[:, 2].abs() <= 1)
        n = zero.clone()
        n[:, 1] = torch.where(o[:, 1] < 0, -1.0, 1.0)
        return torch.where(ok, t, inf), n
    if kind == L.GEOMETRY_SPHERE:
        tc, dd = -_dot(o, d), _dot(d, d)
        sq = _dot(o, o) * dd - tc * tc
        # The path's test bounds sq by 1, the squared radius, where |d|^2 times
        # that is meant: small spheres lose their rims, and past the rim of a
        # large one the distance is NaN, which no closest hit takes and which
        # blocks a shadow ray that reaches the sphere's box.
        delta = torch.sqrt(torch.clamp(dd - sq, min=0.0))
        near, far = (tc - delta) / dd, (tc + delta) / dd
        t = torch.where(near > 0, near, far)
        p = o + d * t[:, None]
        out = torch.where((tc > 0) & (sq <= 1) & (sq <= dd) & (t > 0), t, inf)
        if any_hit:
            box = _hit(L.GEOMETRY_BOX, o, d)[0]
            out = torch.where((tc > 0) & (sq <= 1) & (sq > dd), box, out)
        return out, torch.where((near > 0)[:, None], p, -p)
    if kind == L.GEOMETRY_BOX:
        sign = torch.where(d < 0, -1.0, 1.0).double()
        near, near_axis = ((-sign - o) / d).max(1)
        far, far_axis = ((sign - o) / d).min(1)
        inside = near < 0
        t, axis = torch.where(inside, far, near), torch.where(inside, far_axis, near_axis)
        ok = (far >= 0) & (far >= torch.clamp(near, min=0.0))
        n = zero.scatter(1, axis[:, None], -torch.gather(sign, 1, axis[:, None]))   # both cases face the ray
        return torch.where(ok, t, inf), n
    best, normal = inf, zero   # the tetrahedron's four faces
    a, h = _TET, _TET_HALF
    faces = [((-a, -a, -a), (-a, a, -a), (a, -h, -a, h, h, a, -h, a, -a)),
             ((-a, -a, -a), (a, -a, -a), (h, h, a, -h, a, -a, a, -h, -a)),
             ((-a, -a, -a), (-a, -a, a), (-h, a, -a, a, -h, -a, h, h, a)),
             ((a, -a, a), (a, a, a), (-a, h, a, h, h, a, h, -a, a))]
    for point, face_normal, m in faces:
        point, n = o.new_tensor(point), o.new_tensor(face_normal)
        facing = _dot(n, d)
        t = _dot(n, point - o) / facing
        q = o + d * t[:, None] - point
        u = m[0] * q[:, 0] + m[3] * q[:, 1] + m[6] * q[:, 2]
        v = m[1] * q[:, 0] + m[4] * q[:, 1] + m[7] * q[:, 2]
        ok = (t > 0) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t < best)
        best = torch.where(ok, t, best)
        normal = torch.where(ok[:, None], torch.where((facing > 0)[:, None], -n, n), normal)
    return best, normal


def _trace(geometries, o, d, any_hit=False):
    """Closest hit over all primitives: distance, geometry index, world normal."""
    o = o + d * 1e-4
    best = torch.full_like(o[:, 0], math.inf)
    index = torch.full_like(best, -1, dtype=torch.int64)
    normal = torch.zeros_like(o)
    for i, g in enumerate(geometries):
        axis, w, s = (o.new_tensor(np.asarray(g[k], np.float64)) for k in ("axis", "amount", "scale"))
        p = o.new_tensor(np.asarray(g["position"], np.float64))
        t, n = _hit(int(g["type"]), _rotate(-axis, w, o - p) / s, _rotate(-axis, w, d) / s, any_hit)
        closer = t < best
        best, index = torch.where(closer, t, best), torch.where(closer, i, index)
        normal = torch.where(closer[:, None], _unit(_rotate(axis, w, s * n)), normal)
    return best, index, normal, o


def _implicit_frame(case, viewport):
    """One beauty frame of an implicit scene whose paths end at the first hit."""
    scene = _workload(case).scene
    s = 2 if case["ssaa"] else 1
    W, H = case["width"] * s, case["height"] * s
    P = viewport.camera.projection(case["width"], case["height"], case["ssaa"])
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    vec = lambda v: torch.tensor(np.asarray(v, np.float64), device=dev)   # noqa: E731
    xyz = lambda k: vec(P[k])                                             # noqa: E731
    y, x = torch.meshgrid(torch.arange(H, device=dev), torch.arange(W, device=dev), indexing="ij")
    x, y = x.reshape(-1), y.reshape(-1)
    d = _unit(xyz("start") + xyz("down") * y[:, None].double() + xyz("right") * x[:, None].double())
    eye = xyz("camera_position")
    distance, index, N, o = _trace(scene.geometries, eye.expand_as(d), d)
    hit = index >= 0
    position = o + d * torch.where(hit, distance, 0.0)[:, None]
    material = scene.materials[np.asarray(scene.geometries["material_id"])]
    pick = lambda k: vec(material[k])[index.clamp(min=0)]                 # noqa: E731
    albedo, rough, refl, brdf = pick("albedo"), pick("roughness"), pick("reflectivity"), pick("brdf")
    R = d - 2.0 * _dot(d, N)[:, None] * N
    color = torch.zeros_like(d)
    for light in scene.lights:
        to = vec(light["position"]) - position
        far = torch.sqrt(_dot(to, to))
        Ldir = to / far[:, None]
        cosine = torch.clamp(_dot(Ldir, N), 0.0, 1.0)
        blocked = _trace(scene.geometries, position, Ldir, True)[0] < far
        half = torch.clamp(_dot(N, _unit(Ldir - d)), 0.0, 1.0) ** 16
        mirror = torch.clamp(_dot(R, Ldir), 0.0, 1.0) ** 4
        spec = torch.where(brdf == L.BRDF_LAMBERT, 0.0, torch.where(brdf == L.BRDF_PHONG, mirror, half))
        f = albedo * (rough / math.pi)[:, None] + refl * (spec * (1.0 - rough))[:, None]
        add = f * vec(light["color"]) * (cosine * float(light["intensity"]) / far ** 2)[:, None]
        color = color + torch.where((hit & (cosine > 0) & ~blocked)[:, None], add, 0.0)
    reach = distance.clone()   # the glow of the lights themselves, up to the hit
    for light in scene.lights:
        intensity = float(light["intensity"])
        limit = reach * (64.0 / intensity)
        rc = (vec(light["position"]) - o) * (64.0 / intensity)
        b, c = _dot(d, rc), _dot(rc, rc) - 1.0
        h = b * b - c
        root = torch.sqrt(torch.clamp(h, min=0.0))
        seen = (h >= 0) & (b + root > 0) & (b - root < limit)
        tn, tf = torch.clamp(b - root, min=0.0), torch.minimum(b + root, limit)
        inside = lambda t: c * t - b * t * t + t ** 3 / 3.0               # noqa: E731
        density = 0.75 * (inside(tn) - inside(tf))
        reach = torch.where(seen, limit * (intensity / 64.0), reach)
        color = color + torch.where(seen[:, None], vec(light["color"]) * (4.0 * density ** 8)[:, None], 0.0)
    t = torch.clamp(color - 0.004, min=0.0)
    t = (6.2 * t * t + 0.5 * t) / (6.2 * t * t + 1.7 * t + 0.06)
    pixels = torch.cat([torch.clamp(t, 0.0, 1.0) ** 2, torch.ones_like(t[:, :1])], 1)
    m = xyz("inverted_camera_rotation").reshape(9)
    v = position - eye
    depth = torch.where(hit, m[2] * v[:, 0] + m[5] * v[:, 1] + m[8] * v[:, 2], math.inf)
    if case["ssaa"]:   # a pixel's four samples lie together
        order = (torch.div(y, 2, rounding_mode="floor") * case["width"] + torch.div(x, 2, rounding_mode="floor")) * 4 \
            + 2 * (y % 2) + x % 2
        pixels = torch.empty_like(pixels).index_copy_(0, order, pixels)
        depth = torch.empty_like(depth).index_copy_(0, order, depth)
    return pixels, depth
