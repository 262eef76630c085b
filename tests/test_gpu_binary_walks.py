"""GPU: meshes whose BVH has no four-wide form are walked by the same persistent
kernels over the binary one.

Such are BVHs with a box outside its parent's and lopsided ones whose four-wide
walk could have more than 64 nodes waiting; one of them in a scene takes every
mesh to the binary walks.  Frames equal the fused engine's bit for bit, for
shared walks (few rays) and others, and take nowhere near the time of tracing
every ray whole."""
import numpy as np
import pytest

from slimtracincpp_b200 import layout as L
from slimtracincpp_b200 import native, scenes
from slimtracincpp_b200.renderer import RayTracingRenderer, Viewport
from slimtracincpp_b200.scene import Camera, MeshAsset, Scene, geometry, light

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def tower(levels=52, shrink=0.7):
    """Ever smaller squares in front of one another; level k's BVH node has a
    node of square k's two triangles, the larger box, and level k + 1's."""
    size = shrink ** np.arange(levels)
    depth = 0.3 * (1.0 - size)
    corners = np.array([(-1, -1), (1, -1), (1, 1), (-1, 1)], np.float64)
    positions = np.concatenate([corners[None] * size[:, None, None], np.repeat(-depth, 4).reshape(-1, 4, 1)], 2)
    quad = np.arange(4 * levels, dtype=np.uint32).reshape(-1, 4)
    mesh = MeshAsset.build(positions.reshape(-1, 3).astype(np.float32),
                           np.concatenate([quad[:, [0, 1, 2]], quad[:, [0, 2, 3]]]))
    mesh.triangles = mesh.triangles[np.argsort(-np.abs(mesh.triangles["position"][:, 0]), kind="stable")].copy()
    half, z = np.abs(mesh.triangles["position"][::2, 0]), mesh.triangles["position"][::2, 2]      # as built
    nodes = [np.zeros((), L.BVH_NODE)]

    def put(i, k, count, first=None):
        """Node i: `count` levels from k on; children next, or a leaf of triangle `first`."""
        nodes[i]["min"] = (-half[k], -half[k], z[k + count - 1])
        nodes[i]["max"] = (half[k], half[k], z[k])
        if first is not None:
            nodes[i]["first_index"], nodes[i]["leaf_count"] = first, 1
        else:
            nodes[i]["first_index"] = len(nodes)
            nodes.extend(np.zeros((), L.BVH_NODE) for _ in range(2))
            return len(nodes) - 2

    def square(i, k):
        c = put(i, k, 1)
        put(c, k, 1, 2 * k)
        put(c + 1, k, 1, 2 * k + 1)

    at = 0
    for k in range(levels - 1):
        c = put(at, k, levels - k)
        square(c, k)
        at = c + 1
    square(at, levels - 1)
    mesh.nodes = np.array(nodes, L.BVH_NODE)
    mesh.height = levels + 1
    return mesh


def assets(kind):
    out = [MeshAsset.build(p, i, normals=n, normal_indices=i)
           for p, i, n in (scenes.icosphere(4), scenes.heightfield(np.random.default_rng(3), 65, 0.3))]
    if kind == "not nested":
        out[0].nodes[len(out[0].nodes) // 2]["max"] += np.float32(0.25)
    if kind == "lopsided":
        out.append(tower())
    return out


def scene_of(kind):
    meshes = assets(kind)
    rng = np.random.default_rng(4)
    mirror = L.default_material(albedo=0.4, roughness=0.2, flags=L.MATERIAL_IS_REFLECTIVE, reflectivity=0.5)
    geos = [geometry(L.GEOMETRY_QUAD, 0, (0, -0.5, 0), (9, 1, 9))]
    for i in range(8):
        axis, amount = scenes.random_quat(rng) if i % 2 else ((0, 0, 0), 1.0)
        geos.append(geometry(L.GEOMETRY_MESH, i % 2, (-3 + 2 * (i % 4), 0.6 + 2.0 * (i // 4), float(i // 4)),
                             (1.2, 1.0, 1.2), axis, amount, mesh_id=(i + i // 4) % len(meshes)))
    lights = [light((1, 0.9, 0.8), (0.3, -0.8, 0.6), 1.5, flags=L.LIGHT_IS_DIRECTIONAL | L.LIGHT_IS_SHADOWING),
              light((0.5, 0.7, 1.0), (2.0, 6.0, -3.0), 20.0)]
    camera = Camera(np.eye(3, dtype=np.float32), np.array([0.0, 1.6, -8.0], np.float32), 1.6)
    materials = [L.default_material(albedo=0.7, roughness=0.5), mirror]
    return Scene(np.array(geos), np.array(materials), np.array(lights), meshes=meshes), camera


def rendered(r, view):
    n = view.width * view.height
    pixels, depths = torch.full((n, 4), -1.0, device="cuda"), torch.full((n,), -1.0, device="cuda")
    torch.cuda.synchronize()
    r.render_to_device(view, pixels.data_ptr(), depths.data_ptr())
    native.check(native.lib().slimSynchronize(0))
    return pixels.cpu().numpy().view(np.uint32), depths.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("size", [(65, 49), (641, 481)])
@pytest.mark.parametrize("kind", ["not nested", "lopsided"])
def test_frames_equal_the_fused_engines(kind, size):
    scene, camera = scene_of(kind)
    view = Viewport(camera, *size)
    try:
        native.set_render_options(engine=L.ENGINE_MEGAKERNEL)
        r = RayTracingRenderer(scene, 4)
        pixels, depths = rendered(r, view)
        assert len(np.unique(pixels)) > 500
        for count_work in (False, True):
            native.set_render_options(engine=L.ENGINE_WAVEFRONT, count_work=count_work)
            for _ in range(3):
                p, d = rendered(r, view)
                assert np.array_equal(d, depths)
                assert np.array_equal(p, pixels)
    finally:
        native.set_render_options(engine=L.ENGINE_AUTO)


def test_not_traced_whole():
    """The headline frame with one box of each mesh outside its parent's: 1.3
    times the time of the wide walks; 2.8 times when each ray was traced whole."""
    w = scenes.config2()
    view = Viewport(w.camera, 1920, 1080)
    n = view.width * view.height
    pixels, depths = torch.empty((n, 4), device="cuda"), torch.empty((n,), device="cuda")
    stream = torch.cuda.Stream()
    times = []
    for nested in (True, False):
        if not nested:
            for m in w.scene.meshes:
                m.nodes[len(m.nodes) // 2]["max"] += np.float32(1e-2)
        r = RayTracingRenderer(w.scene, 2)
        taken = []
        for _ in range(12):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            r.render_to_device(view, pixels.data_ptr(), depths.data_ptr(), stream.cuda_stream)
            b.record(stream)
            native.check(native.lib().slimSynchronize(stream.cuda_stream))
            taken.append(a.elapsed_time(b))
        times.append(float(np.median(taken[3:])))
    assert times[1] < 2.0 * times[0], times
