"""The persistent mesh walks over the four-wide BVH against the walk over the
binary one: the wavefront engine's frames equal the fused engine's bit for
bit, for rays parallel to an axis, flat meshes, leaves of more than two
triangles and boxes that do not nest (which have no wide form)."""
import numpy as np
import pytest

from slimtracincpp_b200 import layout as L
from slimtracincpp_b200 import native, scenes
from slimtracincpp_b200.renderer import RayTracingRenderer, Viewport
from slimtracincpp_b200.scene import Camera, MeshAsset, Scene, geometry, light

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def merged_leaves(mesh, most):
    """The mesh with the bottom of its BVH merged to leaves of up to `most` triangles."""
    nodes, out, stack = mesh.nodes, [mesh.nodes[0].copy()], [(0, 0)]

    def span(i):
        n = nodes[i]
        if n["leaf_count"]:
            return int(n["first_index"]), int(n["leaf_count"])
        (a, ca), (b, cb) = span(int(n["first_index"])), span(int(n["first_index"]) + 1)
        return min(a, b), ca + cb

    while stack:
        src, dst = stack.pop()
        first, count = span(src)
        if count <= most:
            out[dst]["first_index"], out[dst]["leaf_count"] = first, count
            continue
        out[dst]["first_index"] = len(out)
        for c in (int(nodes[src]["first_index"]), int(nodes[src]["first_index"]) + 1):
            out.append(nodes[c].copy())
            stack.append((c, len(out) - 1))
    mesh.nodes = np.array(out, L.BVH_NODE)
    return mesh


def meshes(kind):
    sphere = scenes.icosphere(3)
    field = scenes.heightfield(np.random.default_rng(3), 17, 0.0 if kind == "flat" else 0.3)
    out = [MeshAsset.build(p, i, normals=n, normal_indices=i) for p, i, n in (sphere, field)]
    if kind == "wide leaves":
        out = [merged_leaves(m, 7) for m in out]
    if kind == "not nested":
        k = len(out[0].nodes) // 2
        out[0].nodes[k]["max"] += np.float32(0.25)
    return out


@pytest.mark.parametrize("turned", [False, True])
@pytest.mark.parametrize("kind", ["plain", "flat", "wide leaves", "not nested"])
def test_frames_equal_the_binary_walks(kind, turned):
    rng = np.random.default_rng(4)
    # unturned instances and a straight camera: the centre column and row of
    # primary rays, and every shadow ray of the first light, are parallel to
    # an axis of the meshes' own spaces
    mirror = L.default_material(albedo=0.4, roughness=0.2, flags=L.MATERIAL_IS_REFLECTIVE, reflectivity=0.5)
    materials = [L.default_material(albedo=0.7, roughness=0.5), mirror]
    geos = []
    for i in range(6):
        axis, amount = scenes.random_quat(rng) if turned else ((0, 0, 0), 1.0)
        geos.append(geometry(L.GEOMETRY_MESH, i % 2, (-3 + 3 * (i % 3), 1.0 + 2.0 * (i // 3), float(i // 3)),
                             (1.2, 1.0, 1.2), axis, amount, mesh_id=(i + i // 3) % 2))
    lights = [light((1, 0.9, 0.8), (0.0, -0.8, 0.6), 1.5, flags=L.LIGHT_IS_DIRECTIONAL | L.LIGHT_IS_SHADOWING),
              light((0.5, 0.7, 1.0), (2.0, 6.0, -3.0), 20.0)]
    scene = Scene(np.array(geos), np.array(materials), np.array(lights), meshes=meshes(kind))
    camera = Camera(np.eye(3, dtype=np.float32), np.array([0.0, 2.0, -9.0], np.float32), 1.6)
    view = Viewport(camera, 129, 97)
    frames = []
    try:
        for engine in (L.ENGINE_MEGAKERNEL, L.ENGINE_WAVEFRONT):
            native.set_render_options(engine=engine)
            r = RayTracingRenderer(scene, max_depth=3)
            pixels = torch.full((129 * 97, 4), -1.0, device="cuda")
            depths = torch.full((129 * 97,), -1.0, device="cuda")
            r.render_to_device(view, pixels.data_ptr(), depths.data_ptr())
            native.check(native.lib().slimSynchronize(0))
            frames.append((pixels.cpu().numpy().view(np.uint32), depths.cpu().numpy().view(np.uint32)))
    finally:
        native.set_render_options(engine=L.ENGINE_AUTO)
    assert len(np.unique(frames[0][0])) > 100
    assert np.array_equal(frames[0][1], frames[1][1])
    assert np.array_equal(frames[0][0], frames[1][0])
