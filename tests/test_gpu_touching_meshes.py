"""GPU: mesh instances that touch each other and implicit primitives.

Where two surfaces meet, the order in which the reference's walk reaches them
decides between hits at the same distance, and between a hit and one that
rounding puts in front of its own box.  The wavefront engine tests them in
another order and traces the rays in question whole: its frames equal the
fused engine's walk bit for bit, however its launches interleave, for few
rays (whose mesh walks are shared) and for many, near the origin and for
short rays far from it."""
import numpy as np
import pytest

from slimtracincpp_b200 import layout as L
from slimtracincpp_b200 import native, scenes
from slimtracincpp_b200.renderer import RayTracingRenderer, Viewport
from slimtracincpp_b200.scene import Camera, MeshAsset, Scene, geometry, light

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

REPEATS = 4


def asset(builder):
    positions, indices, normals = builder
    return MeshAsset.build(positions, indices, normals=normals, normal_indices=indices)


def touching_scene(kind, turned, far):
    """The touching pair around `far`, and spheres that split the scene BVH."""
    rng = np.random.default_rng(11)
    axis, amount = scenes.random_quat(rng) if turned else ((0, 0, 0), 1.0)
    at = np.array(far, np.float64)
    flat = [asset(scenes.heightfield(np.random.default_rng(3), n, 0.0)) for n in (17, 24)]
    sphere = asset(scenes.icosphere(3))
    meshes = [flat[0], flat[1], sphere]
    geos = []

    def put(what, material, scale=(1.0, 1.0, 1.0), mesh=0, shift=(0.0, 0.0, 0.0)):
        geos.append(geometry(what, material, tuple(at + np.array(shift)), scale, axis, amount, mesh_id=mesh))

    if kind == "coincident":        # one mesh twice, and once more through an inner vertex ring
        for material in (0, 1):
            put(L.GEOMETRY_MESH, material, mesh=2)
        put(L.GEOMETRY_MESH, 2, mesh=0)
        put(L.GEOMETRY_MESH, 1, mesh=0)
    elif kind == "mesh on quad":
        put(L.GEOMETRY_QUAD, 0, (1.3, 1.0, 1.1))
        put(L.GEOMETRY_MESH, 1, (1.0, 1.0, 1.0), 0)
        put(L.GEOMETRY_QUAD, 2, (0.6, 1.0, 0.7))
    elif kind == "mesh on mesh":
        put(L.GEOMETRY_MESH, 0, (1.0, 1.0, 1.0), 0)
        put(L.GEOMETRY_MESH, 1, (0.8, 0.7, 1.2), 1)
    else:                           # "mesh on box": flat meshes on a box's top and in its bottom
        put(L.GEOMETRY_BOX, 0, (0.9, 1.0, 0.8))
        if not turned:
            put(L.GEOMETRY_MESH, 1, (0.7, 1.0, 0.7), 0, (0.0, 1.0, 0.0))
            put(L.GEOMETRY_MESH, 2, (1.4, 1.0, 1.4), 1, (0.0, -1.0, 0.0))
        else:
            put(L.GEOMETRY_MESH, 1, (0.9, 1.0, 0.8), 2)
    for i in range(6):
        geos.insert(i // 2, geometry(L.GEOMETRY_SPHERE, i % 3, tuple(at + (2.0 * i - 5.0, 1.5 + 0.3 * i, 3.0)), 0.5))
    materials = [L.default_material(albedo=(0.9, 0.2, 0.2), roughness=0.6, brdf=L.BRDF_LAMBERT),
                 L.default_material(albedo=(0.2, 0.9, 0.2), roughness=0.2, flags=L.MATERIAL_IS_REFLECTIVE,
                                    reflectivity=0.6),
                 L.default_material(albedo=(0.2, 0.2, 0.9), roughness=0.4)]
    lights = [light((1, 1, 1), (0.2, -0.8, 0.5), 1.2, flags=L.LIGHT_IS_DIRECTIONAL | L.LIGHT_IS_SHADOWING),
              light((1, 0.8, 0.6), tuple(at + (-3.0, 6.0, -4.0)), 25.0)]
    camera = Camera.look_at(at + (0.4, 1.7, -3.1), at, 50.0)
    return Scene(np.array(geos), np.array(materials), np.array(lights), meshes=meshes), camera


def frame(scene, view, engine):
    native.set_render_options(engine=engine)
    r = RayTracingRenderer(scene, 3)
    n = view.width * view.height
    out = []
    for _ in range(1 if engine == L.ENGINE_MEGAKERNEL else REPEATS):
        pixels, depths = torch.full((n, 4), -1.0, device="cuda"), torch.full((n,), -1.0, device="cuda")
        torch.cuda.synchronize()
        r.render_to_device(view, pixels.data_ptr(), depths.data_ptr())
        native.check(native.lib().slimSynchronize(0))
        out.append((pixels.cpu().numpy().view(np.uint32), depths.cpu().numpy().view(np.uint32)))
    return out


@pytest.mark.parametrize("size", [(49, 37), (513, 385)])
@pytest.mark.parametrize("far", [(0.0, 0.0, 0.0), (410.0, 130.0, -270.0)])
@pytest.mark.parametrize("turned", [False, True])
@pytest.mark.parametrize("kind", ["coincident", "mesh on quad", "mesh on mesh", "mesh on box"])
def test_touching_surfaces_resolve_in_the_walks_order(kind, turned, far, size):
    scene, camera = touching_scene(kind, turned, far)
    view = Viewport(camera, *size)
    try:
        (pixels, depths), = frame(scene, view, L.ENGINE_MEGAKERNEL)
        assert len(np.unique(pixels)) > 100
        for p, d in frame(scene, view, L.ENGINE_WAVEFRONT):
            assert np.array_equal(d, depths)
            assert np.array_equal(p, pixels)
    finally:
        native.set_render_options(engine=L.ENGINE_AUTO)
