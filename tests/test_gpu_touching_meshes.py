"""GPU: mesh instances that touch each other and implicit primitives.

Where two surfaces meet, the order in which the reference's walk reaches them
decides between hits at the same distance, and between a hit and one that
rounding puts in front of its own box.  The wavefront engine tests them in
another order and traces the rays in question whole: its frames equal the
fused engine's walk bit for bit, however its launches interleave, for few
rays (whose mesh walks are shared) and for many, near the origin, far from it
and for short rays there."""
import functools

import numpy as np
import pytest

from slimtracincpp_b200 import layout as L
from slimtracincpp_b200 import native, scenes
from slimtracincpp_b200.renderer import RayTracingRenderer, Viewport
from slimtracincpp_b200.scene import Camera, MeshAsset, Scene, geometry, light

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

REPEATS = 4
IN_A_BOX = ("in a box", "in a box, grouped")


def asset(builder, shift=0.0, raised=0):
    """The mesh, shifted along x; its vertices beyond 0.9 on the `raised` side of x lifted."""
    positions, indices, normals = builder
    positions = positions.copy()
    positions[:, 1] += np.float32(0.4) * (positions[:, 0] * raised > 0.9)
    positions[:, 0] += np.float32(shift)
    return MeshAsset.build(positions, indices, normals=normals, normal_indices=indices)


@functools.cache
def assets():
    flat = [asset(scenes.heightfield(np.random.default_rng(3), n, 0.0), shift, raised)
            for n, shift, raised in ((17, 0, 0), (24, 0, 0), (65, 0, -1), (65, 1.25, 1))]
    return [*flat, asset(scenes.icosphere(3))]


def touching_scene(kind, turned, far, side, distance):
    """The touching surfaces around `far`, seen from one side or the other, and
    spheres that split the scene BVH."""
    rng = np.random.default_rng(11)
    axis, amount = scenes.random_quat(rng) if turned else ((0, 0, 0), 1.0)
    at = np.array(far, np.float64)
    geos = []

    def put(what, material, scale=(1.0, 1.0, 1.0), mesh=0, shift=(0.0, 0.0, 0.0)):
        geos.append(geometry(what, material, tuple(at + np.array(shift)), scale, axis, amount, mesh_id=mesh))

    if kind == "coincident":        # meshes twice in the same place
        for material in (0, 1):
            put(L.GEOMETRY_MESH, material, mesh=4)
        put(L.GEOMETRY_MESH, 2, mesh=0)
        put(L.GEOMETRY_MESH, 1, mesh=0)
    elif kind == "overlapping":     # one transform, so the same distances, but other boxes
        put(L.GEOMETRY_MESH, 0, mesh=2)
        put(L.GEOMETRY_MESH, 1, mesh=3)
    elif kind == "quad beside":     # likewise; the mesh reaches beyond the quad
        put(L.GEOMETRY_QUAD, 0)
        put(L.GEOMETRY_MESH, 1, mesh=3)
    elif kind in IN_A_BOX:          # on its floor, seen from inside; the mesh's leaf comes first or second
        put(L.GEOMETRY_BOX, 0, (2.0, 1.0, 2.0), 0, (0.5 * side, 1.0, 0.0))
        put(L.GEOMETRY_MESH, 1)
        if kind == "in a box, grouped":     # the mesh's leaf is further down the BVH than the box's
            for x in (-0.3, 0.2, 0.4):
                put(L.GEOMETRY_SPHERE, 2, (0.05, 0.05, 0.05), 0, (x, 0.2, -0.9))
    elif kind == "mesh on quad":
        put(L.GEOMETRY_QUAD, 0, (1.3, 1.0, 1.1))
        put(L.GEOMETRY_MESH, 1, (1.0, 1.0, 1.0), 0)
        put(L.GEOMETRY_QUAD, 2, (0.6, 1.0, 0.7))
    elif kind == "quad aside":      # one of them first in the BVH, then the other
        put(L.GEOMETRY_QUAD, 0, shift=(0.4 * side, 0.0, 0.0))
        put(L.GEOMETRY_MESH, 1)
    elif kind == "mesh on mesh":
        put(L.GEOMETRY_MESH, 0, (1.0, 1.0, 1.0), 0, (0.3 * side, 0.0, 0.0))
        put(L.GEOMETRY_MESH, 1, (0.8, 0.7, 1.2), 1)
    else:                           # "mesh on box": flat meshes on a box's top and in its bottom
        put(L.GEOMETRY_BOX, 0, (0.9, 1.0, 0.8))
        if not turned:
            put(L.GEOMETRY_MESH, 1, (0.7, 1.0, 0.7), 0, (0.0, 1.0, 0.0))
            put(L.GEOMETRY_MESH, 2, (1.4, 1.0, 1.4), 1, (0.0, -1.0, 0.0))
        else:
            put(L.GEOMETRY_MESH, 1, (0.9, 1.0, 0.8), 4)
    for i in range(0 if kind in IN_A_BOX or kind == "quad aside" else 6):
        geos.insert(i // 2, geometry(L.GEOMETRY_SPHERE, i % 3, tuple(at + (2.0 * i - 5.0, 1.5 + 0.3 * i, 3.0)), 0.5))
    materials = [L.default_material(albedo=(0.9, 0.2, 0.2), roughness=0.6, brdf=L.BRDF_LAMBERT),
                 L.default_material(albedo=(0.2, 0.9, 0.2), roughness=0.2, flags=L.MATERIAL_IS_REFLECTIVE,
                                    reflectivity=0.6),
                 L.default_material(albedo=(0.2, 0.2, 0.9), roughness=0.4)]
    lights = [light((1, 1, 1), (0.2, -0.8, 0.5), 1.2, flags=L.LIGHT_IS_DIRECTIONAL | L.LIGHT_IS_SHADOWING),
              light((1, 0.8, 0.6), tuple(at + (-3.0, 6.0, -4.0)), 25.0)]
    camera = Camera.look_at(at + distance * np.array([2.6 * side, 1.4, -1.7]), at, 50.0)
    return Scene(np.array(geos), np.array(materials), np.array(lights), meshes=assets()), camera


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
@pytest.mark.parametrize("far,distance", [((0.0, 0.0, 0.0), 1.0), ((410.0, 130.0, -270.0), 1.0),
                                          ((410.0, 130.0, -270.0), 0.03)])
@pytest.mark.parametrize("side", [-1, 1])
@pytest.mark.parametrize("turned", [False, True])
@pytest.mark.parametrize("kind", ["coincident", "overlapping", "quad beside", "quad aside", *IN_A_BOX,
                                  "mesh on quad", "mesh on mesh", "mesh on box"])
def test_touching_surfaces_resolve_in_the_walks_order(kind, turned, side, far, distance, size):
    scene, camera = touching_scene(kind, turned, far, side, distance)
    view = Viewport(camera, *size)
    try:
        (pixels, depths), = frame(scene, view, L.ENGINE_MEGAKERNEL)
        assert distance < 1.0 or np.isfinite(depths.view(np.float32)).sum() > 50
        for p, d in frame(scene, view, L.ENGINE_WAVEFRONT):
            assert np.array_equal(d, depths)
            assert np.array_equal(p, pixels)
    finally:
        native.set_render_options(engine=L.ENGINE_AUTO)
