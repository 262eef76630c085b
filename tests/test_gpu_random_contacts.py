"""GPU: random scenes of objects on a coarse grid, so that many touch, overlap or
coincide, near the origin and far from it, of 2 to 40 objects: every engine's
frames equal the tree walk's of a fused frame that counts its work, bit for bit."""
import functools

import numpy as np
import pytest

from slimtracincpp_b200 import layout as L
from slimtracincpp_b200 import native, scenes
from slimtracincpp_b200.renderer import RayTracingRenderer, Viewport
from slimtracincpp_b200.scene import Camera, MeshAsset, Scene, geometry, light

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@functools.cache
def assets():
    corners = np.array([[x, y, z] for x in (-1, 1) for y in (-1, 1) for z in (-1, 1)], np.float32)
    sides = [(0, 1, 3, 2), (4, 6, 7, 5), (0, 4, 5, 1), (2, 3, 7, 6), (0, 2, 6, 4), (1, 5, 7, 3)]
    cube = corners, np.array([t for a, b, c, d in sides for t in ((a, b, c), (a, c, d))], np.uint32)
    flat = scenes.heightfield(np.random.default_rng(1), 13, 0.0)
    hills = scenes.heightfield(np.random.default_rng(2), 17, 0.3)
    return [MeshAsset.build(m[0], m[1]) for m in (cube, scenes.icosphere(2), flat, hills)]


def random_scene(rng):
    far = np.zeros(3) if rng.random() < 0.6 else rng.integers(-500, 500, 3).astype(float)
    kinds = [L.GEOMETRY_MESH, L.GEOMETRY_MESH, L.GEOMETRY_BOX, L.GEOMETRY_SPHERE, L.GEOMETRY_TET, L.GEOMETRY_QUAD]
    geos = []
    for _ in range(int(rng.choice([2, 4, 7, 12, 20, 31, 40]))):
        scale = tuple(float(x) for x in rng.choice([0.5, 1.0, 1.0, 1.5], 3)) if rng.random() < 0.5 else (1.0, 1.0, 1.0)
        turn = rng.random()
        axis, amount = [np.float32(0)] * 3, np.float32(1)
        if turn >= 0.8:
            axis, amount = scenes.random_quat(rng)
        elif turn >= 0.6:                       # a quarter turn about an axis
            axis[int(rng.integers(3))] = amount = np.float32(np.sqrt(0.5))
        flags = L.GEOMETRY_IS_VISIBLE | L.GEOMETRY_IS_SHADOWING
        if rng.random() < 0.15:
            flags |= L.GEOMETRY_IS_TRANSPARENT
        geos.append(geometry(int(rng.choice(kinds)), int(rng.integers(4)), tuple(far + rng.integers(-4, 5, 3) * 0.5),
                             scale, tuple(axis), amount, mesh_id=int(rng.integers(4)), flags=flags))
    M = L.default_material
    materials = [M(albedo=(0.9, 0.2, 0.2), roughness=0.6, brdf=L.BRDF_LAMBERT),
                 M(albedo=(0.2, 0.9, 0.2), roughness=0.2, flags=L.MATERIAL_IS_REFLECTIVE, reflectivity=0.6),
                 M(albedo=(0.2, 0.2, 0.9), roughness=0.4),
                 M(albedo=0.05, roughness=0.25, flags=L.MATERIAL_IS_REFRACTIVE, ior=1.5, reflectivity=0.03)]
    sun = (0.2, -0.8, 0.5) if rng.random() < 0.5 else (0.0, -1.0, 0.0)
    lights = [light((1, 1, 1), sun, 1.2, flags=L.LIGHT_IS_DIRECTIONAL | L.LIGHT_IS_SHADOWING),
              light((1, 0.8, 0.6), tuple(far + rng.integers(-4, 5, 3) + 0.25), 25.0)]
    if rng.random() < 0.4:
        camera = Camera(np.eye(3, dtype=np.float32), (far + (0, 0.5 * rng.integers(-2, 3), -5.0)).astype(np.float32), 1.3)
    else:
        at = far + rng.normal(size=3) * float(rng.choice([0.3, 2.0, 5.0])) + (0.01, 0, 0.02)
        camera = Camera.look_at(at, far, 60.0)
    return Scene(np.array(geos), np.array(materials), np.array(lights), meshes=assets()), camera


def frame(scene, view, depth, engine, count_work):
    native.set_render_options(engine=engine, count_work=count_work)
    r = RayTracingRenderer(scene, depth)
    n = view.width * view.height
    pixels, depths = torch.full((n, 4), -1.0, device="cuda"), torch.full((n,), -1.0, device="cuda")
    torch.cuda.synchronize()
    r.render_to_device(view, pixels.data_ptr(), depths.data_ptr())
    native.check(native.lib().slimSynchronize(0))
    return pixels.cpu().numpy().view(np.uint32), depths.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("block", range(6))
def test_engines_agree(block):
    try:
        for seed in range(25 * block, 25 * block + 25):
            rng = np.random.default_rng(seed)
            scene, camera = random_scene(rng)
            width, height = [(49, 37), (97, 65), (301, 211), (641, 487)][int(rng.choice(4, p=[0.35, 0.3, 0.25, 0.1]))]
            view, depth = Viewport(camera, width, height), int(rng.integers(1, 6))
            pixels, depths = frame(scene, view, depth, L.ENGINE_MEGAKERNEL, True)
            for engine, count_work in ((L.ENGINE_MEGAKERNEL, False), (L.ENGINE_WAVEFRONT, False),
                                       (L.ENGINE_WAVEFRONT, False), (L.ENGINE_WAVEFRONT, True)):
                p, d = frame(scene, view, depth, engine, count_work)
                assert np.array_equal(d, depths) and np.array_equal(p, pixels), (seed, engine, count_work)
    finally:
        native.set_render_options(engine=L.ENGINE_AUTO)
