"""Scenes of up to 32 BVH leaves are traced leaf by leaf instead of down the
tree: frames equal, bit for bit, those of the tree walk (which a frame that
counts its work takes), on implicit, textured and mesh scenes, for objects
that touch, for every leaf count around the limit, and after a GPU refit."""
import numpy as np
import pytest

from slimtracincpp_b200 import layout as L
from slimtracincpp_b200 import native, scenes
from slimtracincpp_b200.renderer import RayTracingRenderer, Viewport
from slimtracincpp_b200.scene import Camera, Scene, geometry, light

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def frame(w, engine, count_work, moved=False):
    native.set_render_options(engine=engine, count_work=count_work)
    try:
        st = w.settings
        r = RayTracingRenderer(w.scene, int(st["max_depth"]), int(st["skybox_color_texture_id"]),
                               int(st["skybox_radiance_texture_id"]), int(st["skybox_irradiance_texture_id"]))
        if moved:
            rest = w.scene.geometries.copy()
            w.scene.geometries["position"][1:] += np.float32(0.3)
            native.check(native.lib().slimUploadGeometries(w.scene.ptr))
            native.check(native.lib().slimRefitSceneBVH(0))
            w.scene.geometries[:] = rest
        n = w.width * w.height
        pixels, depths = torch.full((n, 4), -1.0, device="cuda"), torch.full((n,), -1.0, device="cuda")
        torch.cuda.synchronize()
        r.render_to_device(Viewport(w.camera, w.width, w.height), pixels.data_ptr(), depths.data_ptr())
        native.check(native.lib().slimSynchronize(0))
        return pixels.cpu().numpy().view(np.uint32), depths.cpu().numpy().view(np.uint32)
    finally:
        native.set_render_options(engine=L.ENGINE_AUTO)


def blocks(count):
    """`count` unit boxes side by side on a floor they touch, some of them in
    exactly the same place, seen along the axes."""
    materials = [L.default_material(albedo=0.8, roughness=0.6, brdf=L.BRDF_LAMBERT),
                 L.default_material(albedo=0.5, roughness=0.3, flags=L.MATERIAL_IS_REFLECTIVE, reflectivity=0.6)]
    kinds = [L.GEOMETRY_BOX, L.GEOMETRY_SPHERE, L.GEOMETRY_TET, L.GEOMETRY_QUAD]
    geos = [geometry(L.GEOMETRY_QUAD, 0, (0, 0, 0), (12, 1, 12))]
    for i in range(count - 1):
        j = i - 1 if i % 5 == 4 else i
        geos.append(geometry(kinds[0] if j % 2 else kinds[j % 4], i % 2, (2.0 * (j % 6) - 5.0, 1.0, 2.0 * (j // 6) - 3.0)))
    lights = [light((1, 1, 1), (0.0, -0.8, 0.6), 1.2, flags=L.LIGHT_IS_DIRECTIONAL | L.LIGHT_IS_SHADOWING),
              light((1, 0.8, 0.6), (-3.0, 5.0, -4.0), 15.0)]
    scene = Scene(np.array(geos), np.array(materials), np.array(lights))
    camera = Camera(np.eye(3, dtype=np.float32), np.array([0.0, 1.0, -11.0], np.float32), 1.2)
    return scenes.Workload("blocks", scene, camera, 97, 65, L.default_settings(max_depth=4))


def workload(name):
    return {"features": lambda: scenes.feature_scene(3, 96, 54, 4),
            "implicit": lambda: scenes.config1(5, 160, 90),
            "textured": lambda: scenes.small_textured_scene(2, 128, 72),
            "mesh": lambda: scenes.small_mesh_scene(1, 128, 72)}[name]()


@pytest.mark.parametrize("engine", [L.ENGINE_MEGAKERNEL, L.ENGINE_WAVEFRONT])
@pytest.mark.parametrize("name", ["features", "implicit", "textured", "mesh"])
def test_frames_equal_the_tree_walk(name, engine):
    w = workload(name)
    for moved in (False, True):
        a, b = frame(w, engine, False, moved), frame(w, engine, True, moved)
        assert len(np.unique(a[0])) > 100
        assert np.array_equal(a[1], b[1])
        assert np.array_equal(a[0], b[0])


@pytest.mark.parametrize("engine", [L.ENGINE_MEGAKERNEL, L.ENGINE_WAVEFRONT])
@pytest.mark.parametrize("count", [1, 2, 3, 31, 32, 33])
def test_touching_objects_around_the_limit(count, engine):
    w = blocks(count)
    a, b = frame(w, engine, False), frame(w, engine, True)
    assert np.array_equal(a[1], b[1])
    assert np.array_equal(a[0], b[0])
