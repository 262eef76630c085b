"""GPU: a frame captured into a caller's CUDA graph follows later uploads.

Geometries and the scene BVH are uploaded in place (same counts), so a replay
renders the scene as it is then: moved objects whose rebuilt BVH has its
leaves at other nodes, objects made visible or shadowing, and a refit.  Both
engines, with and without mesh instances, with and without allocations."""
import numpy as np
import pytest

from slimtracincpp_b200 import layout as L
from slimtracincpp_b200 import native, scenes
from slimtracincpp_b200.renderer import RayTracingRenderer, Viewport, make_canvas
from slimtracincpp_b200.scene import Camera, MeshAsset, Scene, geometry, light

torch = pytest.importorskip("torch")

WIDTH, HEIGHT, DEPTH = 161, 97, 3


def moved_objects(rng, with_meshes):
    """A dozen objects at random places over a floor."""
    geos = [geometry(L.GEOMETRY_QUAD, 0, (0, -1.5, 0), (14, 1, 14))]
    kinds = [L.GEOMETRY_BOX, L.GEOMETRY_SPHERE, L.GEOMETRY_TET, L.GEOMETRY_MESH]
    for i in range(12):
        kind = kinds[i % (4 if with_meshes else 3)]
        geos.append(geometry(kind, i % 2, tuple(rng.uniform((-6, -1, -3), (6, 3, 5))), mesh_id=0))
    return geos


def leaves_of(scene):
    n = scene.bvh_nodes[:int(scene.data["bvh_node_count"])]
    return tuple(np.nonzero(n["leaf_count"])[0])


def scene_of(with_meshes):
    materials = [L.default_material(albedo=0.8, roughness=0.6, brdf=L.BRDF_LAMBERT),
                 L.default_material(albedo=0.5, roughness=0.3, flags=L.MATERIAL_IS_REFLECTIVE, reflectivity=0.6)]
    lights = [light((1, 1, 1), (0.3, -0.8, 0.5), 1.2, flags=L.LIGHT_IS_DIRECTIONAL | L.LIGHT_IS_SHADOWING),
              light((1, 0.8, 0.6), (-3.0, 6.0, -4.0), 25.0)]
    meshes = []
    if with_meshes:
        positions, indices, normals = scenes.icosphere(2)
        meshes = [MeshAsset.build(positions, indices, normals=normals, normal_indices=indices)]
    return Scene(np.array(moved_objects(np.random.default_rng(5), with_meshes)), np.array(materials), np.array(lights),
                 meshes=meshes)


def other_leaves(scene, with_meshes):
    """Geometries in new places whose rebuilt BVH has as many nodes and leaves elsewhere."""
    before, count = leaves_of(scene), int(scene.data["bvh_node_count"])
    rest = scene.geometries.copy()
    for seed in range(6, 400):
        scene.geometries[:] = np.array(moved_objects(np.random.default_rng(seed), with_meshes))
        scene.build_bvh()
        if int(scene.data["bvh_node_count"]) == count and leaves_of(scene) != before:
            out = scene.geometries.copy()
            scene.geometries[:] = rest
            scene.build_bvh()
            return out
    raise AssertionError("every rebuild has the same leaves")


@pytest.mark.parametrize("with_meshes", [False, True])
def test_rebuilds_move_the_leaves(with_meshes):
    scene = scene_of(with_meshes)
    before = leaves_of(scene)
    scene.geometries[:] = other_leaves(scene, with_meshes)
    scene.build_bvh()
    assert leaves_of(scene) != before


@pytest.mark.gpu
@pytest.mark.parametrize("no_alloc", [False, True])
@pytest.mark.parametrize("with_meshes", [False, True])
@pytest.mark.parametrize("engine", [L.ENGINE_MEGAKERNEL, L.ENGINE_WAVEFRONT])
@pytest.mark.parametrize("change", ["moved", "visible", "shadowing", "refit"])
def test_replays_follow_the_uploads(change, engine, with_meshes, no_alloc):
    scene = scene_of(with_meshes)
    flags = {"visible": L.GEOMETRY_IS_SHADOWING, "shadowing": L.GEOMETRY_IS_VISIBLE}
    if change in flags:
        scene.geometries["flags"][1:] = flags[change]
    camera = Camera(np.eye(3, dtype=np.float32), np.array([0.0, 1.0, -11.0], np.float32), 1.4)
    view = Viewport(camera, WIDTH, HEIGHT)
    canvas, _, _ = make_canvas(WIDTH, HEIGHT, view.antialias)
    projection = camera.projection(WIDTH, HEIGHT)
    stream = torch.cuda.Stream()
    n = WIDTH * HEIGHT

    def buffers():
        return torch.full((n, 4), -1.0, device="cuda"), torch.full((n,), -1.0, device="cuda")

    def render(target):
        call = native.lib().slimRenderToDeviceNoAlloc if no_alloc else native.lib().slimRenderToDevice
        native.check(call(native.ptr(canvas), native.ptr(projection), native.ptr(r.settings), target[0].data_ptr(),
                          target[1].data_ptr(), stream.cuda_stream))

    try:
        native.set_render_options(engine=engine)
        r = RayTracingRenderer(scene, DEPTH)
        before, replayed, direct = buffers(), buffers(), buffers()
        torch.cuda.synchronize()
        render(before)
        native.check(native.lib().slimSynchronize(stream.cuda_stream))
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            render(replayed)
        if change in flags:
            scene.geometries["flags"][1:] = L.GEOMETRY_IS_VISIBLE | L.GEOMETRY_IS_SHADOWING
        else:
            scene.geometries[:] = other_leaves(scene, with_meshes)
        native.check(native.lib().slimUploadGeometries(scene.ptr))
        if change == "moved":
            scene.build_bvh()
            native.check(native.lib().slimUploadSceneBVH(scene.ptr))
        if change == "refit":
            native.check(native.lib().slimRefitSceneBVH(0))
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        render(direct)
        native.check(native.lib().slimSynchronize(stream.cuda_stream))
    finally:
        native.set_render_options(engine=L.ENGINE_AUTO)
    for a, b, c in zip(before, replayed, direct):
        a, b, c = (t.cpu().numpy().view(np.uint32) for t in (a, b, c))
        assert a.shape == c.shape and (change == "shadowing" and a.ndim == 1 or not np.array_equal(a, c))
        assert np.array_equal(b, c)
