"""GPU: a frame captured into a caller's CUDA graph outlives an upload of other
meshes of the same sizes.  Every array of the scene stays in place then, those
of the four-wide mesh BVHs too, although they may hold more nodes than before."""
import numpy as np
import pytest

from slimtracincpp_b200 import layout as L
from slimtracincpp_b200 import native, scenes
from slimtracincpp_b200.renderer import RayTracingRenderer, Viewport
from slimtracincpp_b200.scene import Camera, MeshAsset, Scene, geometry, light

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def scene_of(seed):
    """A heightfield of 512 triangles and 511 BVH nodes: 89 four-wide nodes of
    seed 0, 107 of seed 8."""
    positions, indices, normals = scenes.heightfield(np.random.default_rng(seed), 17, 0.3)
    mesh = MeshAsset.build(positions, indices, normals=normals, normal_indices=indices)
    assert len(mesh.nodes) == 511
    geos = [geometry(L.GEOMETRY_MESH, 0, (x, 0.0, 1.0), 1.4) for x in (-1.5, 1.5)]
    lights = [light((1, 0.9, 0.8), (0.3, -0.8, 0.6), 1.5, flags=L.LIGHT_IS_DIRECTIONAL | L.LIGHT_IS_SHADOWING)]
    return Scene(np.array(geos), np.array([L.default_material(albedo=0.7, roughness=0.5)]), np.array(lights),
                 meshes=[mesh])


def test_replay_after_uploading_other_meshes():
    view = Viewport(Camera.look_at((0.0, 2.5, -5.0), (0.0, 0.0, 0.0), 50.0), 129, 97)
    n = view.width * view.height
    stream = torch.cuda.Stream()
    direct, replayed = [(torch.full((n, 4), -1.0, device="cuda"), torch.full((n,), -1.0, device="cuda"))
                        for _ in range(2)]
    torch.cuda.synchronize()

    def render(r, target):
        r.render_to_device(view, target[0].data_ptr(), target[1].data_ptr(), stream.cuda_stream)

    try:
        native.set_render_options(engine=L.ENGINE_WAVEFRONT)
        first = RayTracingRenderer(scene_of(0), 3)
        render(first, direct)
        native.check(native.lib().slimSynchronize(stream.cuda_stream))
        before = direct[0].cpu().numpy()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            render(first, replayed)
        second = RayTracingRenderer(scene_of(8), 3)
        graph.replay()
        torch.cuda.synchronize()
        render(second, direct)
        native.check(native.lib().slimSynchronize(stream.cuda_stream))
    finally:
        native.set_render_options(engine=L.ENGINE_AUTO)
    assert not np.array_equal(before, direct[0].cpu().numpy())
    for a, b in zip(direct, replayed):
        assert np.array_equal(a.cpu().numpy().view(np.uint32), b.cpu().numpy().view(np.uint32))
