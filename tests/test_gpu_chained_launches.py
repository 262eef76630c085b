"""GPU: a frame's launches follow one another without the gap of a full
hand-over.  Frames whose launches are handed over in full -- with stage
events between them, or captured into a graph -- have the same pixels and
depths bit for bit, from canvases of a few warps to banded ones, with and
without meshes, also straight after a GPU refit and for frames in a row."""
import numpy as np
import pytest

from slimtracincpp_b200 import layout as L
from slimtracincpp_b200 import native, scenes
from slimtracincpp_b200.renderer import RayTracingRenderer, Viewport

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def workload(name, width, height):
    if name == "textured":
        return scenes.small_textured_scene(2, width, height)
    return scenes.feature_scene(3, width, height, 4)


@pytest.mark.parametrize("name", ["features", "textured"])
@pytest.mark.parametrize("width,height", [(7, 5), (97, 65), (640, 480), (1025, 771)])
def test_chained_frames_equal_unchained(name, width, height):
    w = workload(name, width, height)
    st = w.settings
    depth = 8
    stream = torch.cuda.Stream()
    n = width * height
    out = [(torch.full((n, 4), -1.0, device="cuda"), torch.full((n,), -1.0, device="cuda")) for _ in range(3)]
    torch.cuda.synchronize()

    def render(target):
        r.render_to_device(Viewport(w.camera, width, height), target[0].data_ptr(), target[1].data_ptr(),
                           stream.cuda_stream)

    try:
        native.set_render_options(engine=L.ENGINE_WAVEFRONT)
        r = RayTracingRenderer(w.scene, depth, int(st["skybox_color_texture_id"]),
                               int(st["skybox_radiance_texture_id"]), int(st["skybox_irradiance_texture_id"]))
        native.check(native.lib().slimRefitSceneBVH(stream.cuda_stream))
        for _ in range(3):
            render(out[0])
        native.set_render_options(engine=L.ENGINE_WAVEFRONT, profile_stages=True)
        render(out[1])
        native.set_render_options(engine=L.ENGINE_WAVEFRONT)
        native.check(native.lib().slimSynchronize(stream.cuda_stream))
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            render(out[2])
        graph.replay()
        torch.cuda.synchronize()
    finally:
        native.set_render_options(engine=L.ENGINE_AUTO)
    first = [t.cpu().numpy().view(np.uint32) for t in out[0]]
    assert (first[0] != np.float32(-1.0).view(np.uint32)).any()
    for other in out[1:]:
        for a, b in zip(first, other):
            assert np.array_equal(a, b.cpu().numpy().view(np.uint32))
