"""GPU: a frame's training set is dealt out to its Adam steps in turn.

The set lies in the order in which the frame's blocks appended their queries, so
a step over a contiguous part of it sees one region of the picture only.  With a
learning rate of nothing the weights stand still, and the loss that the frame's
last step reports is that of its part: near the whole set's, however the set is
divided."""
import numpy as np
import pytest

from slimtracincpp_b200 import layout as L
from slimtracincpp_b200 import native, scenes
from slimtracincpp_b200.radiance_cache import RadianceCache
from slimtracincpp_b200.renderer import RayTracingRenderer, Viewport

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def losses(batches, overlap):
    """The last step's loss and the steps taken, per batch size (as a share of the queries)."""
    w = scenes.small_textured_scene(1, 256, 144, max_depth=6)
    st = w.settings
    view = Viewport(w.camera, w.width, w.height)
    n = w.width * w.height
    pixels, depths = torch.empty((n, 4), device="cuda"), torch.empty((n,), device="cuda")
    r = RayTracingRenderer(w.scene, int(st["max_depth"]), int(st["skybox_color_texture_id"]),
                           int(st["skybox_radiance_texture_id"]), int(st["skybox_irradiance_texture_id"]))
    out, queries = [], 0
    try:
        for share in batches:
            batch = int(np.ceil(share * queries)) if queries else 1 << 16
            cache = RadianceCache.configure(cache_depth=2, train_samples=1 << 16, batch=batch, seed=3,
                                            learning_rate=1e-20, overlap=overlap)
            native.set_render_options(engine=L.ENGINE_WAVEFRONT, radiance_cache=L.CACHE_ON)
            r.render_to_device(view, pixels.data_ptr(), depths.data_ptr())
            native.check(native.lib().slimSynchronize(0))
            s = cache.stats()
            assert s["queries"] == s["train_samples"] > 1000
            queries = s["queries"]
            out.append((s["loss"], s["steps"]))
    finally:
        native.set_render_options(engine=L.ENGINE_WAVEFRONT)
    return out, queries


@pytest.mark.parametrize("overlap", [False, True])
def test_last_step_sees_the_whole_picture(overlap):
    shares = (1.0, 1.0, 0.97, 0.5, 0.33, 0.24)
    out, queries = losses(shares, overlap)
    whole = out[0][0]
    for share, (loss, steps) in zip(shares, out):
        parts = int(np.ceil(queries / np.ceil(share * queries)))
        assert steps == parts
        # a part holds a quarter of the set at least; the spread of its mean is
        # well below a tenth for samples in no order
        assert abs(loss - whole) < 0.1 * whole, (share, loss, whole)
