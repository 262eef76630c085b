"""GPU: launches of many rays test the leaves of a scene one by one up to 16
leaves, launches of few up to 32.  Frames equal the tree walk's (which a frame
that counts its work takes) on both sides of either limit."""
import numpy as np
import pytest

from slimtracincpp_b200 import layout as L
from test_gpu_listed_leaves import blocks, frame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine", [L.ENGINE_MEGAKERNEL, L.ENGINE_WAVEFRONT])
@pytest.mark.parametrize("width,height", [(512, 512), (521, 512)])      # 2^18 rays are few
@pytest.mark.parametrize("count", [16, 17, 32])
def test_frames_equal_the_tree_walk(count, width, height, engine):
    w = blocks(count)
    w.width, w.height = width, height
    a, b = frame(w, engine, False), frame(w, engine, True)
    assert len(np.unique(a[0])) > 100
    assert np.array_equal(a[1], b[1])
    assert np.array_equal(a[0], b[0])
