"""GPU: radiance-cache queries and training steps with more tiles than CTAs.

A query's CTAs hold three groups with a tile each, and tiles go round the CTAs
first: groups beyond the first work only past two tiles per SM, and a group
takes a second tile only past six.  Rows are independent, so a large query
equals the same rows asked in slices that one group of each CTA answers, bit for
bit.  A training CTA takes a second tile past one per SM."""
import numpy as np
import pytest

from oracle import nrc_oracle as N
from slimtracincpp_b200 import scenes
from slimtracincpp_b200.radiance_cache import RadianceCache
from slimtracincpp_b200.renderer import RayTracingRenderer

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

TILE = 128


@pytest.fixture(scope="module")
def cache():
    w = scenes.feature_scene(0, 32, 18)
    RayTracingRenderer(w.scene, max_depth=2)
    return RadianceCache.configure(seed=1)


def features(rng, n):
    f = np.zeros((n, 16), np.float32)
    f[:, 0:3] = rng.uniform(0, 1, (n, 3))
    f[:, 3] = rng.uniform(0.05, 1, n)
    for at in (4, 8):
        v = rng.normal(size=(n, 3))
        f[:, at:at + 3] = v / np.linalg.norm(v, axis=1, keepdims=True)
    f[:, 12:15] = rng.uniform(0, 1, (n, 3))
    return f


def params(rng):
    return N.pack([rng.uniform(-1, 1, s) * np.sqrt(6.0 / s[1]) for s in N.SHAPES]).astype(np.float32)


def sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("tiles_per_sm,odd", [(2, 1), (4, 77), (6, 77), (13, 5)])
def test_large_queries_equal_small_ones(cache, tiles_per_sm, odd):
    rng = np.random.default_rng(tiles_per_sm)
    weights = params(rng)
    cache.weights = weights
    n = tiles_per_sm * sms() * TILE + odd
    f = features(rng, n)
    df = torch.from_numpy(f).cuda()
    whole, sliced = torch.full((2, n + 1, 4), -1.0, device="cuda")
    torch.cuda.synchronize()
    cache.query(df.data_ptr(), n, whole.data_ptr())
    step = 40 * TILE
    for o in range(0, n, step):
        cache.query(df[o:].data_ptr(), min(step, n - o), sliced[o:].data_ptr())
    torch.cuda.synchronize()
    assert torch.equal(whole, sliced)
    assert (whole[n] == -1.0).all() and (whole[:n, :3] >= 0.0).all()
    rows = rng.integers(0, n, 500)
    rows[-1] = n - 1
    err = np.abs(np.log(whole.cpu().numpy()[rows, :3] + N.LOG_OFFSET) - np.log(N.infer(weights, f[rows]) + N.LOG_OFFSET))
    assert err.max() < 0.05 and np.quantile(err, 0.99) < 5e-3       # the bars of test_gpu_nrc.py


def test_gradients_of_several_tiles_per_cta(cache):
    rng = np.random.default_rng(5)
    weights = params(rng)
    cache.weights = weights
    n = 2 * sms() * TILE + 77
    f, t = features(rng, n), rng.uniform(0, 2, (n, 4)).astype(np.float32)
    df, dt = torch.from_numpy(f).cuda(), torch.from_numpy(t).cuda()
    torch.cuda.synchronize()
    cache.train(df.data_ptr(), dt.data_ptr(), n)
    torch.cuda.synchronize()
    g = cache.gradients()
    ref, loss = N.gradients(weights, f, t)
    o = 0
    for r, c in N.SHAPES:
        a, b = g[o:o + r * c], ref[o:o + r * c]
        assert np.linalg.norm(a - b) < 2e-2 * np.linalg.norm(b), (r, c)
        o += r * c
    assert abs(cache.stats()["loss"] - loss) <= 1e-3 * loss
