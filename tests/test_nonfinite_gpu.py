"""Directions and cameras that no walk through EMPTY boxes may judge: NaN,
infinite, or so long that the time per voxel underflows.  What such a ray samples
is what the sampler makes of its positions (NaN for NaN); the march, and the
passes that settle a large view's misses, must answer as the general path (the
full sampler, no EMPTY space) does."""
import itertools

import numpy as np
import pytest

from conftest import assert_bits_equal
from test_multi_empty_gpu import _scene_objects
from test_settle_gpu import _both
from test_tiled_gpu import _params

pytestmark = pytest.mark.gpu

RATES = [np.nan, np.inf, -np.inf, 3e38, -1e38, 1e30, -1e20, 1e17, 0.0, 1e-12, -1e-44, 0.6, -0.8]


@pytest.fixture(scope="module", params=[False, True], ids=["one", "several"])
def scene(request, small_scene):
    from rkifield_b200.engine import Context
    v = small_scene["vox"]
    objs = _scene_objects(small_scene) if request.param else [small_scene["obj"]]
    ctx = Context(pool_capacity=v.n_bricks + 1024)
    ctx.set_brick_pool(v.words)
    ctx.upload_brick_maps(v.map)
    ctx.upload_objects(objs)
    yield ctx
    ctx.close()


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("tmax", [1e-3, 32.0, 1e4, np.inf, np.nan])
def test_rays(scene, mode, tmax):
    d = np.array(list(itertools.product(RATES, repeat=3)), np.float32)
    o = np.random.default_rng(4).uniform(-15.0, 15.0, d.shape).astype(np.float32)
    t = np.full(len(d), tmax, np.float32)
    tu = scene.tuning()
    try:
        got = scene.trace(o, d, t, mode, _params(0))
        tu.no_empty_path = 1
        scene.set_tuning(tu)
        ref = scene.trace(o, d, t, mode, _params(0))
    finally:
        tu.no_empty_path = 0
        scene.set_tuning(tu)
    for k in ("t", "flags"):
        assert_bits_equal(got[k], ref[k], k)


@pytest.mark.parametrize("rate", [np.nan, np.inf, -np.inf, 3e38, 1e30, 1e19])
@pytest.mark.parametrize("field", ["position", "forward", "right", "up", "jitter"])
def test_views(scene, small_scene, field, rate):
    from rkifield_b200 import scenes
    w, h = 515, 257
    cam = scenes.seeded_camera(small_scene["spec"], w, h, seed=5)
    getattr(cam, field)[1] = rate
    _both(scene, cam, _params(0), w, h)
