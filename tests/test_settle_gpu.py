"""Views large enough for the settling passes, point queries and secondary
rays at the sizes where their kernels' splits change.

A launch whose views hold 131,072 work ids or more settles their misses before
the march; the general path (the full sampler, no EMPTY space) has no such
step.  Both must write the same bits: over one object and several, the three
strategies, cameras outside and inside the grid, odd sizes (padded tiles), other
tile shapes, step budgets that end a ray before it leaves the grid, and the
index after edits, whose brick distances the walks read."""
import ctypes as C

import numpy as np
import pytest

from conftest import assert_bits_equal
from test_edit_gpu import _op
from test_multi_empty_gpu import _scene_objects
from test_tiled_gpu import PLANES, _params

pytestmark = pytest.mark.gpu


def _both(ctx, cam, p, w, h, tile=(8, 4)):
    """The view with the passes and through the general path."""
    tu = ctx.tuning()
    keep = (tu.tile_w, tu.tile_h, tu.no_empty_path)
    try:
        tu.tile_w, tu.tile_h, tu.no_empty_path = tile[0], tile[1], 0
        ctx.set_tuning(tu)
        got = ctx.march(cam, p, w, h, reference_planes=True)
        tu.no_empty_path = 1
        ctx.set_tuning(tu)
        ref = ctx.march(cam, p, w, h, reference_planes=True)
    finally:
        tu.tile_w, tu.tile_h, tu.no_empty_path = keep
        ctx.set_tuning(tu)
    for k in PLANES:
        assert_bits_equal(got[k], ref[k], f"{w}x{h} {tile}: {k}")
    return got


@pytest.fixture(scope="module")
def one(small_scene):
    from rkifield_b200.engine import Context
    ctx = Context(pool_capacity=small_scene["vox"].n_bricks * 2 + 4096, keep_reference_pool=False)
    ctx.voxelize(small_scene["prims"], small_scene["vp"])
    yield ctx
    ctx.close()


# 512x256 holds exactly 131,072 ids, 511x256 pads to them, 504x256 stays below
@pytest.mark.parametrize("size,tile", [((512, 256), (8, 4)), ((511, 256), (8, 4)), ((504, 256), (8, 4)),
                                       ((521, 263), (8, 4)), ((517, 301), (16, 2)), ((433, 389), (5, 3)), ((530, 270), (16, 16)),
                                       ((1, 140000), (8, 4))])
def test_view_sizes_and_tiles(one, small_scene, size, tile):
    from rkifield_b200 import scenes
    cam = scenes.seeded_camera(small_scene["spec"], *size, seed=4)
    _both(one, cam, _params(0), *size, tile)


@pytest.mark.parametrize("inside", [False, True])
@pytest.mark.parametrize("steps,far", [(1, 1e4), (7, 1e4), (40, 1e4), (128, 20.0), (300, 1e4)])
def test_step_budgets_and_reach(one, small_scene, steps, far, inside):
    """Rays that run out of steps, end past max_distance or leave the grid."""
    from rkifield_b200 import scenes
    spec = small_scene["spec"]
    w, h = 523, 259
    cam = (scenes.camera_uniforms((0.7, 1.3, -0.4), (9.0, 2.0, 5.0), w, h) if inside
           else scenes.seeded_camera(spec, w, h, seed=6))
    p = _params(0)
    p.hard_max_steps = steps
    p.scene.max_steps = max(1, steps // 2)
    p.scene.max_distance = far
    _both(one, cam, p, w, h)


def test_against_the_oracle(oracle, small_scene):
    from rkifield_b200 import scenes
    from rkifield_b200.engine import Context
    v = small_scene["vox"]
    sc = oracle.Scene([small_scene["obj"]], pool_words=v.words, brick_maps=v.map)
    ctx = Context(pool_capacity=v.n_bricks + 1024)
    try:
        ctx.set_brick_pool(v.words)
        ctx.upload_brick_maps(v.map)
        ctx.upload_objects([small_scene["obj"]])
        w, h = 515, 257
        cam = scenes.seeded_camera(small_scene["spec"], w, h, seed=9)
        ref = oracle.march(sc, cam, _params(0), w, h, with_reference_planes=True)
        got = ctx.march(cam, _params(0), w, h, reference_planes=True)
        for k in PLANES:
            assert_bits_equal(got[k], ref[k], k)
    finally:
        ctx.close()


@pytest.mark.parametrize("strategy", ["brute", "tiled", "bvh"])
@pytest.mark.parametrize("several", [False, True])
def test_strategies(small_scene, strategy, several):
    from rkifield_b200 import _abi as abi
    from rkifield_b200 import engine, scenes
    v = small_scene["vox"]
    objs = _scene_objects(small_scene) if several else [small_scene["obj"]]
    ctx = engine.Context(pool_capacity=v.n_bricks + 1024)
    try:
        ctx.set_brick_pool(v.words)
        ctx.upload_brick_maps(v.map)
        ctx.upload_objects(objs)
        if strategy == "bvh":
            ctx.upload_bvh(engine.object_bvh(objs))
        code = {"brute": abi.RKF_STRATEGY_BRUTE, "tiled": abi.RKF_STRATEGY_TILED, "bvh": abi.RKF_STRATEGY_BVH}
        w, h = 519, 261
        for seed in (3, 8):
            got = _both(ctx, scenes.seeded_camera(small_scene["spec"], w, h, seed=seed), _params(code[strategy]), w, h)
            assert 0.01 < ((got["flags"] & 1) != 0).mean() < 0.99
    finally:
        ctx.close()


def test_views_between_edits(small_scene):
    """Each edit writes its index into the one before last, and lowers the brick
    distances around it."""
    from rkifield_b200 import scenes
    from rkifield_b200.engine import Context
    ctx = Context(pool_capacity=small_scene["vox"].n_bricks * 2 + 20000, keep_reference_pool=False)
    try:
        ctx.voxelize(small_scene["prims"], small_scene["vp"])
        rng = np.random.default_rng(3)
        w, h = 512, 258
        epoch = ctx.info()["epoch"]
        for k in range(5):
            at = rng.uniform(-10.0, 10.0, 3)
            ctx.edit(_op(0, at, 0.8, 3))
            cam = scenes.camera_uniforms(at + np.array([3.0, 2.0, 4.0]), at, w, h)
            got = _both(ctx, cam, _params(0), w, h)
            assert ((got["flags"] & 1) != 0).any()
        assert ctx.info()["epoch"] > epoch
    finally:
        ctx.close()


@pytest.mark.parametrize("n_objs", [1, 2, 7])
def test_point_counts_agree(small_scene, n_objs):
    """A point's answer does not depend on how many are asked with it: block
    edges (16 points), and both sides of the page-locked path's limit."""
    from rkifield_b200.engine import Context
    v = small_scene["vox"]
    objs = [small_scene["obj"]] if n_objs == 1 else _scene_objects(small_scene)[:n_objs]
    ctx = Context(pool_capacity=v.n_bricks + 1024)
    try:
        ctx.set_brick_pool(v.words)
        ctx.upload_brick_maps(v.map)
        ctx.upload_objects(objs)
        rng = np.random.default_rng(n_objs)
        pts = rng.uniform(-18.0, 18.0, (17600, 3)).astype(np.float32)
        d, g, m = ctx.query_points(pts)
        g = g.reshape(-1, 3)
        for n in (1, 2, 15, 16, 17, 33, 300, 17400, 17500):
            d2, g2, m2 = ctx.query_points(pts[-n:])
            assert_bits_equal(d2, d[-n:], f"{n}: distance")
            assert_bits_equal(g2.reshape(-1, 3), g[-n:], f"{n}: gradient")
            np.testing.assert_array_equal(m2, m[-n:])
    finally:
        ctx.close()


def test_occlusion_counts_agree(one):
    """The taps of a point are lanes of one warp: block edges (32 points)."""
    rng = np.random.default_rng(8)
    pos = rng.uniform(-16.0, 16.0, (5000, 3)).astype(np.float32)
    nrm = rng.standard_normal((5000, 3))
    nrm = (nrm / np.linalg.norm(nrm, axis=1, keepdims=True)).astype(np.float32)
    ao = one.sdf_ao(pos, nrm)
    assert 0.0 <= ao.min() < 1.0
    for n in (1, 7, 8, 9, 31, 32, 33, 4097):
        assert_bits_equal(one.sdf_ao(pos[-n:], nrm[-n:]), ao[-n:], str(n))


@pytest.mark.parametrize("size", [(1, 1), (37, 11), (64, 8)])
def test_secondary_rays_per_pixel(one, small_scene, size):
    """Each ray of a call with several lights and occlusion rays is the ray of the
    call that asks for it alone, at counts that do not divide a block; rays to a
    light end at it, and missed pixels own dead rays."""
    from rkifield_b200 import _abi as abi
    from rkifield_b200 import cudart, scenes
    w, h = size
    n = w * h
    cam = scenes.seeded_camera(small_scene["spec"], w, h, seed=2)
    view = one.march(cam, _params(0), w, h)
    dev = {k: cudart.DeviceArray(view[k].size, view[k].dtype).upload(view[k]) for k in ("t", "normal", "flags")}
    lights = np.array([[3.0, 20.0, -4.0], [0.0, 9.0, 1.0], [-12.0, 4.0, 8.0]], np.float32)
    gb = abi.rkf_gbuffer()
    gb.t, gb.normal, gb.flags, gb.mem = dev["t"].ptr, dev["normal"].ptr, dev["flags"].ptr, abi.RKF_MEM_DEVICE

    def rays(lt, ao):
        lt = np.ascontiguousarray(lt, np.float32)
        arrs = [cudart.DeviceArray(max(1, c * n * k), np.float32) for k in (len(lt), ao) for c in (3, 3, 1)]
        hits = C.c_uint32()
        abi.check(one.lib.rkf_secondary_rays(one.h, C.byref(cam), w, h, C.byref(gb), lt.ctypes.data, len(lt), ao, 1.0,
                                             77, *[a.ptr for a in arrs], C.byref(hits), None), "secondary rays")
        return [a.download() for a in arrs], hits.value

    hit = (view["flags"].reshape(-1) & 1) != 0
    full, hits = rays(lights, 5)
    assert hits == hit.sum()
    for k in range(3):
        alone, hits = rays(lights[k:k + 1], 0)
        assert hits == hit.sum()
        for a, b, c in zip(full[:3], alone[:3], (3, 3, 1)):
            assert_bits_equal(a.reshape(n, 3, c)[:, k], b.reshape(n, c), f"light {k}")
    few, hits = rays(lights[:0], 2)
    assert hits == hit.sum()
    for a, b, c in zip(full[3:], few[3:], (3, 3, 1)):
        assert_bits_equal(a.reshape(n, 5, c)[:, :2], b.reshape(n, 2, c), "occlusion")
    assert rays(lights[:0], 0)[1] == hit.sum()
    o, d, t = full[0].reshape(n, 3, 3)[hit], full[1].reshape(n, 3, 3)[hit], full[2].reshape(n, 3)[hit]
    # about ten roundings of 2^-24 of the length, the light and the origin
    off = np.abs(o.astype(np.float64) + d.astype(np.float64) * t[..., None] - lights)
    assert (off <= 1e-6 * (t[..., None] + np.abs(lights) + np.abs(o))).all()
    assert (full[2].reshape(n, 3)[~hit] == -1.0).all() and (full[5].reshape(n, 5)[~hit] == -1.0).all()
