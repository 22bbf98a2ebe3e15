"""The settling passes where their lists find no room: a view takes them in parts of
what the context's lists hold (those of a 1920x1080 view at first), which a failed
growth does not lose; the outputs are the general path's, ray batches of the same
launch included.  And the launches that take the passes: views of 131,072 ids on."""
import ctypes as C

import numpy as np
import pytest

from conftest import assert_bits_equal
from test_failures_gpu import inject  # noqa: F401
from test_launch_stats_gpu import _stats
from test_tiled_gpu import _params
from test_trace_gpu import _rays

pytestmark = pytest.mark.gpu

PLANES = ("t", "normal", "slot", "material", "flags")


@pytest.fixture()
def ctx(small_scene):
    from rkifield_b200.engine import Context
    with Context(pool_capacity=small_scene["vox"].n_bricks * 2 + 4096, keep_reference_pool=False) as c:
        c.voxelize(small_scene["prims"], small_scene["vp"])
        yield c


def _batch(ctx, cam, w, h, rays):
    """A view and a ray batch in one launch, into device planes; the launches."""
    from rkifield_b200 import _abi as abi
    from rkifield_b200 import cudart, engine
    n = rays[2].size
    planes, hits = cudart.device_gbuffer(w * h), cudart.device_gbuffer(n)
    dev = [cudart.DeviceArray(a.size, np.float32).upload(a) for a in rays]
    view, batch = (abi.rkf_view * 1)(), (abi.rkf_ray_batch * 1)()
    view[0].camera, view[0].width, view[0].height = cam, w, h
    view[0].out = engine._gb_struct(cudart.gbuffer_ptrs(planes), abi.RKF_MEM_DEVICE)
    b = batch[0]
    b.origins, b.dirs, b.tmax, b.n, b.mode = dev[0].ptr, dev[1].ptr, dev[2].ptr, n, abi.RKF_TRACE_CLOSEST
    for k, v in cudart.gbuffer_ptrs(hits).items():
        setattr(b.out, k, v)
    b.out.mem = abi.RKF_MEM_DEVICE
    before = _stats(ctx)[0]
    tu = ctx.tuning()
    abi.check(ctx.lib.rkf_march_batch(ctx.h, view, 1, batch, 1, C.byref(_params(0)), C.byref(tu)), "batch")
    return [p[k].download() for p in (planes, hits) for k in PLANES], _stats(ctx)[0] - before


def _general(ctx, *a):
    tu = ctx.tuning()
    try:
        tu.no_empty_path = 1
        ctx.set_tuning(tu)
        return _batch(ctx, *a)[0]
    finally:
        tu.no_empty_path = 0
        ctx.set_tuning(tu)


def test_parts(ctx, small_scene, inject):  # noqa: F811
    from rkifield_b200 import scenes
    w, h = 3001, 2003  # 6.0 M ids: three parts of the lists of 2.1 M
    cam = scenes.seeded_camera(small_scene["spec"], w, h, seed=4)
    rays = [np.ascontiguousarray(a, np.float32).ravel() for a in _rays(5000, seed=1)]
    ref = _general(ctx, cam, w, h, rays)
    held = ctx.info()["device_bytes"]
    inject(0)
    got, launches = _batch(ctx, cam, w, h, rays)
    inject(-1)
    assert launches == 9 and ctx.info()["device_bytes"] == held
    for a, b in zip(got, ref):
        assert_bits_equal(a, b, "parts")
    got, launches = _batch(ctx, cam, w, h, rays)  # with room: at once
    assert launches == 3 and ctx.info()["device_bytes"] > held
    for a, b in zip(got, ref):
        assert_bits_equal(a, b, "at once")


@pytest.mark.parametrize("size,launches", [((512, 256), 3), ((504, 256), 1)])
def test_views_that_settle(ctx, small_scene, size, launches):
    from rkifield_b200 import scenes
    rays = [np.ascontiguousarray(a, np.float32).ravel() for a in _rays(100, seed=1)]
    cam = scenes.seeded_camera(small_scene["spec"], *size, seed=4)
    assert _batch(ctx, cam, *size, rays)[1] == launches


def test_tile_order_below_the_passes(ctx, small_scene):
    """The heaviest-first order where it still acts on a whole launch: three kernels
    before the march, and the same outputs."""
    from rkifield_b200 import scenes
    rays = [np.ascontiguousarray(a, np.float32).ravel() for a in _rays(100, seed=1)]
    cam = scenes.seeded_camera(small_scene["spec"], 504, 256, seed=6)
    ref = _general(ctx, cam, 504, 256, rays)
    tu = ctx.tuning()
    tu.order_tiles = 1
    ctx.set_tuning(tu)
    got, launches = _batch(ctx, cam, 504, 256, rays)
    assert launches == 4
    for a, b in zip(got, ref):
        assert_bits_equal(a, b, "ordered")


def test_autotune_orders_bands_of_settled_views(ctx, small_scene):
    """The settled launch ignores the tile order, the host bands take it."""
    from rkifield_b200 import _abi as abi
    from rkifield_b200 import cudart, engine, scenes
    w, h = 640, 360
    keep = cudart.device_gbuffer(w * h)
    view = (abi.rkf_view * 1)()
    view[0].camera, view[0].width, view[0].height = scenes.seeded_camera(small_scene["spec"], w, h, seed=4), w, h
    view[0].out = engine._gb_struct(cudart.gbuffer_ptrs(keep), abi.RKF_MEM_DEVICE)
    tu = abi.rkf_batch_tuning()
    abi.check(ctx.lib.rkf_autotune(ctx.h, view, 1, None, 0, C.byref(_params(0)), C.byref(tu)), "autotune")
    assert tu.order_tiles == 1
