"""Views of one object off the EMPTY path (a rotated transform): marched by the kernel
of several objects where that is the faster one, with the outputs of the oracle under
the brute, tiled and BVH strategies, and of ray batches by the kernel of one."""
import numpy as np
import pytest

from conftest import assert_bits_equal
from test_multi_empty_gpu import _rotation
from test_tiled_gpu import PLANES, _params
from test_trace_gpu import _rays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("strategy", ["brute", "tiled", "bvh"])
def test_rotated_object(oracle, small_scene, strategy):
    from rkifield_b200 import _abi as abi
    from rkifield_b200 import engine, scenes
    v = small_scene["vox"]
    obj = abi.rkf_gpu_object.from_buffer_copy(small_scene["obj"])
    rot = _rotation((1.0, 2.0, 3.0), 0.4)
    for c in range(3):
        for a in range(3):
            obj.inverse_world[4 * c + a] = float(np.float32(rot[a][c]))
    for a in range(3):
        obj.aabb_min[a], obj.aabb_max[a] = -32.0, 32.0
    bvh = engine.build_bvh([(0, (-32.0,) * 3, (32.0,) * 3), (0, (-32.0,) * 3, (32.0,) * 3)])
    sc = oracle.Scene([obj], pool_words=v.words, brick_maps=v.map, bvh=bvh)
    p = _params({"brute": abi.RKF_STRATEGY_BRUTE, "tiled": abi.RKF_STRATEGY_TILED, "bvh": abi.RKF_STRATEGY_BVH}[strategy])
    with engine.Context(pool_capacity=v.n_bricks + 1024) as ctx:
        ctx.set_brick_pool(v.words)
        ctx.upload_brick_maps(v.map)
        ctx.upload_objects([obj])
        ctx.upload_bvh(bvh)
        for w, h, seed in ((203, 101, 3), (521, 256, 8)):
            cam = scenes.seeded_camera(small_scene["spec"], w, h, seed=seed)
            ref = oracle.march(sc, cam, p, w, h, with_reference_planes=True)
            got = ctx.march(cam, p, w, h, reference_planes=True)
            assert ctx.lib.rkf_testing_last_variant(ctx.h) == 1
            for k in PLANES:
                assert_bits_equal(got[k], ref[k], f"{w}x{h} {k}")
            assert ((ref["flags"] & 1) != 0).any()
        if strategy != "bvh":  # NaN rays sample NaN, of one object in either kernel: out of steps
            cam.forward[0] = np.nan
            assert (ctx.march(cam, _params(0), 97, 61)["flags"] == 4).all()
        if strategy == "brute":
            o, d, tmax = _rays(3000, seed=2)
            for mode in (0, 1, 2):
                ref = oracle.trace(sc, o.ravel(), d.ravel(), tmax, mode, p)
                got = ctx.trace(o, d, tmax, mode, p)
                for k in ref:
                    if k in got:
                        assert_bits_equal(got[k], ref[k], f"mode {mode} {k}")
