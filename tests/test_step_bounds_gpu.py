"""Rays of tens of thousands of EMPTY steps, whose t drifts from steps * step by
the roundings of its sums: the bounds that settle a ray without stepping it must
hold that drift.  In a grid 33,000 bricks long whose brick extent lies just above
(below) half a unit in the last place of t, t gains (loses) some 15 steps; a ray
that leaves the grid about when its steps run out ends past its reach in place of
out of steps, or the other way round."""
import numpy as np
import pytest

from rkifield_b200 import _abi as abi

LONG = 33000  # as far as the boxes of one walk reach


def _object(voxel_size):
    """An EMPTY grid LONG x 8 x 8; the world's origin lies 3.5 bricks inside it."""
    o = abi.rkf_gpu_object()
    be = np.float32(voxel_size) * np.float32(8.0)
    gs = np.array([LONG, 8, 8], np.float32) * be
    off = np.float32(3.5) * be
    for a in range(4):
        o.inverse_world[5 * a] = 1.0
    for a in range(3):
        o.aabb_min[a], o.aabb_max[a] = float(-0.5 * gs[a]), float(0.5 * gs[a])
        o.brick_map_dims[a], o.accumulated_scale[a] = (LONG, 8, 8)[a], 1.0
    o.inverse_world[12] = float(off - gs[0] * np.float32(0.5))
    o.aabb_min[0], o.aabb_max[0] = float(-off), float(gs[0] - off)
    o.voxel_size, o.sdf_type, o.object_id = float(np.float32(voxel_size)), abi.RKF_SDF_VOXELIZED, 1
    # the last voxel's centre, past which the sampler clamps
    return o, float(be), float(gs[0]) - float(off) - 0.5 * float(be) / 8.0


@pytest.mark.gpu
@pytest.mark.parametrize("ulps", [504.52, 504.48])
def test_drift_of_long_rays(oracle, ulps):
    from rkifield_b200.engine import Context
    obj, be, end = _object(ulps / 256.0 / 8.0)  # t lies in [2^15, 2^16) for half of the steps: an ulp is 2^-8
    brick_map = np.full(LONG * 64, abi.EMPTY_SLOT, np.uint32)
    words = np.zeros(1024, np.uint32)
    sc = oracle.Scene([obj], pool_words=words, brick_maps=brick_map)
    p = abi.rkf_march_params()
    abi.march_params_default(p)
    p.scene.hit_threshold, p.scene.max_steps, p.near_surface_threshold = 0.1, 128, 0.02
    p.scene.max_distance = end + 0.4 * be
    o, d = np.zeros(3, np.float32), np.array([1.0, 0.0, 0.0], np.float32)
    tmax = np.array([p.scene.max_distance], np.float32)
    cam = abi.rkf_camera()
    cam.forward[0] = 1.0  # (right and up zero: every pixel's ray is the same)
    flags = []
    with Context(pool_capacity=1024) as ctx:
        ctx.set_brick_pool(words)
        ctx.upload_brick_maps(brick_map)
        ctx.upload_objects([obj])
        mid = int(end / be)  # steps without the drift
        for steps in range(mid - 24, mid + 30, 2):
            p.hard_max_steps = steps
            want = int(oracle.trace(sc, o, d, tmax, 0, p)["flags"][0])
            assert int(ctx.trace(o, d, tmax, 0, p)["flags"][0]) == want, steps
            if not flags or want != flags[-1][1]:
                flags.append((steps, want))
        # views settle their tiles and rays before the march: around the change
        assert [f for _, f in flags] == [4, 0]
        for steps in (flags[1][0] - 6, flags[1][0] + 4):
            p.hard_max_steps = steps
            got = ctx.march(cam, p, 512, 256)["flags"]
            assert (got == (4 if steps < flags[1][0] else 0)).all(), steps
        assert ctx.lib.rkf_testing_last_variant(ctx.h) == 2  # the empty-space path marched it
