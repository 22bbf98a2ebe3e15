"""Several voxelized objects of different voxel sizes, whose EMPTY values differ: a run
inside one object's EMPTY space takes that object's value, whichever its place among
the objects.  Views (below and above the settling limit) and ray batches in the three
modes, bit-exact with the oracle under the three strategies."""
import numpy as np
import pytest

from conftest import assert_bits_equal
from test_tiled_gpu import PLANES, _params
from test_trace_gpu import _rays

pytestmark = pytest.mark.gpu


def _small_grid(first_map, voxel_size, at):
    """A 6 x 5 x 4 grid of voxel_size around `at` with three bricks of the pool."""
    from rkifield_b200 import _abi as abi
    o = abi.rkf_gpu_object()
    dims, be = (6, 5, 4), np.float32(voxel_size) * np.float32(8.0)
    for a in range(4):
        o.inverse_world[5 * a] = 1.0
    for a in range(3):
        half = 0.5 * dims[a] * float(be)
        o.inverse_world[12 + a] = -float(at[a])
        o.aabb_min[a], o.aabb_max[a] = at[a] - half, at[a] + half
        o.brick_map_dims[a], o.accumulated_scale[a] = dims[a], 1.0
    o.voxel_size, o.sdf_type, o.object_id = float(np.float32(voxel_size)), abi.RKF_SDF_VOXELIZED, 9
    o.brick_map_offset = first_map
    m = np.full(120, abi.EMPTY_SLOT, np.uint32)
    m[[31, 62, 88]] = (0, 1, 2)
    return o, m


@pytest.mark.parametrize("strategy", ["brute", "tiled", "bvh"])
@pytest.mark.parametrize("first", [True, False], ids=["small-first", "small-last"])
def test_voxel_sizes(oracle, small_scene, strategy, first):
    from rkifield_b200 import _abi as abi
    from rkifield_b200 import engine, scenes
    v = small_scene["vox"]
    objs, maps = [small_scene["obj"]], [v.map]
    for vs, at in ((0.11, (21.0, 3.0, -19.0)), (0.013, (-19.0, -20.0, 7.0))):
        o, m = _small_grid(sum(x.size for x in maps), vs, at)
        objs.append(o)
        maps.append(m)
    if first:
        objs = objs[::-1]
    bvh = engine.object_bvh(objs)
    maps = np.concatenate(maps)
    sc = oracle.Scene(objs, pool_words=v.words, brick_maps=maps, bvh=bvh)
    p = _params({"brute": abi.RKF_STRATEGY_BRUTE, "tiled": abi.RKF_STRATEGY_TILED, "bvh": abi.RKF_STRATEGY_BVH}[strategy])
    with engine.Context(pool_capacity=v.n_bricks + 1024) as ctx:
        ctx.set_brick_pool(v.words)
        ctx.upload_brick_maps(maps)
        ctx.upload_objects(objs)
        ctx.upload_bvh(bvh)
        for w, h, seed in ((256, 144, 3), (521, 263, 8)):
            cam = scenes.seeded_camera(small_scene["spec"], w, h, seed=seed)
            ref = oracle.march(sc, cam, p, w, h, with_reference_planes=True)
            got = ctx.march(cam, p, w, h, reference_planes=True)
            for k in PLANES:
                assert_bits_equal(got[k], ref[k], f"{w}x{h} {k}")
        if strategy == "brute":
            o, d, tmax = _rays(6000, seed=2)
            for mode in (0, 1, 2):
                ref = oracle.trace(sc, o.ravel(), d.ravel(), tmax, mode, p)
                got = ctx.trace(o, d, tmax, mode, p)
                for k in ref:
                    if k in got:
                        assert_bits_equal(got[k], ref[k], f"mode {mode} {k}")
