"""The runs over EMPTY samples round as the sampler's chain does: rays of a few EMPTY
steps to a brick, where t is small enough for a last-place difference of a step to
show in it (the brick's values lie below the hit threshold, so a ray ends with the t of
its first sample there).  Bit-exact with the oracle, in the three modes."""
import numpy as np
import pytest

from conftest import assert_bits_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("voxel_size", [0.1, 0.07, 0.04])
def test_short_runs(oracle, voxel_size):
    from rkifield_b200 import _abi as abi
    from rkifield_b200.engine import Context
    dims, be = (6, 5, 5), np.float32(voxel_size) * np.float32(8.0)
    o = abi.rkf_gpu_object()
    for a in range(4):
        o.inverse_world[5 * a] = 1.0
    for a in range(3):
        half = 0.5 * dims[a] * float(be)
        o.aabb_min[a], o.aabb_max[a], o.brick_map_dims[a], o.accumulated_scale[a] = -half, half, dims[a], 1.0
    o.voxel_size, o.sdf_type, o.object_id = float(np.float32(voxel_size)), abi.RKF_SDF_VOXELIZED, 1
    brick_map = np.full(150, abi.EMPTY_SLOT, np.uint32)
    brick_map[[40, 77, 110]] = 0
    words = np.zeros(1024, np.uint32)
    words[0::2] = int(np.float16(0.1 * float(be)).view(np.uint16)) | (5 << 16)
    sc = oracle.Scene([o], pool_words=words, brick_maps=brick_map)
    p = abi.rkf_march_params()
    abi.march_params_default(p)
    p.scene.hit_threshold, p.near_surface_threshold, p.scene.max_steps = 0.25 * float(be), 0.02, 128
    rng = np.random.default_rng(1)
    n = 400_000
    org = (rng.uniform(-0.5, 0.5, (n, 3)) * np.array(dims) * float(be)).astype(np.float32)
    d = rng.standard_normal((n, 3)).astype(np.float32)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    tmax = np.full(n, 4.0 * float(be), np.float32)
    with Context(pool_capacity=64) as ctx:
        ctx.set_brick_pool(words)
        ctx.upload_brick_maps(brick_map)
        ctx.upload_objects([o])
        for mode in (0, 1, 2):
            ref = oracle.trace(sc, org.ravel(), d.ravel(), tmax, mode, p)
            got = ctx.trace(org, d, tmax, mode, p)
            assert_bits_equal(got["t"], ref["t"], f"mode {mode}")
            np.testing.assert_array_equal(got["flags"], ref["flags"])
        assert ctx.lib.rkf_testing_last_variant(ctx.h) == 2  # the EMPTY path
