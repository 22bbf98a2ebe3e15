"""The empty-space distances at brick resolution, against a chessboard distance
transform of the exported index: after a voxelization, an additive edit, and edits
that carve INTERIOR blocks open, whose views (settled misses first) must stay those
of the general path."""
import ctypes as C

import numpy as np
import pytest
from scipy.ndimage import distance_transform_cdt

from test_edit_gpu import _op
from test_settle_gpu import _both
from test_tiled_gpu import _params

pytestmark = pytest.mark.gpu

CAP, EMPTY, INTERIOR = 8, 0xFFFFFFFF, 0xFFFFFFFE


def _check(ctx):
    from rkifield_b200 import _abi as abi
    idx = ctx.export_index()
    n = C.c_uint64()
    abi.check(ctx.lib.rkf_testing_export_leaf_dist(ctx.h, None, C.byref(n)), "leaf_dist")
    got = np.zeros(n.value, np.uint8)
    abi.check(ctx.lib.rkf_testing_export_leaf_dist(ctx.h, got.ctypes.data, C.byref(n)), "leaf_dist")
    leaves = idx["leaves"].reshape(-1, 8, 8, 8)
    off, nx, ny, nz = (int(v) for v in idx["obj_top_info"][:4])
    top = idx["top"][off:off + nx * ny * nz]
    bricks = np.repeat(top[:, None], 512, 1).reshape(-1, 8, 8, 8)
    is_leaf = top < INTERIOR
    bricks[is_leaf] = leaves[top[is_leaf]]
    # the bricks of the whole grid, z, y, x, with a border the transform never reaches past
    grid = bricks.reshape(nz, ny, nx, 8, 8, 8).transpose(0, 3, 1, 4, 2, 5).reshape(nz * 8, ny * 8, nx * 8)
    d = np.minimum(distance_transform_cdt(grid == EMPTY, "chessboard"), CAP)
    want = d.reshape(nz, 8, ny, 8, nx, 8).transpose(0, 2, 4, 1, 3, 5).reshape(-1, 512)
    np.testing.assert_array_equal(got.reshape(-1, 512)[top[is_leaf]], want[is_leaf])
    return top


def test_distances_and_interior_edits(small_scene):
    from rkifield_b200 import scenes
    from rkifield_b200.engine import Context
    prims = small_scene["prims"][:12].copy()
    big = prims[:1].copy()
    big["type"], big["centre"], big["params"], big["bound_radius"] = 0, (0.0, 0.0, 0.0), (7.0, 0.0, 0.0), 7.02
    prims = np.concatenate([prims, big])
    with Context(pool_capacity=200_000, keep_reference_pool=False) as ctx:
        ctx.voxelize(prims, scenes.voxelize_params(small_scene["spec"], prims))
        top = _check(ctx)
        assert (top == INTERIOR).sum() > 4 and (top < INTERIOR).sum() > 4 and (top == EMPTY).sum() > 4
        ctx.edit(_op(0, (-11.0, 9.0, 2.0), 0.9, 3))
        _check(ctx)
        rng = np.random.default_rng(2)
        w, h = 521, 256
        for k in range(3):
            at = rng.uniform(-1.5, 1.5, 3)
            ctx.edit(_op(1, at, 1.3, 3))  # within INTERIOR blocks
            carved = _check(ctx)
            assert (carved == INTERIOR).sum() < (top == INTERIOR).sum()
            for eye, to in ((at, at + np.array([1.0, 0.3, 0.2])), (np.array([14.0, 3.0, 9.0]), at)):
                got = _both(ctx, scenes.camera_uniforms(eye, to, w, h), _params(0), w, h)
                assert ((got["flags"] & 1) != 0).any()


def test_block_field_of_a_second_object(small_scene):
    """An edit lowers the block distances of its own object, wherever its grid lies
    in the field: exact around additive edits in each of two objects, and the views of
    both are those of the general path."""
    from rkifield_b200 import scenes
    from rkifield_b200.engine import Context
    from test_empty_dist_gpu import _chebyshev, _field
    from test_multi_vox_gpu import _moved
    with Context(pool_capacity=200_000, keep_reference_pool=False) as ctx:
        for k in range(2):
            prims = small_scene["prims"][5 * k:5 * k + 5].copy()
            ctx.voxelize(prims, scenes.voxelize_params(small_scene["spec"], prims, object_id=k + 1))
        ctx.update_objects([ctx.object(0), _moved(ctx.object(1), (40.0, 3.0, -2.0), 2)], [0, 1])
        rng = np.random.default_rng(5)
        for k in (1, 0, 1):
            half = 0.4 * np.array([ctx.object(k).brick_map_dims[a] for a in range(3)]) * 0.32
            at = rng.uniform(-half, half)
            op = _op(0, at, 0.7, 3)
            op.object_index = k
            ctx.edit(op)
            idx = ctx.export_index()
            field, want = _field(ctx), _chebyshev(idx["top"], idx["obj_top_info"])
            assert (field <= want).all() and ((field == 0) == (want == 0)).all()
            to = at + (np.array([40.0, 3.0, -2.0]) if k else 0.0)
            _both(ctx, scenes.camera_uniforms(to + np.array([6.0, 4.0, 7.0]), to, 521, 256), _params(0), 521, 256)
