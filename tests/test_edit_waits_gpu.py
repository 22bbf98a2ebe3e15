"""A direct edit waits for marches on other streams only where it makes an epoch:
one that is refused, meets no brick or changes none returns while they run."""
import pytest

from test_edit_gpu import _op
from test_tiled_gpu import _params

pytestmark = pytest.mark.gpu


def test_edits_that_change_nothing_wait_for_nothing(small_scene):
    from cuda.bindings import runtime as rt

    from rkifield_b200 import cudart, scenes
    from rkifield_b200.engine import Context, RkfError
    w, h = 5120, 2880
    with Context(pool_capacity=small_scene["vox"].n_bricks * 2 + 4096, keep_reference_pool=False) as ctx:
        ctx.voxelize(small_scene["prims"], small_scene["vp"])
        ctx.edit(_op(0, (0.0, 0.0, 0.0), 0.5, 3))
        cam = scenes.seeded_camera(small_scene["spec"], w, h, seed=4)
        planes = cudart.device_gbuffer(w * h)
        out = cudart.gbuffer_ptrs(planes)
        s = cudart.Stream()
        edits = (_op(0, (500.0, 0.0, 0.0), 0.5, 3),   # beside the grid
                 _op(1, (0.0, 30.0, 0.0), 0.2, 3),    # nothing to take away there
                 _op(9, (0.0, 0.0, 0.0), 0.5, 3))     # no such edit
        ctx.march_async(cam, _params(0), 64, 64, out, s.ptr)
        s.synchronize()
        epoch = ctx.info()["epoch"]
        for op in edits:
            ctx.march_async(cam, _params(0), w, h, out, s.ptr)  # some ten milliseconds
            try:
                ctx.edit(op)
                assert op.edit_type != 9
            except RkfError:
                assert op.edit_type == 9
            running = rt.cudaStreamQuery(s.handle)[0] == rt.cudaError_t.cudaErrorNotReady
            s.synchronize()
            assert running, f"edit type {op.edit_type} waited for the march"
        assert ctx.info()["epoch"] == epoch
