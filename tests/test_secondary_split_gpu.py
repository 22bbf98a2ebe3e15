"""Secondary rays of one or two occlusion rays a pixel (a thread per pixel) are those
of a call that asks for more (a thread per ray), bit for bit, at counts that do not
divide a block."""
import ctypes as C

import numpy as np
import pytest

from conftest import assert_bits_equal
from test_tiled_gpu import _params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(1, 1), (37, 11), (64, 8)])
def test_few_rays_per_pixel(small_scene, small_ctx, size):
    from rkifield_b200 import _abi as abi
    from rkifield_b200 import cudart, scenes
    w, h = size
    n = w * h
    cam = scenes.seeded_camera(small_scene["spec"], w, h, seed=2)
    view = small_ctx.march(cam, _params(0), w, h)
    dev = {k: cudart.DeviceArray(view[k].size, view[k].dtype).upload(view[k]) for k in ("t", "normal", "flags")}
    lights = np.array([[3.0, 20.0, -4.0], [0.0, 9.0, 1.0], [-12.0, 4.0, 8.0]], np.float32)
    gb = abi.rkf_gbuffer()
    gb.t, gb.normal, gb.flags, gb.mem = dev["t"].ptr, dev["normal"].ptr, dev["flags"].ptr, abi.RKF_MEM_DEVICE

    def rays(nl, ao):
        arrs = [cudart.DeviceArray(max(1, c * n * k), np.float32) for k in (nl, ao) for c in (3, 3, 1)]
        hits = C.c_uint32()
        abi.check(small_ctx.lib.rkf_secondary_rays(small_ctx.h, C.byref(cam), w, h, C.byref(gb), lights.ctypes.data, nl,
                                                   ao, 1.0, 77, *[a.ptr for a in arrs], C.byref(hits), None), "rays")
        return [a.download().reshape(n, k, c) if k else None for a, (k, c) in
                zip(arrs, [(k, c) for k in (nl, ao) for c in (3, 3, 1)])], hits.value

    full, hits = rays(3, 3)
    assert hits == ((view["flags"] & 1) != 0).sum()
    for nl, ao in ((0, 1), (0, 2), (1, 1), (1, 2), (2, 1), (2, 2), (3, 2), (2, 0)):
        few, count = rays(nl, ao)
        assert count == hits
        for a, b in zip(full, few):
            if b is not None:
                assert_bits_equal(np.ascontiguousarray(a[:, :b.shape[1]]), b, f"{nl} lights, {ao} occlusion rays")
