"""Point queries, ambient occlusion and the baseline march over as many objects
as their kernels' copy of the object table holds (198 records of 248 bytes in
48 KB), and one less and more, up to 300: bit-exact with the oracle."""
import numpy as np
import pytest

from conftest import assert_bits_equal
from test_many_objects_gpu import _context, _objects
from test_tiled_gpu import PLANES, _params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_objs", [2, 12, 13, 32, 33, 163, 164, 198, 199, 300])
def test_queries_over_many_objects(oracle, small_scene, n_objs):
    from rkifield_b200 import scenes
    v = small_scene["vox"]
    objs = _objects(small_scene, n_objs - 1, seed=n_objs)
    assert len(objs) == n_objs
    sc = oracle.Scene(objs, pool_words=v.words, brick_maps=v.map)
    rng = np.random.default_rng(n_objs)
    pts = rng.uniform(-32.0, 32.0, (3001, 3)).astype(np.float32)
    nrm = rng.standard_normal((3001, 3))
    nrm = (nrm / np.linalg.norm(nrm, axis=1, keepdims=True)).astype(np.float32)
    d_ref, g_ref, m_ref = oracle.query_points(sc, pts.ravel())
    ao_ref = oracle.sdf_ao(sc, pts.ravel(), nrm.ravel())
    ctx = _context(small_scene, objs)
    try:
        for n in (1, 3001):
            d, g, m = ctx.query_points(pts[:n])
            assert_bits_equal(d, d_ref[:n], "distance")
            assert_bits_equal(g, g_ref[:3 * n], "gradient")
            assert_bits_equal(m, m_ref[:n], "material")
            assert_bits_equal(ctx.sdf_ao(pts[:n], nrm[:n]), ao_ref[:n], "occlusion")
        if n_objs in (164, 198):
            w, h = 48, 32
            cam = scenes.camera_uniforms((45.0, 22.0, 55.0), (0.0, -4.0, 0.0), w, h)
            ref = oracle.march(sc, cam, _params(0), w, h, with_reference_planes=True)
            got = ctx.march(cam, _params(0), w, h, reference_planes=True, plain=True)
            for k in PLANES:
                assert_bits_equal(got[k], ref[k], k)
    finally:
        ctx.close()


@pytest.mark.parametrize("n_objs", [0, 1, 12, 13, 198, 199])
def test_distances_alone(small_scene, n_objs):
    """A query without gradients answers as one with them, on both sides of the
    sizes at which it takes a thread per point."""
    import ctypes as C

    from rkifield_b200 import _abi as abi
    objs = ([small_scene["obj"]] if n_objs == 1 else _objects(small_scene, n_objs - 1, seed=3)) if n_objs else []
    ctx = _context(small_scene, objs)
    try:
        pts = np.random.default_rng(n_objs).uniform(-32.0, 32.0, (32769, 3)).astype(np.float32)
        d_ref, _, m_ref = ctx.query_points(pts)
        for n in (1, 16383, 16384, 32767, 32768, 32769):
            for want_d, want_m in ((True, False), (False, True), (True, True)):
                d, m = np.zeros(n, np.float32), np.zeros(n, np.uint16)
                abi.check(ctx.lib.rkf_query_points(ctx.h, pts.ctypes.data, n, d.ctypes.data if want_d else None, None,
                                                   m.ctypes.data if want_m else None, abi.RKF_MEM_HOST), "query")
                assert_bits_equal(d, d_ref[:n] if want_d else 0 * d, f"{n}: distance")
                np.testing.assert_array_equal(m, m_ref[:n] if want_m else 0 * m)
    finally:
        ctx.close()
