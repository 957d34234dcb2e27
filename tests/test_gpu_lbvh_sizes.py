"""The LBVH of animated entities (csrc/bvh.cu kBoxPyramid, kLbvh): node boxes from a pyramid of aligned groups.

Sizes sit around a group, a tile of 512 primitives, one and several tiles, and an odd number of them. A hit
does not depend on the tree, so the scan of a mesh built by the LBVH is byte for byte that of the SAH tree,
whose builder is checked against the host's.
"""
import numpy as np
import pytest

from tests.test_gpu_collapse import cast, down_rays

pytestmark = pytest.mark.gpu

DEVICE_SAH, DEVICE_LBVH = 0, 2


@pytest.mark.parametrize("triangles", [1, 2, 3, 5, 31, 511, 512, 513, 1023, 1025, 1537, 8191, 70001])
@pytest.mark.parametrize("coincident", [False, True])
def test_scan_equals_the_sah_trees(rgl, triangles, coincident):
    rng = np.random.default_rng(triangles)
    c = np.zeros((triangles, 3)) if coincident else rng.uniform(-20, 20, (triangles, 3))
    v = (c[:, None, :] + rng.uniform(-1, 1, (triangles, 3, 3))).astype(np.float32).reshape(-1, 3)
    xy = (rng.uniform(-1, 1, (8192, 2)) * (1.0 if coincident else 20.0)).astype(np.float32)
    xy[0] = v.reshape(-1, 3, 3)[0, :, :2].mean(axis=0)
    lib = rgl.lib()
    got = []
    try:
        for builder in (DEVICE_SAH, DEVICE_LBVH):
            rgl.check(lib.rgl_gb300_configure_blas_builder(builder))
            rgl.entity_set_id(rgl.entity_create(rgl.mesh_create(v, np.arange(3 * triangles, dtype=np.int32).reshape(triangles, 3))), 3)
            _, out = cast(rgl, down_rays(xy, np.float32(40.0)))
            assert out[2].any()
            got.append([o.tobytes() for o in out])
            rgl.check(lib.rgl_cleanup())
            rgl.check(lib.rgl_configure_logging(rgl.RGL_LOG_LEVEL_OFF, None, False))
    finally:
        rgl.check(lib.rgl_gb300_configure_blas_builder(DEVICE_SAH))
    assert got[0] == got[1]
