"""Vertices that are not numbers, or infinite, in meshes and animations: their triangles are never hit (no
comparison of the exact test holds), and nobody else's hit may change, whichever builder made the tree. A NaN
coordinate leaves the box of its triangle's other vertices; an infinite one makes boxes infinite up to the
root, and the slab test must still enter them.
"""
import numpy as np
import pytest

from tests.test_gpu_collapse import cast, down_rays

pytestmark = pytest.mark.gpu

DEVICE_SAH, HOST_SAH, DEVICE_LBVH = 0, 1, 2


def soup(rng, triangles):
    c = rng.uniform(-20, 20, (triangles, 1, 3))
    return (c + rng.uniform(-1, 1, (triangles, 3, 3))).astype(np.float32)


def with_broken(rng, clean, kind):
    """`clean` with a triangle in ten more, one vertex of each broken in one to three coordinates."""
    extra = soup(rng, max(1, len(clean) // 10))
    for t in extra:
        which = rng.choice(3, size=rng.integers(1, 4), replace=False)
        t[rng.integers(0, 3), which] = {"nan": np.nan, "inf": np.inf, "-inf": -np.inf}[kind]
    at = np.sort(rng.integers(0, len(clean) + 1, len(extra)))
    return np.ascontiguousarray(np.insert(clean, at, extra, axis=0))


def scan(rgl, v, xy):
    mesh = rgl.mesh_create(v.reshape(-1, 3), np.arange(3 * len(v), dtype=np.int32).reshape(-1, 3))
    rgl.entity_set_id(rgl.entity_create(mesh), 3)
    out = cast(rgl, down_rays(xy, np.float32(40.0)))[1]
    rgl.check(rgl.lib().rgl_cleanup())
    rgl.check(rgl.lib().rgl_configure_logging(rgl.RGL_LOG_LEVEL_OFF, None, False))
    return out


@pytest.mark.parametrize("kind", ["nan", "inf", "-inf"])
@pytest.mark.parametrize("triangles", [7, 300, 1100, 9000])
def test_nobody_elses_hit_changes(rgl, kind, triangles):
    rng = np.random.default_rng(triangles)
    clean = soup(rng, triangles)
    xy = rng.uniform(-20, 20, (4096, 2)).astype(np.float32)
    xy[0] = clean[0, :, :2].mean(axis=0)
    broken = with_broken(rng, clean, kind)
    assert len(broken) > len(clean)
    lib = rgl.lib()
    want = [o.tobytes() for o in scan(rgl, clean, xy)]
    try:
        for builder in (DEVICE_SAH, DEVICE_LBVH):
            rgl.check(lib.rgl_gb300_configure_blas_builder(builder))
            got = scan(rgl, broken, xy)
            assert got[2].any()
            assert [o.tobytes() for o in got] == want
    finally:
        rgl.check(lib.rgl_gb300_configure_blas_builder(DEVICE_SAH))
