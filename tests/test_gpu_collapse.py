"""The wide collapse (csrc/collapse.cuh): eight lanes per wide node, in one block for the TLAS of up to
2,048 instances and in one cooperative launch for meshes and larger TLASes.

Sizes sit around what a node, a warp and a block hold at once (8 children, 4 nodes, 16 nodes of a
128-thread block) and around the grid's growth (one block per 256 primitives) and the one-block limit.
A mesh's tree is compared with the host builder's (node bytes equal, scans byte-identical); a TLAS is
checked by casting one ray straight down on every instance of a spaced grid: each must hit its own
instance, at the distance that follows from the poses (exact in float: small integers and halves).
"""
import ctypes as C

import numpy as np
import pytest

from robotecgpulidar_gb300 import scenes

pytestmark = pytest.mark.gpu

DEVICE_SAH, HOST_SAH = 0, 1


def down_rays(xy, z):
    """Rays at (x, y, z) whose local +Z is world -Z."""
    m = np.zeros((len(xy), 3, 4), np.float32)
    m[:, 0, 0], m[:, 1, 1], m[:, 2, 2] = 1.0, -1.0, -1.0
    m[:, 0, 3], m[:, 1, 3], m[:, 2, 3] = xy[:, 0], xy[:, 1], z
    return m


def cast(rgl, rays):
    n = {k: rgl.node() for k in ("rays", "trace", "out")}
    fields = [rgl.RGL_FIELD_DISTANCE_F32, rgl.RGL_FIELD_ENTITY_ID_I32, rgl.RGL_FIELD_IS_HIT_I32, rgl.RGL_FIELD_XYZ_VEC3_F32]
    rgl.rays_from_mat3x4f(n["rays"], rays)
    rgl.raytrace(n["trace"])
    rgl.points_yield(n["out"], fields)
    rgl.chain(n["rays"], n["trace"], n["out"])
    rgl.graph_run(n["rays"])
    return n, [rgl.result(n["out"], f) for f in fields]


@pytest.mark.parametrize("count", [1, 2, 7, 8, 9, 33, 64, 65, 257, 2047, 2048, 2049, 4097])
def test_every_instance_is_found(rgl, count):
    side = int(np.ceil(np.sqrt(count)))
    k = np.arange(count)
    xy = np.stack([4.0 * (k % side), 4.0 * (k // side)], axis=1).astype(np.float32)
    height = (k % 5).astype(np.float32)
    mesh = rgl.mesh_create(*(lambda m: (m.vertices, m.indices))(scenes.cube_mesh(0.5)))
    ents = []
    for i in range(count):
        e = rgl.entity_create(mesh)
        rgl.entity_set_transform(e, scenes.translation(xy[i, 0], xy[i, 1], height[i]))
        rgl.entity_set_id(e, 10 + i)
        ents.append(e)
    rays = down_rays(xy + np.float32(0.125), np.float32(32.0))
    n, (dist, ent, hit, _) = cast(rgl, rays)
    assert hit.all()
    assert (ent == 10 + k).all()
    assert (dist == 32.0 - (height + 0.5)).all()
    # moved: the rebuild (or refit) after poses changed, heights reversed
    for i in range(count):
        rgl.entity_set_transform(ents[i], scenes.translation(xy[i, 0], xy[i, 1], 4.0 - height[i]))
    rgl.graph_run(n["rays"])
    dist, ent = rgl.result(n["out"], rgl.RGL_FIELD_DISTANCE_F32), rgl.result(n["out"], rgl.RGL_FIELD_ENTITY_ID_I32)
    assert (ent == 10 + k).all()
    assert (dist == 32.0 - (4.5 - height)).all()


@pytest.mark.parametrize("triangles", [1, 2, 3, 4, 15, 16, 17, 64, 127, 255, 256, 257, 511, 513, 4095, 10007])
def test_mesh_tree_equals_the_host_builders(rgl, triangles):
    rng = np.random.default_rng(triangles)
    c = rng.uniform(-6, 6, size=(triangles, 3)).astype(np.float32)
    v = (c[:, None, :] + rng.uniform(-1, 1, size=(triangles, 3, 3))).astype(np.float32).reshape(-1, 3)
    got = []
    lib = rgl.lib()
    try:
        for builder in (HOST_SAH, DEVICE_SAH):
            rgl.check(lib.rgl_gb300_configure_blas_builder(builder))
            mesh = rgl.mesh_create(v, np.arange(3 * triangles, dtype=np.int32).reshape(triangles, 3))
            rgl.entity_set_id(rgl.entity_create(mesh), 3)
            xy = rng.uniform(-7, 7, size=(4096, 2)).astype(np.float32) if not got else xy
            _, out = cast(rgl, down_rays(xy, np.float32(20.0)))
            nb, tb, ni = C.c_int64(), C.c_int64(), C.c_int32()
            rgl.check(lib.rgl_gb300_scene_get_stats(C.byref(nb), C.byref(tb), C.byref(ni)))
            got.append((nb.value, [o.tobytes() for o in out]))
            rgl.check(lib.rgl_cleanup())
            rgl.check(lib.rgl_configure_logging(rgl.RGL_LOG_LEVEL_OFF, None, False))
    finally:
        rgl.check(lib.rgl_gb300_configure_blas_builder(DEVICE_SAH))
    assert got[0][0] == got[1][0]
    assert got[0][1] == got[1][1]
