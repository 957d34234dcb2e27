"""Structure builds without the host in between, in kept device memory (csrc/build_memory.cpp, kSahLevels).

A mesh whose splits each take off one of ten clusters is deeper than an even tree, with a level per
cluster: the tree is the host builder's. Meshes that come and go reuse storage that was freed;
the scans must see the mesh that is there. Freed storage goes back to the device with rgl_cleanup.
"""
import ctypes as C

import numpy as np
import pytest

from robotecgpulidar_gb300 import scenes
from tests.test_gpu_collapse import DEVICE_SAH, HOST_SAH, cast, down_rays

pytestmark = pytest.mark.gpu


def nested_clusters(clusters, per_cluster):
    """Clusters at 4000, 4000 / 64, 4000 / 64^2, ... from the origin, each a tenth of that wide: of 32 bins
    over what is left, all but the farthest cluster share the first."""
    rng = np.random.default_rng(clusters)
    scale = (4000.0 / 64.0 ** np.arange(clusters)).repeat(per_cluster)
    c = np.stack([scale * rng.uniform(0.95, 1.05, scale.size), scale * rng.uniform(0.95, 1.05, scale.size), rng.uniform(-1, 1, scale.size)], 1)
    d = rng.uniform(-1, 1, (scale.size, 3, 3)) * np.stack([0.01 * scale, 0.01 * scale, np.full_like(scale, 0.1)], 1)[:, None, :]
    v = (c[:, None, :] + d).astype(np.float32).reshape(-1, 3)
    return v, np.arange(v.shape[0], dtype=np.int32).reshape(-1, 3), scale


@pytest.mark.parametrize("clusters,per_cluster", [(3, 700), (10, 2100), (12, 3000)])
def test_trees_deeper_than_an_even_one(rgl, clusters, per_cluster):
    v, idx, scale = nested_clusters(clusters, per_cluster)
    rng = np.random.default_rng(1)
    xy = (scale[::7, None] * rng.uniform(0.95, 1.05, (scale[::7].size, 2))).astype(np.float32)
    lib = rgl.lib()
    got = []
    try:
        for builder in (HOST_SAH, DEVICE_SAH):
            rgl.check(lib.rgl_gb300_configure_blas_builder(builder))
            rgl.entity_set_id(rgl.entity_create(rgl.mesh_create(v, idx)), 3)
            _, out = cast(rgl, down_rays(xy, np.float32(20.0)))
            nb, tb, ni = C.c_int64(), C.c_int64(), C.c_int32()
            rgl.check(lib.rgl_gb300_scene_get_stats(C.byref(nb), C.byref(tb), C.byref(ni)))
            got.append((nb.value, [o.tobytes() for o in out]))
            assert out[2].any()
            rgl.check(lib.rgl_cleanup())
            rgl.check(lib.rgl_configure_logging(rgl.RGL_LOG_LEVEL_OFF, None, False))
    finally:
        rgl.check(lib.rgl_gb300_configure_blas_builder(DEVICE_SAH))
    assert got[0] == got[1]


def sheet(cells, height):
    g = np.linspace(-8, 8, cells + 1).astype(np.float32)
    x, y = np.meshgrid(g, g, indexing="ij")
    v = np.stack([x.ravel(), y.ravel(), np.full(x.size, height, np.float32)], 1)
    a = (np.arange(cells)[:, None] * (cells + 1) + np.arange(cells)).reshape(-1)
    return v, np.concatenate([np.stack([a, a + 1, a + cells + 1], 1), np.stack([a + 1, a + cells + 2, a + cells + 1], 1)]).astype(np.int32)


def test_meshes_that_come_and_go(rgl):
    """Sheets of their own height and resolution, two alive at a time, the newest on top: the scan is, byte
    for byte, that of the newest sheet alone in a fresh state."""
    sheets = [sheet(cells, 0.5 * k) for k, cells in enumerate([1, 40, 7, 180, 64, 2, 180, 33, 90, 5])]
    xy = np.random.default_rng(3).uniform(-7.9, 7.9, (2048, 2)).astype(np.float32)
    fields = [rgl.RGL_FIELD_DISTANCE_F32, rgl.RGL_FIELD_ENTITY_ID_I32, rgl.RGL_FIELD_IS_HIT_I32, rgl.RGL_FIELD_XYZ_VEC3_F32]
    alone = []
    for k, (v, idx) in enumerate(sheets):
        rgl.entity_set_id(rgl.entity_create(rgl.mesh_create(v, idx)), 100 + k)
        alone.append([o.tobytes() for o in cast(rgl, down_rays(xy, np.float32(16.0)))[1]])
        rgl.check(rgl.lib().rgl_cleanup())
        rgl.check(rgl.lib().rgl_configure_logging(rgl.RGL_LOG_LEVEL_OFF, None, False))
    alive, node = [], None
    for k, (v, idx) in enumerate(sheets):
        mesh = rgl.mesh_create(v, idx)
        ent = rgl.entity_create(mesh)
        rgl.entity_set_id(ent, 100 + k)
        alive.append((mesh, ent))
        if len(alive) > 2:
            old_mesh, old_ent = alive.pop(0)
            rgl.check(rgl.lib().rgl_entity_destroy(old_ent))
            rgl.check(rgl.lib().rgl_mesh_destroy(old_mesh))
        if node is None:
            node, out = cast(rgl, down_rays(xy, np.float32(16.0)))
        else:
            rgl.graph_run(node["rays"])
            out = [rgl.result(node["out"], f) for f in fields]
        assert [o.tobytes() for o in out] == alone[k]


def test_cleanup_gives_the_storage_back(rgl):
    import torch

    lib = rgl.lib()
    rng = np.random.default_rng(4)
    n = 400_000  # about 90 MB of storage and temporaries
    v = rng.uniform(-10, 10, (3 * n, 3)).astype(np.float32)
    free = []
    for _ in range(3):
        rgl.entity_create(rgl.mesh_create(v, np.arange(3 * n, dtype=np.int32).reshape(n, 3)))
        cast(rgl, down_rays(np.zeros((64, 2), np.float32), np.float32(20.0)))
        rgl.check(lib.rgl_cleanup())
        rgl.check(lib.rgl_configure_logging(rgl.RGL_LOG_LEVEL_OFF, None, False))
        free.append(torch.cuda.mem_get_info()[0])
        assert free[-1] > torch.cuda.mem_get_info()[1] // 2
    assert abs(free[2] - free[0]) < 16 << 20  # nothing is kept from one to the next
