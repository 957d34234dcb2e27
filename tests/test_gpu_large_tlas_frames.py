"""Scenes above the one-block TLAS limit (2,048 instances) that move in batched frames: the refit and the enter
records are part of the captured frame."""
import numpy as np
import pytest

from robotecgpulidar_gb300 import scenes
from tests.test_gpu_collapse import down_rays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [2049, 3000])
def test_moved_instances_are_found_in_every_frame(rgl, count):
    side = int(np.ceil(np.sqrt(count)))
    k = np.arange(count)
    xy = np.stack([4.0 * (k % side), 4.0 * (k // side)], axis=1).astype(np.float32)
    cube = scenes.cube_mesh(0.5)
    mesh = rgl.mesh_create(cube.vertices, cube.indices)
    ents = [rgl.entity_create(mesh) for _ in range(count)]
    for i, e in enumerate(ents):
        rgl.entity_set_id(e, 10 + i)
        rgl.entity_set_transform(e, scenes.translation(xy[i, 0], xy[i, 1], 0.0))
    heads = []
    for part in (k[: count // 2], k[count // 2:]):
        n = {q: rgl.node() for q in ("rays", "trace", "out")}
        rgl.rays_from_mat3x4f(n["rays"], down_rays(xy[part] + np.float32(0.125), np.float32(32.0)))
        rgl.raytrace(n["trace"])
        rgl.points_yield(n["out"], [rgl.RGL_FIELD_DISTANCE_F32, rgl.RGL_FIELD_ENTITY_ID_I32])
        rgl.chain(n["rays"], n["trace"], n["out"])
        heads.append((n, part))
    batch = rgl.batch_create([n["rays"] for n, _ in heads])
    rgl.batch_configure_schedule(batch, autotune=False)
    try:
        rgl.batch_run(batch)
        height = np.zeros(count, np.float32)
        for frame in range(4):
            moved = k[frame::3]
            height[moved] = (moved % 5 + frame).astype(np.float32)
            for i in moved:
                rgl.entity_set_transform(ents[i], scenes.translation(xy[i, 0], xy[i, 1], float(height[i])))
            rgl.batch_run(batch)
            for n, part in heads:
                assert (rgl.result(n["out"], rgl.RGL_FIELD_ENTITY_ID_I32) == 10 + part).all()
                assert (rgl.result(n["out"], rgl.RGL_FIELD_DISTANCE_F32) == 31.5 - height[part]).all()
        assert rgl.batch_stats(batch)["replays"] >= 2
    finally:
        rgl.batch_destroy(batch)
