"""Scenes whose instance count crosses the one-block TLAS limit (2,048) downwards, and small scenes beside
large ones: each keeps its own build scratch, and the one-block kernel's shared-memory limit is not
lowered by a smaller scene."""
import numpy as np
import pytest

from robotecgpulidar_gb300 import scenes

pytestmark = pytest.mark.gpu


def grid(rgl, scene, mesh, count):
    ents = []
    for i in range(count):
        e = rgl.entity_create_in(scene, mesh)
        rgl.entity_set_transform(e, scenes.translation(4.0 * (i % 64), 4.0 * (i // 64), 0.0))
        rgl.entity_set_id(e, 10 + i)
        ents.append(e)
    return ents


def ids_below(rgl, scene, count):
    i = np.arange(count)
    m = np.zeros((count, 3, 4), np.float32)
    m[:, 0, 0], m[:, 1, 1], m[:, 2, 2] = 1.0, -1.0, -1.0
    m[:, 0, 3], m[:, 1, 3], m[:, 2, 3] = 4.0 * (i % 64) + 0.125, 4.0 * (i // 64) + 0.125, 8.0
    n = {k: rgl.node() for k in ("rays", "trace", "out")}
    rgl.rays_from_mat3x4f(n["rays"], m)
    rgl.raytrace_in(n["trace"], scene)
    rgl.points_yield(n["out"], [rgl.RGL_FIELD_ENTITY_ID_I32])
    rgl.chain(n["rays"], n["trace"], n["out"])
    rgl.graph_run(n["rays"])
    return rgl.result(n["out"], rgl.RGL_FIELD_ENTITY_ID_I32)


@pytest.mark.parametrize("small", [1, 5, 2048])
def test_scene_shrinks_below_the_limit(rgl, small):
    scene, cube = rgl.scene_create(), scenes.cube_mesh(0.5)
    mesh = rgl.mesh_create(cube.vertices, cube.indices)
    ents = grid(rgl, scene, mesh, 2100)
    assert (ids_below(rgl, scene, 2100) == 10 + np.arange(2100)).all()
    for e in ents[small:]:
        rgl.check(rgl.lib().rgl_entity_destroy(e))
    assert (ids_below(rgl, scene, small) == 10 + np.arange(small)).all()


def test_small_scene_beside_a_large_one(rgl):
    cube = scenes.cube_mesh(0.5)
    mesh = rgl.mesh_create(cube.vertices, cube.indices)
    large, little = rgl.scene_create(), rgl.scene_create()
    ents = grid(rgl, large, mesh, 2000)
    assert (ids_below(rgl, large, 2000) == 10 + np.arange(2000)).all()
    grid(rgl, little, mesh, 3)
    assert (ids_below(rgl, little, 3) == 10 + np.arange(3)).all()
    rgl.entity_set_id(ents[1999], 7)  # the large scene's rebuild after the small one's
    assert ids_below(rgl, large, 2000)[1999] == 7
