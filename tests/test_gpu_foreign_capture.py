"""Another part of the process captures a CUDA graph while the library gives scene storage back: the
capture must come through. A wait for the whole device would end it (it is not allowed while any stream of
the context is being captured), so freed storage waits for the events of the work that may read it.

The capture runs in thread-local mode on the test's thread, the library's calls on another one.
"""
import ctypes as C
import threading

import numpy as np
import pytest

from robotecgpulidar_gb300 import scenes
from tests.test_gpu_collapse import cast, down_rays

pytestmark = pytest.mark.gpu


def captured(calls):
    """Runs `calls` on a thread of its own inside a capture of this one and replays what was captured."""
    import torch

    x = torch.zeros(1024, device="cuda")
    stream, graph, failure = torch.cuda.Stream(), torch.cuda.CUDAGraph(), []

    def work():
        try:
            calls()
        except Exception as e:  # noqa: BLE001: reported by the test's thread
            failure.append(e)

    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        graph.capture_begin(capture_error_mode="thread_local")
        x += 1.0
        t = threading.Thread(target=work)
        t.start()
        t.join()
        graph.capture_end()
    graph.replay()
    torch.cuda.synchronize()
    assert not failure, failure
    assert (x == 1.0).all()


def cube(rgl):
    m = scenes.cube_mesh(0.5)
    return rgl.mesh_create(m.vertices, m.indices)


RAY = down_rays(np.array([[0.1, 0.2]], np.float32), np.float32(8.0))


def test_meshes_go_while_another_library_captures(rgl):
    lib = rgl.lib()
    mesh = cube(rgl)
    ent = rgl.entity_create(mesh)
    nodes, (dist, _, hit, _) = cast(rgl, RAY)
    assert hit.all()

    def calls():
        rgl.check(lib.rgl_entity_destroy(ent))
        rgl.check(lib.rgl_mesh_destroy(mesh))
        rgl.entity_create(cube(rgl))
        rgl.graph_run(nodes["rays"])
        assert rgl.result(nodes["out"], rgl.RGL_FIELD_IS_HIT_I32).all()
        rgl.check(lib.rgl_cleanup())
        rgl.check(lib.rgl_configure_logging(rgl.RGL_LOG_LEVEL_OFF, None, False))

    captured(calls)


def test_a_served_scene_grows_while_another_library_captures(rgl):
    scene, mesh = rgl.scene_create(), cube(rgl)
    srv = rgl.Server(1 << 30, 2)
    try:
        pattern = srv.add_pattern(RAY)
        identity = scenes.translation(0.0, 0.0, 0.0)

        def ask():
            req = srv.submit(scene, pattern, identity, rgl.RGL_RETURN_FIRST, 0.1, 100.0)
            srv.wait(req)
            assert len(srv.result(req, rgl.RGL_FIELD_ENTITY_ID_I32)) == 1

        rgl.entity_create_in(scene, mesh)
        ask()
        for k in range(8):  # the instance records move: their old place is freed by the server's thread
            rgl.entity_set_transform(rgl.entity_create_in(scene, mesh), scenes.translation(4.0 * (k + 1), 0.0, 0.0))
        captured(ask)
    finally:
        srv.destroy()
