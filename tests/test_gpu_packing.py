"""Tasks of the traversal: lane groups (up to 8 samples a beam), pooled samples (more), one lane per beam,
and the beams a task takes, which depend on the launch's size. Every packing must write the same bytes:
the sample counts sit around the switch (8 / 9), a warp's lanes (32 / 33) and the largest pattern (64), the
beam counts around a warp, a task's limit and the sizes at which a task takes one beam more."""
import numpy as np
import pytest

from robotecgpulidar_gb300 import scenes

pytestmark = pytest.mark.gpu

PATTERNS = [(0, 0), (1, 1), (1, 7), (1, 8), (2, 8), (1, 31), (1, 32), (3, 19), (3, 21)]


@pytest.mark.parametrize("layers,vertices", PATTERNS)
@pytest.mark.parametrize("beams", [1, 31, 33, 4864, 4865, 20011])
def test_every_packing_writes_the_same(rgl, layers, vertices, beams):
    lib = rgl.lib()
    rgl.spawn_scene(scenes.million_scene(seed=8, instances=6, spheres=2, cells=40, extent=80.0))
    rays = scenes.lidar_rays(1, beams, -12.0)
    fields = [rgl.RGL_FIELD_XYZ_VEC3_F32, rgl.RGL_FIELD_DISTANCE_F32, rgl.RGL_FIELD_ENTITY_ID_I32, rgl.RGL_FIELD_IS_HIT_I32]
    shaded = fields + [rgl.RGL_FIELD_INTENSITY_F32, rgl.RGL_FIELD_NORMAL_VEC3_F32, rgl.RGL_FIELD_INCIDENT_ANGLE_F32]
    for mode, wanted in ((rgl.RGL_RETURN_FIRST_LAST, fields), (rgl.RGL_RETURN_STRONGEST_SECOND_STRONGEST, shaded)):
        n = {k: rgl.node() for k in ("rays", "pose", "range", "trace", "out")}
        rgl.rays_from_mat3x4f(n["rays"], rays)
        rgl.rays_transform(n["pose"], scenes.trs((1.0, 2.0, 6.0), (0.01, 0.02, 0.3)))
        rgl.rays_set_range(n["range"], [[0.1, 60.0]])
        rgl.raytrace(n["trace"])
        rgl.check(lib.rgl_node_raytrace_configure_return_mode(n["trace"], mode))
        if layers:
            rgl.configure_beam_samples(n["trace"], layers, vertices)
            rgl.check(lib.rgl_node_raytrace_configure_beam_divergence(n["trace"], 0.05, 0.03))
        rgl.points_yield(n["out"], wanted)
        rgl.chain(n["rays"], n["pose"], n["range"], n["trace"], n["out"])
        got = []
        try:
            for packing in (rgl.PACK_SERIAL, rgl.PACK_LANE_GROUP):
                rgl.check(lib.rgl_gb300_configure_trace_schedule(128, packing, 1, 128))
                rgl.graph_run(n["rays"])
                got.append([rgl.result_bytes(n["out"], f).tobytes() for f in wanted])
        finally:
            rgl.check(lib.rgl_gb300_configure_trace_schedule(256, rgl.PACK_LANE_GROUP, 1, 128))
        assert np.frombuffer(got[0][3], np.int32).any()
        for f, a, b in zip(wanted, *got):
            assert a == b, f"field {f} differs between packings"
