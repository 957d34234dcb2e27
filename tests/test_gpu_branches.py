"""Graphs with several raytraces enqueue their branches on several streams. The merged cloud must equal the
concatenation of the sensors' own graphs, byte for byte: with as many branches as streams, one more and
fewer, with a node that two branches share, replayed with new poses and with CUDA graphs off."""
import numpy as np
import pytest

from robotecgpulidar_gb300 import scenes

pytestmark = pytest.mark.gpu


def sensor(rgl, beams, azimuths):
    n = {k: rgl.node() for k in ("rays", "pose", "range", "trace", "cmp")}
    rgl.rays_from_mat3x4f(n["rays"], scenes.lidar_rays(beams, azimuths))
    rgl.rays_transform(n["pose"], scenes.translation(0, 0, 5))
    rgl.rays_set_range(n["range"], [[0.1, 60.0]])
    rgl.raytrace(n["trace"])
    rgl.points_compact_by_field(n["cmp"])
    rgl.chain(n["rays"], n["pose"], n["range"], n["trace"], n["cmp"])
    return n


@pytest.mark.parametrize("count", [2, 3, 8, 9, 10, 12])
@pytest.mark.parametrize("graphs", [True, False])
def test_merged_branches_equal_their_own_runs(rgl, count, graphs):
    lib = rgl.lib()
    rgl.spawn_scene(scenes.million_scene(seed=4, instances=8, spheres=2, cells=40, extent=80.0))
    fields = [rgl.RGL_FIELD_XYZ_VEC3_F32, rgl.RGL_FIELD_DISTANCE_F32, rgl.RGL_FIELD_ENTITY_ID_I32]
    fused = [sensor(rgl, 8 + 3 * i, 100 + 17 * i) for i in range(count)]
    alone = [sensor(rgl, 8 + 3 * i, 100 + 17 * i) for i in range(count)]
    merge, out = rgl.node(), rgl.node()
    rgl.points_spatial_merge(merge, fields)
    rgl.points_format(out, fields)
    rgl.chain(merge, out)
    for s in fused:
        rgl.add_child(s["cmp"], merge)
    # a second consumer of the first sensor's raytrace: its own branch
    extra = rgl.node()
    rgl.points_yield(extra, fields)
    rgl.add_child(fused[0]["trace"], extra)
    outs = []
    for s in alone:
        y = rgl.node()
        rgl.points_yield(y, fields)
        rgl.chain(s["cmp"], y)
        outs.append(y)
    rgl.check(lib.rgl_gb300_configure_cuda_graphs(graphs))
    try:
        for frame in range(3):
            for i, (a, b) in enumerate(zip(fused, alone)):
                tf = scenes.trs((3.0 * i - 10 + frame, 2.0 - i, 4.0 + 0.3 * i), (0.0, 0.01 * i, 0.4 * i + frame))
                rgl.rays_transform(a["pose"], tf)
                rgl.rays_transform(b["pose"], tf)
            rgl.graph_run(fused[0]["rays"])
            got = {f: rgl.result_bytes(merge, f) for f in fields}
            formatted = rgl.result_bytes(out, rgl.RGL_FIELD_DYNAMIC_FORMAT)
            whole = rgl.result(extra, rgl.RGL_FIELD_DISTANCE_F32)
            want = {f: [] for f in fields}
            for s, y in zip(alone, outs):
                rgl.graph_run(s["rays"])
                for f in fields:
                    want[f].append(rgl.result_bytes(y, f))
            for f in fields:
                assert got[f].tobytes() == np.concatenate(want[f]).tobytes(), (frame, f)
            assert formatted.reshape(-1, 20)[:, :12].tobytes() == got[fields[0]].tobytes()
            assert np.isfinite(whole).sum() == len(want[fields[1]][0]) // 4
    finally:
        rgl.check(lib.rgl_gb300_configure_cuda_graphs(True))
