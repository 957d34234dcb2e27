"""Packed points of any layout (csrc/points.cu kFormatWords, kFormatBytes), compacted clouds with fields of
every element size, and merged clouds around the merge's tile.

The oracle is numpy: the packed bytes are the yielded fields' bytes side by side, paddings zero; a
compacted field is the raw field's kept rows; a merged field the inputs' rows after each other. Layouts
hold whole words, words of several fields, fields that straddle words, sizes that are no multiple of
four and points above 256 bytes; the counts sit around a tile of 1,024 points and of 512.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def names(rgl):
    return {"xyz": (rgl.RGL_FIELD_XYZ_VEC3_F32, 12), "dist": (rgl.RGL_FIELD_DISTANCE_F32, 4), "ent": (rgl.RGL_FIELD_ENTITY_ID_I32, 4),
            "ring": (rgl.RGL_FIELD_RING_ID_U16, 2), "ret": (rgl.RGL_FIELD_RETURN_TYPE_U8, 1), "i8": (rgl.RGL_FIELD_INTENSITY_U8, 1),
            "az": (rgl.RGL_FIELD_AZIMUTH_F32, 4), "time": (rgl.RGL_FIELD_TIME_STAMP_F64, 8), "pose": (rgl.RGL_FIELD_RAY_POSE_MAT3x4_F32, 48),
            "p8": (rgl.RGL_FIELD_PADDING_8, 1), "p16": (rgl.RGL_FIELD_PADDING_16, 2), "p32": (rgl.RGL_FIELD_PADDING_32, 4)}


LAYOUTS = ["xyz p32 dist ent", "xyz i8 ret ring az dist", "ret xyz p8 ring", "ring ring", "i8 ret p16", "p16 xyz p16", "ret xyz",
           "i8 p8 ring time p32", "ret pose i8 ring xyz", "pose pose pose pose pose xyz i8 ret p16", "p8 p8 p8 p8", "i8"]


@pytest.mark.parametrize("count", [1, 255, 1025, 5003])
def test_layouts_and_element_sizes(rgl, count):
    f = names(rgl)
    rng = np.random.default_rng(count)
    columns = [k for k in f if k not in ("p8", "p16", "p32")]
    rows = {k: rng.integers(0, 256, (count, f[k][1]), dtype=np.uint8) for k in columns}
    hit = rng.integers(0, 4, count) != 0
    hit[0] = True
    cloud = np.concatenate([hit.astype(np.int32).view(np.uint8).reshape(count, 4)] + [rows[k] for k in columns], axis=1)
    src, compact, kept = rgl.node(), rgl.node(), rgl.node()
    rgl.points_from_array(src, cloud, count, [rgl.RGL_FIELD_IS_HIT_I32] + [f[k][0] for k in columns])
    rgl.points_compact_by_field(compact)
    rgl.points_yield(kept, [f[k][0] for k in columns])
    rgl.chain(src, compact, kept)
    packed = []
    for layout in LAYOUTS:
        node = rgl.node()
        rgl.points_format(node, [f[k][0] for k in layout.split()])
        rgl.chain(compact, node)
        packed.append(node)
    rgl.graph_run(src)
    for k in columns:
        assert rgl.result_bytes(kept, f[k][0]).tobytes() == rows[k][hit].tobytes(), k
    for layout, node in zip(LAYOUTS, packed):
        expected = np.concatenate([rows[k][hit] if k in rows else np.zeros((hit.sum(), f[k][1]), np.uint8) for k in layout.split()], axis=1)
        assert rgl.result_bytes(node, rgl.RGL_FIELD_DYNAMIC_FORMAT).tobytes() == expected.tobytes(), layout


@pytest.mark.parametrize("counts", [(1, 1), (511, 512), (513, 3, 2049), (1, 5000, 257, 1023)])
def test_merged_clouds(rgl, counts):
    rng = np.random.default_rng(sum(counts))
    fields = [rgl.RGL_FIELD_XYZ_VEC3_F32, rgl.RGL_FIELD_DISTANCE_F32, rgl.RGL_FIELD_RING_ID_U16, rgl.RGL_FIELD_RETURN_TYPE_U8]
    sizes = [12, 4, 2, 1]
    merge, out = rgl.node(), rgl.node()
    rgl.points_spatial_merge(merge, fields)
    rgl.points_yield(out, fields)
    rgl.chain(merge, out)
    rows, first = [], None
    for c in counts:
        rows.append(rng.integers(0, 256, (c, sum(sizes)), dtype=np.uint8))
        src = rgl.node()
        rgl.points_from_array(src, rows[-1], c, fields)
        rgl.chain(src, merge)
        first = first or src
    rgl.graph_run(first)
    joined, at = np.concatenate(rows), 0
    for field, size in zip(fields, sizes):
        assert rgl.result_bytes(out, field).tobytes() == joined[:, at:at + size].tobytes()
        at += size
