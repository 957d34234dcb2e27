"""Workloads of a lidar simulator on this framework, for timing and for comparing outputs.

A case is a dict of plain values; ``kind`` says which part of a simulator's frame loop it stands for:

* ``scan``: one sensor over a resident scene. Each pass moves the sensor (rays transform), runs the graph and
  reads the results into pinned host buffers, as an engine plugin does every tick.
* ``moving``: the same scan while a share of the scene's entities gets a new pose every pass.
* ``animated``: the same scan over an entity whose vertices are replaced every pass (external animation).
* ``load``: a mesh that was not there before (a streamed terrain tile) is created, scanned once and destroyed.
* ``fusion``: several sensors in one graph, their compacted clouds merged and formatted as one.
* ``batch``: a rig of uneven sensors traced as one batched frame, a fifth of the entities re-posed every frame.
* ``serve``: requests of a fleet of robots, submitted together to the serving loop and read back.

Worlds come from ``robotecgpulidar_gb300.scenes``: ``plain`` is its 20,768-triangle scene in one entity, ``hills`` a
value-noise terrain of ``cells`` x ``cells`` quads with ``instances`` posed spheres of 5,120 triangles each
(cells 512, instances 93: the 1,000,448-triangle scene). Scan shapes are those of the framework's own
configurations (16x1800 .. 128x2048 spinning lidars, a 120x640 solid-state grid) and odd ones near them.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from robotecgpulidar_gb300 import rgl, scenes

RANGE = [0.1, 300.0]
POSES = 4  # sensor and entity poses a state cycles through
XYZ, DIST, ENT, HIT = rgl.RGL_FIELD_XYZ_VEC3_F32, rgl.RGL_FIELD_DISTANCE_F32, rgl.RGL_FIELD_ENTITY_ID_I32, rgl.RGL_FIELD_IS_HIT_I32
FORMATS = {
    # XYZ, distance, entity id: 20 bytes, whole words
    "xyzde": [XYZ, DIST, ENT],
    # x, y, z, intensity u8, return type u8, channel u16, azimuth, elevation, distance, time stamp u32: the
    # point type of autonomous driving stacks, 32 bytes with 1- and 2-byte fields
    "ircaedt": [XYZ, rgl.RGL_FIELD_INTENSITY_U8, rgl.RGL_FIELD_RETURN_TYPE_U8, rgl.RGL_FIELD_RING_ID_U16, rgl.RGL_FIELD_AZIMUTH_F32,
                rgl.RGL_FIELD_ELEVATION_F32, DIST, rgl.RGL_FIELD_TIME_STAMP_U32],
    # what a perception training set stores besides the position: normals, incident angles, ids
    "labels": [XYZ, rgl.RGL_FIELD_NORMAL_VEC3_F32, rgl.RGL_FIELD_INCIDENT_ANGLE_F32, ENT, rgl.RGL_FIELD_RAY_IDX_U32,
               rgl.RGL_FIELD_LASER_RETRO_F32],
}
MODES = {"first": rgl.RGL_RETURN_FIRST, "last": rgl.RGL_RETURN_LAST, "first_last": rgl.RGL_RETURN_FIRST_LAST,
         "last_strongest": rgl.RGL_RETURN_LAST_STRONGEST}
RETURNS = {"first": 1, "last": 1, "first_last": 2, "last_strongest": 2}


def _scan(name, world, channels, azimuths, **more):
    case = {"name": name, "kind": "scan", "world": world, "cells": 0, "instances": 0, "channels": channels, "azimuths": azimuths,
            "layers": 0, "vertices": 0, "mode": "first", "noise": False, "format": ""}
    if world == "hills":
        case |= {"cells": 512, "instances": 93}
    return case | more


def listed():
    return [
        # a 16-channel sensor of a small robot, an odd azimuth count: launches and latency
        _scan("scan-small", "plain", 16, 225),
        # 32 x 1024 first return over a simple scene: the plain single-sensor simulation
        _scan("scan-plain", "plain", 32, 1024),
        # 64 x 2048 with sensor noise, moved into the vehicle's frame, compacted and packed for a publisher
        _scan("scan-publish", "plain", 64, 2048, noise=True, format="xyzde"),
        # 128 x 2048 with five rays a beam and two returns over 1M triangles: the high-end sensor in a city block
        _scan("scan-million", "hills", 128, 2048, layers=1, vertices=4, mode="first_last", noise=True),
        # the default beam divergence pattern (58 rays a beam) with a strongest return (intensity): most rays of all
        _scan("scan-divergent", "hills", 64, 1024, layers=3, vertices=19, mode="last_strongest", format="ircaedt"),
        # a solid-state sensor that labels its points, ragged size
        _scan("scan-labels", "hills", 120, 641, format="labels"),
        # traffic: a fifth of 94 entities moves every tick
        _scan("moving", "hills", 64, 2048, kind="moving", share=0.2),
        # a deforming surface (a tarpaulin, water) of 33,282 triangles
        {"name": "animated", "kind": "animated", "cells": 129, "channels": 32, "azimuths": 1024},
        # a terrain tile of 131,072 triangles streamed in
        {"name": "load", "kind": "load", "cells": 256, "channels": 32, "azimuths": 512},
        # four corner sensors of one vehicle fused into one cloud
        _scan("fusion", "hills", 32, 1024, kind="fusion", sensors=4, cells=256, instances=31),
        # a frame of sixteen uneven sensors
        _scan("batch", "hills", 0, 0, kind="batch", sensors=16, layers=1, vertices=4, mode="first_last", share=0.2),
        # a burst of robots' requests
        {"name": "serve", "kind": "serve", "cells": 512, "instances": 93, "patterns": 8, "requests": 48, "smallest": 10000,
         "largest": 150000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["scan", "scan", "scan", "moving", "animated", "load", "fusion", "batch", "serve"])
    if kind == "animated":
        return {"kind": kind, "cells": _log(rng, 12, 181), "channels": rng.choice([16, 32, 64]), "azimuths": _log(rng, 200, 1500)}
    if kind == "load":
        return {"kind": kind, "cells": _log(rng, 20, 400), "channels": rng.choice([16, 32, 64]), "azimuths": _log(rng, 200, 1500)}
    cells = _log(rng, 64, 512)
    instances = _log(rng, 3, 250)
    if kind == "serve":
        return {"kind": kind, "cells": cells, "instances": instances, "patterns": rng.randint(3, 8), "requests": _log(rng, 4, 48),
                "smallest": 10000, "largest": _log(rng, 30000, 150000)}
    world = "plain" if kind == "scan" and rng.random() < 0.3 else "hills"
    channels = rng.choice([1, 16, 32, 40, 64, 128])
    case = _scan("", world, channels, max(1, _log(rng, 3000, 262144) // channels), kind=kind)
    case.pop("name")
    if world == "hills":
        case |= {"cells": cells, "instances": instances}
    case["mode"] = rng.choice(sorted(MODES))
    case["noise"] = rng.random() < 0.4
    if kind == "scan":
        case["format"] = rng.choice(["", "xyzde", "ircaedt", "labels"])
    if rng.random() < 0.5:
        layers, vertices = rng.choice([(1, 4), (2, 8), (3, 19)])
        fits = 3_800_000 // (channels * (1 + layers * vertices))
        case |= {"layers": layers, "vertices": vertices, "azimuths": max(1, min(case["azimuths"], fits))}
    if kind in ("moving", "batch"):
        case["share"] = rng.uniform(0.05, 1.0)
    if kind == "fusion":
        case |= {"sensors": rng.randint(2, 6), "azimuths": max(1, min(case["azimuths"], 65536 // channels)), "layers": 0, "vertices": 0,
                 "mode": "first"}
    if kind == "batch":
        case |= {"sensors": rng.randint(2, 16), "channels": 0, "azimuths": 0, "layers": 1, "vertices": 4}
    return case


# ---------------------------------------------------------------- inputs


def _world(case, seed):
    if case.get("world", "hills") == "plain":
        return scenes.plain_scene(seed)
    triangles = 2 * case["cells"] ** 2 + 5120 * case["instances"]
    return scenes.million_scene(seed, instances=case["instances"], spheres=8, cells=case["cells"], extent=512.0 * math.sqrt(triangles / 1e6))


def _extent(world):
    return world.heightfield[1] if world.heightfield is not None else 200.0


def _sensor_poses(world, rng, count, height=(1.5, 6.0)):
    """A sensor driving over the terrain: `count` poses some metres apart."""
    extent = _extent(world)
    x, y = rng.uniform(-0.2 * extent, 0.2 * extent, 2)
    yaw, z = rng.uniform(-np.pi, np.pi), rng.uniform(*height)
    out = []
    for k in range(count):
        px, py = x + 2.0 * k * math.cos(yaw), y + 2.0 * k * math.sin(yaw)
        ground = world.ground_height(px, py) if world.heightfield is not None else 0.5
        out.append(scenes.trs((px, py, ground + z), (0.0, 0.0, yaw + 0.02 * k)))
    return out


def _tile(cells, rng, extent=120.0, height=4.0):
    """A heightfield mesh of 2 * cells^2 triangles: smooth waves and a little roughness."""
    x, y = np.meshgrid(np.linspace(0, 1, cells + 1), np.linspace(0, 1, cells + 1))
    h = sum(a * np.sin(2 * np.pi * (u * x + v * y) + p) for a, u, v, p in
            zip(rng.uniform(0.1, 0.4, 6), rng.uniform(0.5, 6, 6), rng.uniform(0.5, 6, 6), rng.uniform(0, 6, 6)))
    return scenes.terrain_mesh(cells, cells, extent, extent, height * 0.3 * h + rng.uniform(0, 0.05, h.shape))


def _pinned(count, width, dtype):
    return torch.zeros((count, width) if width > 1 else (count,), dtype=dtype, pin_memory=True)


class Reader:
    """Pinned host buffers for a node's fields, filled after a run up to the count of points."""

    def __init__(self, node, capacity, fields, point_size=0):
        self.node, self.cnt, self.sz = node, C.c_int32(), C.c_int32()
        self.fields = []
        for f in fields:
            if f == rgl.RGL_FIELD_DYNAMIC_FORMAT:
                buf = _pinned(capacity * point_size, 1, torch.uint8)
            else:
                dt, width = rgl.FIELD_DTYPE[f]
                buf = _pinned(capacity, width, torch.float32 if np.dtype(dt).kind == "f" else torch.int32)
            self.fields.append((f, C.c_void_p(buf.data_ptr()), buf))

    def __call__(self):
        lib = rgl.lib()
        rgl.check(lib.rgl_graph_get_result_size(self.node, self.fields[0][0], C.byref(self.cnt), C.byref(self.sz)))
        for f, p, _ in self.fields:
            rgl.check(lib.rgl_graph_get_result_data(self.node, f, p))
        return [buf for _, _, buf in self.fields], self.cnt.value


class State:
    """What a simulator holds: scenes, meshes, graphs, buffers. Destroyed with the object."""

    def __init__(self, kind):
        self.kind, self.k = kind, 0
        self.graphs, self.meshes, self.scene, self.batch, self.server = [], [], None, None, None

    def __del__(self):
        lib = rgl.lib()
        if self.server is not None:
            self.server.destroy()
        if self.batch is not None:
            lib.rgl_gb300_batch_destroy(self.batch)
        for g in self.graphs:
            lib.rgl_graph_destroy(g)
        if self.scene is not None:
            lib.rgl_gb300_scene_destroy(self.scene)
        for m in self.meshes:
            lib.rgl_mesh_destroy(m)


def _trace_nodes(case, scene, rays, pose, ring=0):
    """rays -> pose -> range [-> ring ids] -> raytrace, linked."""
    n = {k: rgl.node() for k in ("rays", "pose", "range", "trace")}
    rgl.rays_from_mat3x4f(n["rays"], rays)
    rgl.rays_transform(n["pose"], pose)
    rgl.rays_set_range(n["range"], [RANGE])
    rgl.raytrace_in(n["trace"], scene)
    lib = rgl.lib()
    rgl.check(lib.rgl_node_raytrace_configure_return_mode(n["trace"], MODES[case.get("mode", "first")]))
    rgl.check(lib.rgl_node_raytrace_configure_default_intensity(n["trace"], 150.0))
    if case.get("layers"):
        rgl.configure_beam_samples(n["trace"], case["layers"], case["vertices"])
        rgl.check(lib.rgl_node_raytrace_configure_beam_divergence(n["trace"], 0.003, 0.0015))
    head = [n["rays"], n["pose"], n["range"]]
    if ring:
        ids = np.arange(ring, dtype=np.int32)
        n["ring"] = rgl.node()
        rgl.check(lib.rgl_node_rays_set_ring_ids(C.byref(n["ring"]), rgl.ptr(ids), ring))
        head.append(n["ring"])
    rgl.chain(*head, n["trace"])
    return n


def _point_nodes(case, n, seed, vehicle=None):
    """The point nodes after the raytrace: noise, vehicle frame, compaction, output."""
    lib, last = rgl.lib(), n["trace"]
    if case.get("noise"):
        a, d = rgl.node(), rgl.node()
        rgl.check(lib.rgl_node_gaussian_noise_angular_hitpoint(C.byref(a), 0.0, 0.0005, rgl.RGL_AXIS_Z))
        rgl.check(lib.rgl_node_gaussian_noise_distance(C.byref(d), 0.0, 0.02, 0.001))
        rgl.set_noise_seed(a, seed)
        rgl.set_noise_seed(d, seed + 1)
        rgl.chain(last, a, d)
        last = d
    if vehicle is not None:
        t = rgl.node()
        rgl.points_transform(t, vehicle)
        rgl.chain(last, t)
        last = t
    compact, out = rgl.node(), rgl.node()
    rgl.points_compact_by_field(compact)
    if case.get("format"):
        rgl.points_format(out, FORMATS[case["format"]])
    else:
        rgl.points_yield(out, [XYZ, DIST, ENT])
    rgl.chain(last, compact, out)
    return out


def _reader(case, out, beams):
    capacity = beams * RETURNS[case.get("mode", "first")]
    if case.get("format"):
        size = sum(rgl.FIELD_SIZE[f] for f in FORMATS[case["format"]])
        return Reader(out, capacity, [rgl.RGL_FIELD_DYNAMIC_FORMAT], size)
    return Reader(out, capacity, [XYZ, DIST, ENT])


def _mats(poses):
    """3x4 poses as one array the calls point into, and the pointer of each."""
    a = np.ascontiguousarray(np.stack(poses), dtype=np.float32)
    return a, [C.c_void_p(a[i].ctypes.data) for i in range(len(poses))]


def _reposes(world, case, rng):
    """For each of POSES frames the entities that move and their new poses."""
    moving = scenes.Scene(world.meshes, list(world.entities), world.heightfield)
    return [scenes.repose(moving, case["share"], rng) for _ in range(POSES)] if "share" in case else []


def _spawn(st, world):
    st.scene = rgl.scene_create()
    st.meshes, st.entities = rgl.spawn_scene_in(st.scene, world)


def _hold_reposes(st, frames):
    """The frames' new poses as calls: (entity, pointer of its 3x4 pose) pairs."""
    st.moves, st.move_mats = [], []
    for moves in frames:
        a, ptrs = _mats([tf for _, tf in moves]) if moves else (None, [])
        st.move_mats.append(a)
        st.moves.append([(st.entities[i], p) for (i, _), p in zip(moves, ptrs)])


def _inputs(case, seed):
    """Generator, world, sensor poses, moves: the same numbers for prepare() and exact()."""
    rng = np.random.default_rng([seed, 77])
    world = _world(case, seed)
    poses = _sensor_poses(world, rng, POSES)
    return rng, world, poses, _reposes(world, case, rng)


def prepare(case, seed):
    lib = rgl.lib()
    rgl.check(lib.rgl_configure_logging(rgl.RGL_LOG_LEVEL_OFF, None, False))
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(st):
    out = globals()["_run_" + st.kind](st)
    st.k += 1
    return out


# ---------------------------------------------------------------- scan, moving


def _prepare_scan(case, seed):
    st = State(case["kind"])
    rng, world, poses, frames = _inputs(case, seed)
    _spawn(st, world)
    for i, e in enumerate(st.entities):
        rgl.check(rgl.lib().rgl_entity_set_laser_retro(e, 0.25 * (i % 4)))
    st.pose_mats, st.poses = _mats(poses)
    _hold_reposes(st, frames)
    rays = scenes.lidar_rays(case["channels"], case["azimuths"])
    n = _trace_nodes(case, st.scene, rays, st.pose_mats[0], case["channels"] if case["format"] == "ircaedt" else 0)
    vehicle = scenes.trs(rng.uniform(-50, 50, 3), rng.uniform(-np.pi, np.pi, 3)) if case["noise"] else None
    out = _point_nodes(case, n, seed, vehicle)
    st.graphs, st.start, st.pose_node = [n["rays"]], n["rays"], n["pose"]
    st.read = _reader(case, out, rays.shape[0])
    return st


def _run_scan(st):
    lib = rgl.lib()
    rgl.check(lib.rgl_node_rays_transform(C.byref(st.pose_node), st.poses[st.k % POSES]))
    rgl.check(lib.rgl_graph_run(st.start))
    return st.read()


_prepare_moving = _prepare_scan


def _run_moving(st):
    lib = rgl.lib()
    for e, p in st.moves[st.k % POSES]:
        rgl.check(lib.rgl_entity_set_transform(e, p))
    return _run_scan(st)


# ---------------------------------------------------------------- animated, load


def _surface(case, seed):
    """A tile, POSES deformations of it and the sensor's poses above it."""
    rng = np.random.default_rng([seed, 78])
    tile = _tile(case["cells"], rng)
    shapes = []
    for k in range(POSES):
        v = tile.vertices.copy()
        v[:, 2] += (0.5 * np.sin(0.2 * v[:, 0] + k) * np.cos(0.15 * v[:, 1] - 0.7 * k)).astype(np.float32)
        shapes.append(v)
    poses = [scenes.trs((rng.uniform(-20, 20), rng.uniform(-20, 20), rng.uniform(5.0, 9.0)), (0, 0, rng.uniform(-3, 3))) for _ in range(POSES)]
    return tile, shapes, poses


def _prepare_animated(case, seed):
    st = State(case["kind"])
    tile, shapes, poses = _surface(case, seed)
    st.scene = rgl.scene_create()
    st.meshes = [rgl.mesh_create(tile.vertices, tile.indices)]
    st.entities = [rgl.entity_create_in(st.scene, st.meshes[0])]
    rgl.entity_set_transform(st.entities[0], scenes.translation(0, 0, 0))
    st.shapes = [torch.from_numpy(s).pin_memory() for s in shapes]
    st.vertices = tile.vertices.shape[0]
    st.pose_mats, st.poses = _mats(poses)
    rays = scenes.lidar_rays(case["channels"], case["azimuths"])
    n = _trace_nodes(case, st.scene, rays, poses[0])
    out = _point_nodes(case, n, seed)
    st.graphs, st.start, st.pose_node = [n["rays"]], n["rays"], n["pose"]
    st.read = _reader(case, out, rays.shape[0])
    return st


def _run_animated(st):
    rgl.check(rgl.lib().rgl_entity_apply_external_animation(st.entities[0], C.c_void_p(st.shapes[st.k % POSES].data_ptr()), st.vertices))
    return _run_scan(st)


def _prepare_load(case, seed):
    st = State(case["kind"])
    st.tile, shapes, poses = _surface(case, seed)
    st.shapes = [np.ascontiguousarray(s) for s in shapes]
    st.scene = rgl.scene_create()
    st.pose_mats, st.poses = _mats(poses)
    rays = scenes.lidar_rays(case["channels"], case["azimuths"])
    n = _trace_nodes(case, st.scene, rays, poses[0])
    out = _point_nodes(case, n, seed)
    st.graphs, st.start, st.pose_node = [n["rays"]], n["rays"], n["pose"]
    st.read = _reader(case, out, rays.shape[0])
    return st


def _run_load(st):
    mesh = rgl.mesh_create(st.shapes[st.k % POSES], st.tile.indices)
    entity = rgl.entity_create_in(st.scene, mesh)
    out = _run_scan(st)
    rgl.check(rgl.lib().rgl_entity_destroy(entity))
    rgl.check(rgl.lib().rgl_mesh_destroy(mesh))
    return out


# ---------------------------------------------------------------- fusion, batch


def _prepare_fusion(case, seed):
    st = State(case["kind"])
    rng, world, poses, _ = _inputs(case, seed)
    _spawn(st, world)
    st.pose_mats, st.poses = _mats([scenes.trs((1.5 * math.cos(a), 1.5 * math.sin(a), 0.0), (0.0, 0.0, a)) for a in
                                    (2 * math.pi * i / case["sensors"] for i in range(case["sensors"]))])
    # each sensor's mount on the vehicle, moved with the vehicle: one world pose per (frame, sensor)
    st.world_mats, st.world_ptrs = [], []
    for p in poses:
        four = np.vstack([p, [0, 0, 0, 1]]).astype(np.float64)
        a, ptrs = _mats([(four @ np.vstack([m, [0, 0, 0, 1]]).astype(np.float64))[:3].astype(np.float32) for m in st.pose_mats])
        st.world_mats.append(a)
        st.world_ptrs.append(ptrs)
    rays = scenes.lidar_rays(case["channels"], case["azimuths"])
    merge, out = rgl.node(), rgl.node()
    rgl.points_spatial_merge(merge, [XYZ, DIST, ENT])
    rgl.points_format(out, FORMATS["xyzde"])
    rgl.chain(merge, out)
    st.pose_nodes = []
    for i in range(case["sensors"]):
        n = _trace_nodes(case, st.scene, rays, st.world_mats[0][i])
        compact = rgl.node()
        rgl.points_compact_by_field(compact)
        rgl.chain(n["trace"], compact, merge)
        st.pose_nodes.append(n["pose"])
        st.start = n["rays"]
    st.graphs = [st.start]
    st.read = Reader(out, rays.shape[0] * case["sensors"], [rgl.RGL_FIELD_DYNAMIC_FORMAT], 20)
    return st


def _run_fusion(st):
    lib = rgl.lib()
    for n, p in zip(st.pose_nodes, st.world_ptrs[st.k % POSES]):
        rgl.check(lib.rgl_node_rays_transform(C.byref(n), p))
    rgl.check(lib.rgl_graph_run(st.start))
    return st.read()


def _prepare_batch(case, seed):
    st = State(case["kind"])
    world = _world(case, seed)
    _spawn(st, world)
    rng = np.random.default_rng([seed, 79])
    poses = [s.pose for s in scenes.sensor_rig(world, case["sensors"], seed=seed)]
    st.readers, nodes = [], []
    for i, pose in enumerate(poses):
        rays = scenes.Sensor(scenes.SENSOR_PATTERNS[i % len(scenes.SENSOR_PATTERNS)], pose).rays()
        n = _trace_nodes(case, st.scene, rays, pose)
        out = _point_nodes(case, n, seed + i)
        nodes.append(n["rays"])
        st.readers.append(_reader(case, out, rays.shape[0]))
    st.graphs = nodes
    st.batch = rgl.batch_create(nodes)
    _hold_reposes(st, _reposes(world, case, rng))
    return st


def _run_batch(st):
    lib = rgl.lib()
    for e, p in st.moves[st.k % POSES]:
        rgl.check(lib.rgl_entity_set_transform(e, p))
    rgl.check(lib.rgl_gb300_batch_run(st.batch))
    got = [r() for r in st.readers]
    return [buffers for buffers, _ in got], np.asarray([count for _, count in got])


# ---------------------------------------------------------------- serve


def _prepare_serve(case, seed):
    st = State(case["kind"])
    rng = np.random.default_rng([seed, 80])
    world = _world(case, seed)
    _spawn(st, world)
    st.server = rgl.Server(1 << 31)
    patterns = []
    for n in np.geomspace(case["smallest"], case["largest"], case["patterns"]):
        channels = 16 if n < 40_000 else 32 if n < 100_000 else 64
        azimuths = max(1, int(round(n / channels)))
        patterns.append((st.server.add_pattern(scenes.lidar_rays(channels, azimuths)), channels * azimuths))
    extent, st.requests = _extent(world), []
    for i in range(case["requests"]):
        p, beams = patterns[i % len(patterns)]
        x, y = rng.uniform(-0.4 * extent, 0.4 * extent, 2)
        pose = scenes.trs((x, y, world.ground_height(x, y) + rng.uniform(1.0, 3.0)), (0.0, 0.0, rng.uniform(-np.pi, np.pi)))
        st.requests.append((p, pose, beams))
    total = sum(b for _, _, b in st.requests)
    st.out = [(f, _pinned(total, w, t)) for f, w, t in ((XYZ, 3, torch.float32), (DIST, 1, torch.float32), (ENT, 1, torch.int32))]
    return st


def _run_serve(st):
    lib, h = rgl.lib(), st.server.h
    ids = [st.server.submit(st.scene, p, pose, rgl.RGL_RETURN_FIRST, *RANGE) for p, pose, _ in st.requests]
    cnt, sz, at = C.c_int32(), C.c_int32(), 0
    counts = []
    for r in ids:
        st.server.wait(r)
        for f, buf in st.out:
            rgl.check(lib.rgl_gb300_server_get_result_size(h, r, f, C.byref(cnt), C.byref(sz)))
            rgl.check(lib.rgl_gb300_server_get_result_data(h, r, f, C.c_void_p(buf[at:].data_ptr())))
        st.server.release(r)
        counts.append(cnt.value)
        at += cnt.value
    st.server.take_completed()
    return [buf for _, buf in st.out], np.asarray(counts)


# ---------------------------------------------------------------- work, exact


def _beams(case):
    if case["kind"] == "serve":
        return int(case["requests"] * math.sqrt(case["smallest"] * case["largest"]))
    if case["kind"] == "batch":
        return case["sensors"] * 104_000  # the mean of the rig's patterns
    return case["channels"] * case["azimuths"] * case.get("sensors", 1)


def work(case):
    """Bytes: each ray pose once, each point of the output once, the scene's vertices and indices once (an animated or
    loaded mesh is written once more, as given). Flops: per traced ray the transform of its pose and one ray/triangle
    test, what a ray cannot do without."""
    beams = _beams(case)
    samples = 1 + case.get("layers", 0) * case.get("vertices", 0)
    points = beams * RETURNS[case.get("mode", "first")]
    per_point = sum(rgl.FIELD_SIZE[f] for f in FORMATS[case.get("format") or "xyzde"])
    if case["kind"] in ("animated", "load"):
        triangles = 2 * case["cells"] ** 2
        scene = 2 * (12 * triangles + 6 * triangles)
    elif case.get("world") == "plain":
        scene = 18 * 20_768
    else:
        scene = 18 * (2 * case["cells"] ** 2 + 5120 * min(8, case["instances"]))
    return {"bytes": float(48 * beams + per_point * points + scene), "flops": float(beams * samples * (72 + 60))}


def _world_triangles(world):
    out, ids = [], []
    for e in world.entities:
        m = world.meshes[e.mesh]
        v = m.vertices.astype(np.float64) @ e.transform[:, :3].astype(np.float64).T + e.transform[:, 3].astype(np.float64)
        out.append(v[m.indices])
        ids.append(np.full(len(m.indices), e.entity_id, dtype=np.int32))
    return np.concatenate(out), np.concatenate(ids)


def _closest(tri, org, direction):
    """Distance and index of each unit ray's closest hit in 64 bits, tested against every triangle of the clusters (128
    neighbouring triangles) whose bounding spheres the ray meets. inf and -1 without a hit."""
    dev, per = "cuda", 128
    mid = tri.mean(1)
    order = np.lexsort((mid[:, 0], np.floor(mid[:, 1] / 10.0)))
    tri = tri[order]
    t = torch.from_numpy(tri).to(dev)
    pad = -len(tri) % per
    t = torch.cat([t, t[-1:].expand(pad, 3, 3)]) if pad else t
    t = t.reshape(-1, per, 3, 3)
    centre = (t.amin((1, 2)) + t.amax((1, 2))) / 2
    radius = (t - centre[:, None, None]).norm(dim=-1).amax((1, 2)) * (1 + 1e-9) + 1e-9
    o, d = torch.from_numpy(org).to(dev), torch.from_numpy(direction).to(dev)
    best = torch.full((len(o),), math.inf, dtype=torch.float64, device=dev)
    prim = torch.full((len(o),), -1, dtype=torch.int64, device=dev)
    a, e1, e2 = t[:, :, 0], t[:, :, 1] - t[:, :, 0], t[:, :, 2] - t[:, :, 0]
    step = max(1, 40_000_000 // len(t))
    for at in range(0, len(o), step):
        oo, dd = o[at:at + step], d[at:at + step]
        along = dd @ centre.T - (oo * dd).sum(1, keepdim=True)
        off2 = (centre * centre).sum(1) - 2 * oo @ centre.T + (oo * oo).sum(1, keepdim=True) - along * along
        ray, cluster = ((off2 <= radius ** 2 + 1e-6) & (along >= -radius)).nonzero(as_tuple=True)
        for k in range(0, len(ray), 60_000):
            r, c = ray[k:k + 60_000], cluster[k:k + 60_000]
            ro, rd = oo[r][:, None], dd[r][:, None].expand(-1, per, -1)
            p = torch.linalg.cross(rd, e2[c])
            det = (e1[c] * p).sum(-1)
            inv = 1.0 / torch.where(det == 0, torch.full_like(det, math.inf), det)
            s = ro - a[c]
            u = (s * p).sum(-1) * inv
            q = torch.linalg.cross(s, e1[c])
            v = (rd * q).sum(-1) * inv
            dist = (e2[c] * q).sum(-1) * inv
            dist = torch.where((det != 0) & (u >= 0) & (v >= 0) & (u + v <= 1) & (dist > 0), dist, torch.full_like(dist, math.inf))
            dmin, which = dist.min(1)
            r = r + at
            new = best.scatter_reduce(0, r, dmin, "amin")
            wins = (dmin == new[r]) & (dmin < best[r])
            prim[r[wins]] = c[wins] * per + which[wins]
            best = new
    prim = prim.cpu().numpy()
    return best.cpu().numpy(), np.where(prim >= 0, order[np.clip(prim, 0, len(order) - 1)], -1)


def exact(case, seed):
    """XYZ, distance and entity id of the first pass's hits in 64 bits, for the cases that read them unformatted with one
    ray a beam and no noise (the noise's random stream is the framework's own)."""
    if case.get("layers") or case.get("noise") or case.get("format") or case["kind"] in ("fusion", "batch", "serve"):
        return None
    if case["kind"] in ("animated", "load"):
        tile, shapes, poses = _surface(case, seed)
        tri, ids = shapes[0].astype(np.float64)[tile.indices], None
    else:
        _, world, poses, frames = _inputs(case, seed)
        for i, tf in frames[0] if frames else []:
            e = world.entities[i]
            world.entities[i] = scenes.Entity(e.mesh, tf, e.entity_id)
        tri, ids = _world_triangles(world)
    if len(tri) * case["channels"] * case["azimuths"] > 1.5e11:
        return None
    rays = scenes.lidar_rays(case["channels"], case["azimuths"]).astype(np.float64)
    pose = poses[0].astype(np.float64)
    direction = rays[:, :, 2] @ pose[:, :3].T
    direction /= np.linalg.norm(direction, axis=1, keepdims=True)
    org = np.broadcast_to(pose[:, 3], direction.shape).copy()
    dist, prim = _closest(tri, org, direction)
    hit = (dist >= RANGE[0]) & (dist <= RANGE[1])
    entity = ids[prim[hit]] if ids is not None else np.full(int(hit.sum()), rgl.RGL_DEFAULT_ENTITY_ID, dtype=np.int32)
    first = [org[hit] + direction[hit] * dist[hit, None], dist[hit], entity]
    whole = [np.zeros((len(org),) + v.shape[1:], dtype=v.dtype) for v in first]
    for w, v in zip(whole, first):
        w[: len(v)] = v
    return whole, int(hit.sum())
