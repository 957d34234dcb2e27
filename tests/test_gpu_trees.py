"""The device's trees are the host's, node for node: frames, slots, quantised boxes and leaves, read back from
the device and compared as bytes (tests/cpp/tree_harness.cpp). Scans alone do not tell: a hit does not depend
on the tree.

Mesh sizes sit around a warp's range (32), a warp's split (256), the largest range of one block (1,024), the
chunks of the level loop (512) and the pyramid's tiles (512); instance counts around the one-block TLAS
(2,048). Shapes: a soup, a terrain (whose triangles share planes), clusters (a level each), and triangles that
all lie in one place (ranges split in the middle).
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from robotecgpulidar_gb300 import build

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def trees(tmp_path_factory):
    build.build()
    out = str(tmp_path_factory.mktemp("trees") / "libtree_harness.so")
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    objs = sorted(os.path.join(build.OUT_DIR, f) for f in os.listdir(build.OUT_DIR) if f.endswith(".o"))
    subprocess.run([nvcc, "-std=c++17", "-O2", *build.ARCH, "-shared", "-Xcompiler", "-fPIC,-ffp-contract=off", "-Xlinker", "-Bsymbolic", "-I",
                    build.INCLUDE, "-I", build.CSRC, "-o", out, os.path.join(ROOT, "tests", "cpp", "tree_harness.cpp"), *objs, "-lpthread"],
                   check=True)
    lib = C.CDLL(out)
    for f in ("device_mesh_tree", "host_mesh_tree", "device_instance_tree", "host_instance_tree"):
        getattr(lib, f).restype = C.c_int64
    lib.tree_failure.restype = C.c_char_p
    return lib


def tree(lib, name, *args):
    n = getattr(lib, name)(*[a.ctypes.data_as(C.c_void_p) if isinstance(a, np.ndarray) else C.c_int(a) for a in args])
    assert n > 0, lib.tree_failure()
    out = np.empty(n, np.uint8)
    lib.tree_bytes(out.ctypes.data_as(C.c_void_p))
    return out.tobytes()


def mesh(shape, triangles):
    rng = np.random.default_rng(triangles)
    if shape == "terrain":
        side = int(np.ceil(np.sqrt(triangles / 2)))
        g = np.linspace(-50, 50, side + 1)
        x, y = np.meshgrid(g, g, indexing="ij")
        v = np.stack([x.ravel(), y.ravel(), 3 * np.sin(0.3 * x.ravel()) * np.cos(0.2 * y.ravel())], 1)
        a = (np.arange(side)[:, None] * (side + 1) + np.arange(side)).reshape(-1)
        idx = np.stack([a, a + 1, a + side + 1, a + 1, a + side + 2, a + side + 1], 1).reshape(-1, 3)[:triangles]
        return np.ascontiguousarray(v, np.float32), np.ascontiguousarray(idx, np.int32)
    c = rng.uniform(-30, 30, (triangles, 3))
    if shape == "clusters":
        c = (4000.0 / 64.0 ** rng.integers(0, 6, triangles))[:, None] * rng.uniform(0.95, 1.05, (triangles, 3))
    d = rng.uniform(-1, 1, (triangles, 3, 3))
    if shape == "one place":
        c, d = np.full((triangles, 3), 2.0), np.broadcast_to(d[:1], d.shape)
    v = (c[:, None, :] + d).astype(np.float32).reshape(-1, 3)
    return np.ascontiguousarray(v), np.arange(3 * triangles, dtype=np.int32).reshape(-1, 3)


SIZES = [1, 2, 3, 31, 32, 33, 64, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025, 1026, 1535, 1537, 2049, 4095, 4097, 33282, 131072]


@pytest.mark.parametrize("shape", ["soup", "terrain", "clusters", "one place"])
@pytest.mark.parametrize("triangles", SIZES)
@pytest.mark.parametrize("sah", [1, 0])
def test_mesh_tree(trees, shape, triangles, sah):
    v, idx = mesh(shape, triangles)
    args = (v, len(v), idx, len(idx), sah)
    assert tree(trees, "device_mesh_tree", *args) == tree(trees, "host_mesh_tree", *args)


@pytest.mark.parametrize("shape", ["spread", "row", "one place"])
@pytest.mark.parametrize("instances", [1, 2, 7, 8, 9, 31, 33, 94, 250, 257, 1024, 2047, 2048, 2049, 2100, 5000])
def test_instance_tree(trees, shape, instances):
    rng = np.random.default_rng(instances)
    c = rng.uniform(-200, 200, (instances, 3))
    if shape == "row":
        c[:, 1:] = 5.0
    if shape == "one place":
        c[:] = 7.0
    r = rng.uniform(0.5, 5.0, (instances, 3)) if shape != "one place" else np.full((instances, 3), 2.0)
    boxes = np.ascontiguousarray(np.concatenate([c - r, c + r], 1), np.float32)
    assert tree(trees, "device_instance_tree", boxes, instances) == tree(trees, "host_instance_tree", boxes, instances)
