"""The slab test's inverse directions (csrc/trace_core.hpp safeInv) are the same numbers on the device as on
the host, where the traversal's completeness is tested, and correctly rounded."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("inverse") / "libinverse_harness.so")
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    subprocess.run([nvcc, "-std=c++17", "-O3", "-gencode", "arch=compute_103a,code=sm_103a", "-shared", "-Xcompiler", "-fPIC,-ffp-contract=off",
                    "-I", os.path.join(ROOT, "robotecgpulidar_gb300", "csrc"), "-o", out,
                    os.path.join(ROOT, "tests", "cpp", "inverse_harness.cu")], check=True)
    return C.CDLL(out)


def test_device_inverse_equals_the_hosts(harness):
    rng = np.random.default_rng(11)
    d = np.concatenate([
        rng.uniform(-1, 1, 1 << 20),  # components of unit directions
        rng.uniform(-1, 1, 1 << 18) * 10.0 ** rng.uniform(-35, 35, 1 << 18),  # scaled instances
        np.array([0.0, -0.0, 1e-30, -1e-30, 9.9e-31, 1e-40, -1e-40, 1.0, -1.0, 2.0 ** -99, 3.4e38, -3.4e38]),
    ]).astype(np.float32)
    host, device = np.empty_like(d), np.empty_like(d)
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    assert harness.inverses(p(d), p(host), p(device), C.c_int(len(d))) == 0
    assert np.array_equal(host.view(np.uint32), device.view(np.uint32))
    clamped = np.where(np.abs(d) < np.float32(1e-30), np.where(d < 0, np.float32(-1e-30), np.float32(1e-30)), d)
    assert np.array_equal(host, (1.0 / clamped.astype(np.float64)).astype(np.float32))
