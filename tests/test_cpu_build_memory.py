"""Device memory that is kept for later builds (csrc/build_memory.cpp) on a fake CUDA runtime: what the pools
keep serves any other allocation once memory is out, a failed allocation leaves nothing half done, and
freed storage waits for its readers' events and never for the device."""
import ctypes as C
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "robotecgpulidar_gb300", "csrc")


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("memory") / "libmemory_harness.so")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    # -Bsymbolic: the fakes win over a CUDA runtime that the process has loaded
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I", CSRC, "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(cuda, "include"), "-o", out, os.path.join(ROOT, "tests", "cpp", "memory_harness.cpp"),
                    os.path.join(CSRC, "build_memory.cpp"), os.path.join(CSRC, "common.cpp")], check=True)
    return C.CDLL(out)


def test_kept_memory_serves_other_allocations(harness):
    assert harness.kept_memory_serves_other_allocations() == 0


@pytest.mark.parametrize("instances", [1000, 2048, 100_000])
@pytest.mark.parametrize("fitting", [0, 1, 2, 3, 4])
def test_a_failed_tlas_allocation_starts_over(harness, instances, fitting):
    assert harness.a_failed_tlas_allocation_starts_over(instances, fitting) == 0


def test_frees_wait_for_the_readers_alone(harness):
    assert harness.frees_wait_for_the_readers_alone() == 0


def test_every_large_allocation_tries_again_without_what_is_kept():
    bare = []
    for name in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, name)) as f:
            for number, line in enumerate(f, 1):
                code = line.split("//")[0]
                if re.search(r"\b(cudaMalloc|cudaMallocAsync|cudaMallocFromPoolAsync|cudaMallocArray|cudaGraphInstantiate\w*)\(", code) and \
                        "trimAndRetry" not in code:
                    bare.append(f"{name}:{number}: {code.strip()}")
    assert not bare, bare
