"""How a traversal launch is cut into tasks (csrc/beam_tasks.hpp): patterns of which two or more beams fit a
warp's 32 lanes take as few rounds of resident warps as beams side by side allow, however large the launch; a
task's samples stay within the pool, and the division by a pattern's samples is exact for all of them."""
import ctypes as C
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
RESIDENT = 152 * 16


@pytest.fixture(scope="module")
def tasks(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("tasks") / "libtasks_harness.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I", os.path.join(ROOT, "robotecgpulidar_gb300", "csrc"), "-o", out,
                    os.path.join(ROOT, "tests", "cpp", "tasks_harness.cpp")], check=True)
    lib = C.CDLL(out)
    lib.beams_per_task.argtypes = [C.c_int, C.c_int, C.c_int64, C.c_int64, C.c_int]
    lib.sample_factor.restype = C.c_uint32
    return lib


@pytest.mark.parametrize("samples", range(1, 17))
def test_beams_share_a_warps_lanes(tasks, samples):
    most = 32 // samples
    for beams in [1, 31, 2432, 2433, 5000, 10000, 20000, 40000, 80000, 262144, 4 << 20]:
        per = tasks.beams_per_task(samples, beams, beams, RESIDENT, 0)
        assert 1 <= per <= most
        rounds, fewest = -(-beams // (per * RESIDENT)), -(-beams // (most * RESIDENT))
        assert rounds <= max(2, fewest)


@pytest.mark.parametrize("samples", range(1, 65))
def test_samples_of_a_task(tasks, samples):
    for beams in [1, 5000, 40000, 1 << 20, 1 << 30]:
        for cells in (0, 1, 700):
            per = tasks.beams_per_task(samples, min(beams, 1 << 30), beams, RESIDENT, cells)
            if samples <= tasks.lane_group_samples():
                assert 1 <= per and per * samples <= 32
            else:
                assert 1 <= per <= 32 and per * samples <= tasks.pool_samples()
    factor = tasks.sample_factor(samples)
    for i in range(tasks.pool_samples()):
        assert (i * factor) >> 16 == i // samples
