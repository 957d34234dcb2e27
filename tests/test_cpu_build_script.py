"""An edit to any included source makes the objects stale (robotecgpulidar_gb300/build.py): every file that a
translation unit includes by name is among the headers it watches."""
import os
import re

from robotecgpulidar_gb300 import build


def test_every_included_file_is_watched():
    watched = {os.path.realpath(p) for p in build._headers()}
    places = [build.CSRC, build.INCLUDE]
    missing = set()
    for name in os.listdir(build.CSRC):
        path = os.path.join(build.CSRC, name)
        if not os.path.isfile(path):
            continue
        with open(path) as f:
            for inc in re.findall(r'#include\s+["<]([^">]+)[">]', f.read()):
                found = [os.path.realpath(os.path.join(d, inc)) for d in places if os.path.isfile(os.path.join(d, inc))]
                missing |= {p for p in found if p not in watched}
    assert not missing
    assert any(p.endswith(".cuh") for p in watched)


def test_a_changed_kernel_header_makes_an_object_stale(tmp_path):
    obj, src = tmp_path / "x.o", tmp_path / "x.cu"
    src.write_text("")
    obj.write_text("")
    headers = build._headers()
    newest = max(os.path.getmtime(p) for p in headers if p.endswith(".cuh"))
    os.utime(src, (newest - 20, newest - 20))
    os.utime(obj, (newest - 10, newest - 10))
    assert build._stale(str(obj), str(src), headers)
