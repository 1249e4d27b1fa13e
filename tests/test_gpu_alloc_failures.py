"""The staged split search when device memory runs out: tests/cpp/alloc_failures.cpp, linked with the library's objects
so that it can refuse cudaMalloc calls on the host. The call must give its splits with a smaller table or in one pass."""
import glob
import os
import subprocess

import pytest

from curfil_b200 import _build

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_split_search_with_refused_allocations(tmp_path):
    _build.build()
    exe = str(tmp_path / "alloc_failures")
    objects = sorted(glob.glob(os.path.join(_build.BUILD, "*.cu.o")))
    cmd = [_build.NVCC] + _build.ARCH + ["-std=c++17", "-O1", "-Xlinker", "--wrap=cudaMalloc", "-I",
                                         os.path.join(ROOT, "include"),
                                         os.path.join(ROOT, "tests", "cpp", "alloc_failures.cpp")] + objects + \
        ["-o", exe, "-lpthread", "-lz"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    run = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert run.returncode == 0, run.stdout + run.stderr
    assert "\n0 failures" in run.stdout, run.stdout
