"""The staged split search's table plans, host logic only: tests/cpp/stage_tables.cu is compiled with nvcc against the
in-tree library and run on the CPU."""
import os
import subprocess

from curfil_b200 import _build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_stage_tables_invariants(tmp_path):
    lib = _build.build()
    libdir = os.path.dirname(lib)
    exe = str(tmp_path / "stage_tables")
    cmd = [_build.NVCC] + _build.ARCH + ["-std=c++17", "-O1", "--expt-relaxed-constexpr", "-I",
                                         os.path.join(ROOT, "include"),
                                         os.path.join(ROOT, "tests", "cpp", "stage_tables.cu"), "-L", libdir,
                                         "-lcurfil_b200", "-Xlinker", "-rpath", "-Xlinker", libdir, "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    run = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0 and "\n0 failures" in "\n" + run.stdout, run.stdout + run.stderr
