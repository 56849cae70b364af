"""Both variants of the block step (16 and 8 rows per pass), called directly, so
that each of their kernels runs whatever the autotuner would choose: see
step_variants_check.cpp."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_step_variants(tmp_path):
    from gpb import build
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    lib = build.build()
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc())))
    exe = str(tmp_path / "check")
    libdir = os.path.join(cuda, "lib64")
    subprocess.run([cxx, "-O2", "-std=c++17", "-I" + os.path.join(cuda, "include"), "-I" + os.path.join(ROOT, "include"),
                    "-I" + build.CSRC, os.path.join(ROOT, "tests", "step_variants_check.cpp"), "-o", exe, lib,
                    "-L" + libdir, "-lcudart", "-Wl,-rpath," + os.path.dirname(lib), "-Wl,-rpath," + libdir], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and "ok" in out.stdout, out.stdout + out.stderr
