"""What libgpb.so launches, checked on the host: the library runs against a
stand-in for the CUDA runtime (fake_runtime/) that records launches."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _run(tmp_path, name, *args):
    from gpb import build
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    lib = build.build()
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")
    exe = str(tmp_path / name)
    subprocess.run([cxx, "-O1", "-std=c++17", "-pthread", "-rdynamic", "-I" + cuda, "-I" + os.path.join(ROOT, "include"),
                    "-I" + build.CSRC, os.path.join(ROOT, "tests", "fake_runtime", name + ".cpp"), "-o", exe, lib,
                    "-Wl,-rpath," + os.path.dirname(lib), "-Wl,--unresolved-symbols=ignore-in-shared-libs"], check=True)
    out = subprocess.run([exe, *args], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and "ok" in out.stdout, out.stdout + out.stderr


@pytest.mark.parametrize("args", [(), ("grants-fail-first",)])
def test_shared_memory_grants_per_device_and_thread(tmp_path, args):
    _run(tmp_path, "devices_check", *args)


def test_stitch_launches_in_proportion_to_its_boxes(tmp_path):
    _run(tmp_path, "stitch_check")


def test_ucm_launches_in_proportion_to_each_image(tmp_path):
    _run(tmp_path, "ucm_check")


def test_tables_that_do_not_fit_are_an_error(tmp_path):
    _run(tmp_path, "tables_check")
