"""Host-side parts of the kernels' plans, by small programs against their headers."""

import os
import shutil
import subprocess

from conftest import ROOT


def test_hash_slots(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cuda_inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    exe = tmp_path / "hash_slot_check"
    build = subprocess.run(
        ["g++", "-std=c++17", "-O2", "-I", cuda_inc,
         "-I", os.path.join(ROOT, "mojo-libigl_b200", "csrc"),
         os.path.join(ROOT, "tests", "hash_slot_check.cpp"), "-o", str(exe)],
        capture_output=True, text=True, timeout=300)
    assert build.returncode == 0, build.stderr
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0, run.stdout + run.stderr
    assert run.stdout.startswith("ok")


def test_edge_adjoint_partials(tmp_path):
    from igl import _lib

    lib_path = _lib.build()
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cuda_inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    exe = tmp_path / "adjoint_plan_check"
    build = subprocess.run(
        ["g++", "-std=c++17", "-O1", "-I", cuda_inc,
         "-I", os.path.join(ROOT, "mojo-libigl_b200", "csrc"),
         os.path.join(ROOT, "tests", "adjoint_plan_check.cpp"), "-o", str(exe),
         "-L", os.path.dirname(lib_path), "-lwn_b200",
         "-Wl,-rpath," + os.path.dirname(lib_path)],
        capture_output=True, text=True, timeout=300)
    assert build.returncode == 0, build.stderr
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0, run.stdout + run.stderr
    assert run.stdout.startswith("ok")
