"""Waits inside kernels have a limit. When one runs out, a brute-force block searches its queries without the pipeline and
leaves nothing of it behind; a tree build reports that it did not finish (tests/cpp/*_waits.cu, over the library's
internal entry points)."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def compile_cu(tmp_path, name, *extra):
    from libnabo_gb300 import build
    lib = os.path.join(ROOT, "libnabo_gb300", "lib")
    exe = str(tmp_path / name)
    subprocess.run([build.nvcc(), *build.ARCH, "-O1", "-std=c++17", "-Xcompiler", "-ffp-contract=off",
                    "-I", os.path.join(ROOT, "include"), "-I", build.CSRC, os.path.join(ROOT, "tests", "cpp", f"{name}.cu"),
                    "-L", lib, "-lnabo_gb300", "-Xlinker", f"-rpath={lib}", "-Xlinker", "--export-dynamic", "-ldl",
                    *extra, "-o", exe], check=True, capture_output=True, text=True)
    return exe


def test_brute_force_waits_that_run_out(tmp_path):
    r = subprocess.run([compile_cu(tmp_path, "brute_force_waits")], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.count("ok ") == 5, r.stdout + r.stderr


def test_build_waits_that_run_out(tmp_path):
    r = subprocess.run([compile_cu(tmp_path, "build_waits")], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.count("ok ") == 3, r.stdout + r.stderr
