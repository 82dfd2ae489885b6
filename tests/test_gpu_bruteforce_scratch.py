"""The brute force's scratch: without any, the results are the same; a captured search of many queries asks for none
(tests/cpp/brute_force_scratch.cu, whose scratch_alloc takes the place of the library's)."""
import subprocess

import pytest

from test_gpu_bounded_waits import compile_cu

pytestmark = pytest.mark.gpu


def test_scratch_refused_and_captured(tmp_path):
    r = subprocess.run([compile_cu(tmp_path, "brute_force_scratch")], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.count("ok ") == 6, r.stdout + r.stderr
