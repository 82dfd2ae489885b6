"""A build on a stream that may use some of the device's SMs only: the launch of the top levels, whose blocks all have to be
resident, takes as many as the stream has room for, and their working lists leave shared memory when they are too long for it
(tests/cpp/build_in_part.cu)."""
import os
import subprocess

import pytest

from test_gpu_bounded_waits import compile_cu

pytestmark = pytest.mark.gpu


def test_green_context_stream(tmp_path):
    from libnabo_gb300 import build
    stubs = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "lib64", "stubs")
    r = subprocess.run([compile_cu(tmp_path, "build_in_part", "-L", stubs, "-lcuda")], capture_output=True, text=True,
                       timeout=300)
    if r.returncode == 77:
        pytest.skip("no green contexts here")
    assert r.returncode == 0 and r.stdout.count("ok ") == 5, r.stdout + r.stderr
