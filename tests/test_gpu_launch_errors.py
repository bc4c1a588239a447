"""A refused launch is reported by the call that made it and by no other."""
import os
import subprocess

import pytest

from klft_b200.build import ARCH, CSRC, NVCC, ROOT

pytestmark = pytest.mark.gpu


def test_refused_launch_is_reported_once(tmp_path):
    exe = str(tmp_path / "refused_launch")
    subprocess.run([NVCC] + ARCH + ["-std=c++17", "-I" + CSRC, os.path.join(ROOT, "tests", "cxx", "refused_launch.cu"),
                    "-o", exe], check=True, timeout=300)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
