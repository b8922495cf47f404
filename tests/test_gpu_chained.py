"""Chained launches (csrc/chained.cuh) on their own."""
import os
import subprocess

import pytest

from jif3d_gb300 import build as B

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.gpu
def test_refused_launch_leaves_no_error(tmp_path):
    exe = str(tmp_path / "check")
    r = subprocess.run([B.nvcc(), "-O3", "-std=c++17", B.ARCH, "-I", B.CSRC,
                        os.path.join(HERE, "chained_check.cu"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.stdout.strip() == "ok", out.stdout
