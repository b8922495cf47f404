"""Square roots, quotients, sums and conversions on the integer pipes (fp64_int.cuh):
on the host against the processor's FP64, and on the device, with the logarithm
and the arctangent that use them, against their FP64 forms.  Bit for bit."""
import os
import shutil
import subprocess

import pytest

from jif3d_gb300 import build as B

HERE = os.path.dirname(os.path.abspath(__file__))


def _run(cmd, names):
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([cmd[-1]], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    rows = [line.split() for line in out.stdout.strip().splitlines()]
    assert [row[0] for row in rows] == names
    for name, bad, tested in rows:
        assert int(tested) > 1 << 24 and int(bad) == 0, (name, bad, tested)


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_host_bit_exact(tmp_path):
    _run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", B.CSRC,
          os.path.join(HERE, "cpp", "fp64_int_check.cpp"), "-o", str(tmp_path / "check")],
         ["sqrt", "quotient", "convert", "add"])


@pytest.mark.gpu
def test_device_bit_exact(tmp_path):
    _run([B.nvcc(), "-O3", "-std=c++17", B.ARCH, "-I", B.CSRC,
          os.path.join(HERE, "fp64_int_check.cu"), "-o", str(tmp_path / "check")],
         ["sqrt", "log", "atan2", "add"])
