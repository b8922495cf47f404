"""Precision of the fixed-point node terms beside FP64's own.

Angles, on the host: the error in units of the last place, separately for every
power of two of the angle (a small angle is a small difference of a box term's
corners, so it needs its leading bits).  FP64's atan2 of rounded products is the
measure: no root mean square and no largest error may be above its.
"""
import os
import shutil
import subprocess

from jif3d_gb300 import build as B

HERE = os.path.dirname(os.path.abspath(__file__))


def test_angles_no_worse_than_fp64(tmp_path):
    cxx = shutil.which("g++")
    assert cxx, "a host compiler is needed"
    exe = str(tmp_path / "node_angle_check")
    src = os.path.join(HERE, "cpp", "node_angle_check.cpp")
    r = subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", B.CSRC, src, "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0
    rows = [line.split() for line in r.stdout.splitlines()]
    seen = 0
    for comp, power, n, rms, rms64, top, top64 in rows:
        if int(n) < 1000:  # too few to know a root mean square
            continue
        seen += 1
        assert float(rms) <= float(rms64) and float(top) <= float(top64), (comp, power, rms, rms64,
                                                                          top, top64)
    assert seen >= 60
