"""The node kernels component by component, and the offsets that their fixed-point
terms take: what a norm over a whole joint vector, or a count with room to spare,
would not show (the g_z data are 36 to 160 times the tensor's in test_node_fixed's
shapes)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from helpers import relerr
from jif3d_gb300 import build as B, workloads as W
from test_node_fixed import GRAV, SHAPES, _rows, _survey

HERE = os.path.dirname(os.path.abspath(__file__))


def _lines(tmp_path, name):
    cxx = shutil.which("g++")
    assert cxx, "a host compiler is needed"
    exe = str(tmp_path / name)
    r = subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", B.CSRC,
                        os.path.join(HERE, "cpp", name + ".cpp"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0
    return r.stdout.splitlines()


def test_no_offset_of_the_sets_is_left_out(tmp_path):
    rows = [line.split() for line in _lines(tmp_path, "node_fixed_check")]
    assert len(rows) == 24
    for name, which, n, left, *_ in rows:
        assert int(n) == 100000 and int(left) == 0, (name, which, left)


def test_offsets_taken_and_left(tmp_path):
    assert _lines(tmp_path, "node_left_check") == ["taken"] * 11 + ["left"] * 15


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("aligned", [False, True])
def test_joint_components_at_tile_edges(ctx, shape, aligned):
    """1e-10, the parity bound of the FP64 path, for every row of the joint kind:
    its data over the stations, and the gradient of a misfit on that row alone."""
    s = _survey(W.JOINT, *shape, aligned)
    W.setup_context(ctx, s)
    n = s.stations.shape[0]
    J = _rows(s)
    d, ref = ctx.forward(s.model).reshape(n, 10), (J @ s.model).reshape(n, 10)
    w = np.random.default_rng(3).normal(size=n)
    for row in range(10):
        assert relerr(d[:, row], ref[:, row]) <= 1e-10, row
        misfit = np.zeros((n, 10))
        misfit[:, row] = w
        g = ctx.lqderivative(s.model, misfit.ravel())
        assert relerr(g, 2.0 * (w @ J[row::10])) <= 1e-10, row


@pytest.mark.gpu
@pytest.mark.parametrize("kind", [W.SCALAR, W.TENSOR, W.JOINT])
def test_far_offsets_within_the_terms_rounding(ctx, kind):
    """Offsets beyond 2^40 m: the box terms vanish against their nodes' rounding.  The
    data are no more than that: 2^-53 of the largest node term, for the term and for
    each of some 30 additions that a partial sum goes through, over all nodes."""
    s = _survey(kind, 6, 5, 4, 1, False)
    s.stations = np.array([[3e12, 0.0, -1.0]])
    W.setup_context(ctx, s)
    cells = np.pad(s.model.reshape(6, 5, 4), 1)
    weight = np.abs(np.diff(np.diff(np.diff(cells, axis=0), axis=1), axis=2)).sum()
    d = ctx.forward(s.model)
    assert np.all(np.isfinite(d))
    term = np.full(d.size, 30.0)  # ln(6e12) = 29.4; angles up to pi
    if kind != W.TENSOR:  # g_z: its own offsets times those
        term[0] = (3e12 + 500.0) * 30.0 + 500.0 * np.pi
    assert np.all(np.abs(d) <= GRAV * weight * term * 31 * 2.0 ** -53)
