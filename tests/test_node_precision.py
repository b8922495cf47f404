"""Precision of the fixed-point node terms beside FP64's own.

Angles, on the host: the error in units of the last place, separately for every
power of two of the angle (a small angle is a small difference of a box term's
corners, so it needs its leading bits).  FP64's atan2 of rounded products is the
measure: no root mean square and no largest error may be above its.

Data and gradients, on the GPU, each component on its own: g_z is some hundred times
the tensor in a joint vector, and the components lose different numbers of bits
where stations are far away or below the mesh.  Every component is compared with
sums in long double, and its error with that of the same node sums in FP64 (log,
atan2 and products of doubles, added up as the kernels do on a survey of this size:
the data level by level, the columns of a level by lanes and halves, the gradient in
station order).  As the terms round no more than those, over 48 stations or 512 cells, whose root mean square is
known to 15 %, the error stays within twice the FP64 sums' (and a last bit of the
largest value, where those happen to be exact).
"""
import os
import shutil
import subprocess

import numpy as np
import pytest

from jif3d_gb300 import build as B, workloads as W

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


GRAV = 6.67428e-11
N, SIZE = (8, 8, 8), (50.0, 50.0, 25.0)
# the tensor's components in its rows
ROWS = {"xx": 0, "xy": 1, "xz": 2, "yy": 4, "yz": 5, "zz": 8}


def _terms(st, T):
    """Node terms [station][x][y][z] in the type T; beyond double, log(d + r) of a
    negative d without cancellation."""
    d = [st[:, a].astype(T).reshape(-1, 1, 1, 1) -
         (np.arange(N[a] + 1) * T(SIZE[a])).reshape([1] + [-1 if b == a else 1 for b in range(3)])
         for a in range(3)]
    x, y, z = d
    xx, yy, zz = x * x, y * y, z * z
    r = np.sqrt(xx + yy + zz)

    def ln(u, rest):
        v = u + r
        if T is not np.float64:
            with np.errstate(divide="ignore", invalid="ignore"):
                v = np.where(u < 0, rest / (r - u), v)
        return np.log(np.maximum(v, T(2.0) ** -52))
    lx, ly = ln(x, yy + zz), ln(y, xx + zz)
    return {"gz": x * ly + y * lx + z * np.arctan2(z * r, x * y), "xx": np.arctan2(y * z, x * r),
            "yy": np.arctan2(x * z, y * r), "zz": np.arctan2(x * y, z * r),
            "xy": ln(z, xx + yy), "xz": ly, "yz": lx}


def _scale(c):
    return GRAV if c in ("xx", "yy", "zz") else -GRAV


def _differences(v, lead):
    """Differences along the last three axes: of a model padded with zeros (the
    data) or of node sums (the gradient)."""
    for a in (lead, lead + 1, lead + 2):
        v = np.diff(v, axis=a)
    return v


def _model_differences(model):
    """The nodes' differences of the model (summation by parts) as the kernels form
    them: the eight cells of a corner one after the other."""
    cells = np.pad(model.reshape(N), 1)
    rho = np.zeros([n + 1 for n in N])
    for q in range(8):
        a = (q >> 2 & 1, q >> 1 & 1, q & 1)
        cell = cells[tuple(slice(1 - b, n + 2 - b) for b, n in zip(a, N))]
        rho = rho - cell if sum(a) & 1 else rho + cell
    return rho


def _level_sums(v):
    """Sums of [station][x][y][z]: 32 lanes take the columns of a level in turn and
    are added up by halves, then level after level."""
    columns = v.reshape(v.shape[0], -1, v.shape[3])
    rows = -(-columns.shape[1] // 32)
    padded = np.zeros((v.shape[0], rows * 32, v.shape[3]))
    padded[:, :columns.shape[1]] = columns
    lanes = np.add.accumulate(padded.reshape(v.shape[0], rows, 32, -1), axis=1)[:, -1]
    while lanes.shape[1] > 1:
        half = lanes.shape[1] // 2
        lanes = lanes[:, :half] + lanes[:, half:]
    return np.add.accumulate(lanes[:, 0], axis=1)[:, -1]


def _stations(where, depth):
    rng = np.random.default_rng(12)
    st = rng.uniform(0, 1, (48, 3)) * np.array([N[0] * SIZE[0], N[1] * SIZE[1], N[2] * SIZE[2]])
    if where == "below":
        st[:, 2] = N[2] * SIZE[2] + depth
    elif where == "above":
        st[:, 2] = -depth
    elif where == "aside":
        st += [20 * N[0] * SIZE[0], 0.0, 0.0]
        st[:, 2] = -depth
    return st


def _setup(ctx, kind, st):
    rng = np.random.default_rng(5)
    s = W.Survey("precision", np.full(N[0], SIZE[0]), np.full(N[1], SIZE[1]),
                 np.full(N[2], SIZE[2]), (0.0, 0.0, 0.0), st, kind,
                 rng.uniform(0, 3000, N[0] * N[1] * N[2]), bg_thick=np.zeros(0))
    W.setup_context(ctx, s)
    return s


def _rms(v):
    return float(np.sqrt(np.mean(np.square(v.astype(np.longdouble)))))


def _check(name, got, exact, fp64):
    bound = 2.0 * _rms(fp64 - exact) + 2.0 ** -52 * float(np.abs(exact).max())
    assert _rms(got - exact) <= bound, (name, _rms(got - exact), bound)


PLACES = [("below", 1.0), ("below", 500.0), ("below", 2000.0), ("above", 1.0), ("above", 500.0),
          ("above", 2000.0), ("aside", 100.0), ("among", 0.0)]


@pytest.mark.gpu
@pytest.mark.parametrize("where,depth", PLACES)
@pytest.mark.parametrize("kind", [W.SCALAR, W.TENSOR, W.JOINT])
def test_data_of_each_component(ctx, kind, where, depth):
    st = _stations(where, depth)
    s = _setup(ctx, kind, st)
    d = ctx.forward(s.model).reshape(len(st), -1)
    rho = -_model_differences(s.model)
    rho_long = -_differences(np.pad(s.model.reshape(N).astype(np.longdouble), 1), 0)
    long, fp64 = _terms(st, np.longdouble), _terms(st, np.float64)
    comps = (["gz"] if kind != W.TENSOR else []) + (list(ROWS) if kind != W.SCALAR else [])
    for c in comps:
        k = 0 if c == "gz" else ROWS[c] + (kind == W.JOINT)
        exact = _scale(c) * (long[c] * rho_long).reshape(len(st), -1).sum(axis=1)
        sums = _scale(c) * _level_sums(fp64[c] * rho)
        _check(c, d[:, k], exact, sums)


@pytest.mark.gpu
@pytest.mark.parametrize("where,depth", PLACES)
@pytest.mark.parametrize("kind", [W.SCALAR, W.TENSOR, W.JOINT])
def test_gradient_of_each_component(ctx, kind, where, depth):
    st = _stations(where, depth)
    s = _setup(ctx, kind, st)
    w = np.random.default_rng(9).normal(size=len(st))
    long, fp64 = _terms(st, np.longdouble), _terms(st, np.float64)
    rows = {W.SCALAR: 1, W.TENSOR: 9, W.JOINT: 10}[kind]
    comps = (["gz"] if kind != W.TENSOR else []) + (list(ROWS) if kind != W.SCALAR else [])
    for c in comps:
        misfit = np.zeros((len(st), rows))
        misfit[:, 0 if c == "gz" else ROWS[c] + (kind == W.JOINT)] = w
        g = ctx.lqderivative(s.model, misfit.ravel())
        ws = w.reshape(-1, 1, 1, 1)
        exact = 2 * _scale(c) * _differences((ws * long[c]).sum(axis=0), 0).ravel()
        sums = 2 * _scale(c) * _differences(
            np.add.accumulate(ws * fp64[c], axis=0)[-1], 0).ravel()
        _check(c, g, exact, sums)
