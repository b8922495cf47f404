"""The fixed-point node terms (csrc/node_fixed.cuh): on the host against long
double, and the kernels built on them at the edges of their tiles against FP64
sums with log(r + d) formed without cancellation (on deep columns the oracle's
own rounding of r + d, d negative, is worth up to 7e-9 of the data).

Host bounds, from the number formats: a logarithm at scale 2^57 carries a few
units of truncation (2^-54) and the relative error 2^-56 of its argument,
enlarged by r / (r + d) where a negative offset cancels; an angle 2^-56, and
2^-48 of itself where it is small; each is rounded once to FP64.
"""
import os
import shutil
import subprocess

import numpy as np
import pytest

from helpers import oracle_forward, relerr, small_survey
from jif3d_gb300 import build as B, workloads as W

HERE = os.path.dirname(os.path.abspath(__file__))
KINDS = [W.SCALAR, W.TENSOR, W.MAGNETIC, W.JOINT, W.MAG_GRADIENT, W.MAGNETIZATION]


def test_terms_against_long_double(tmp_path):
    cxx = shutil.which("g++")
    assert cxx, "a host compiler is needed"
    exe = str(tmp_path / "node_fixed_check")
    src = os.path.join(HERE, "cpp", "node_fixed_check.cpp")
    r = subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", B.CSRC, src, "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([exe], capture_output=True, text=True, timeout=600).stdout
    rows = [line.split() for line in out.splitlines()]
    assert len(rows) == 24
    for name, which, n, left, *worst in rows:
        # only the sets with cancelling, exactly zero or far-apart offsets leave any
        assert int(left) <= {"1": 0.1, "4": 0.05, "5": 1.0, "2": 0.0}.get(which, 0.001) * int(n), \
            (name, which, left)
        assert all(float(w) <= 1.0 for w in worst), (name, which, worst)


def _survey(kind, nx, ny, nz, nmeas, aligned):
    s = small_survey(kind, nx=nx, ny=ny, nz=nz, nmeas=nmeas, seed=nx + 10 * ny + 100 * nz + kind,
                     bg=False)
    if kind == W.MAGNETIZATION:
        rng = np.random.default_rng(nx)
        s.model = rng.uniform(1, 11, 3 * s.ngrid)
    if aligned:
        # stations above columns, on node planes, and level with the mesh's top
        n = s.stations.shape[0]
        s.stations[:, 0] = s.coords(0)[np.arange(n) % (nx + 1)]
        s.stations[::2, 1] = s.coords(1)[(np.arange(n) % (ny + 1))[::2]]
    return s


GRAV = 6.67428e-11


def _prisms(s, st):
    """Prism values of the seven components [stations][cells] (FP64)."""
    d = [st[:, a].reshape(-1, 1, 1, 1) - s.coords(a).reshape([1] + [-1 if b == a else 1
                                                                   for b in range(3)])
         for a in range(3)]
    x, y, z = d
    xx, yy, zz = x * x, y * y, z * z
    r = np.sqrt(xx + yy + zz)

    def ln(u, rest):
        with np.errstate(divide="ignore", invalid="ignore"):
            return np.log(np.maximum(np.where(u < 0, rest / (r - u), u + r), 2.0 ** -52))
    lx, ly = ln(x, yy + zz), ln(y, xx + zz)
    F = {"gz": x * ly + y * lx + z * np.arctan2(z * r, x * y), "xx": np.arctan2(y * z, x * r),
         "yy": np.arctan2(x * z, y * r), "zz": np.arctan2(x * y, z * r), "xy": ln(z, xx + yy),
         "xz": ly, "yz": lx}
    out = {}
    for k, f in F.items():
        for a in (1, 2, 3):
            f = np.diff(f, axis=a)
        out[k] = (GRAV if k in ("xx", "yy", "zz") else -GRAV) * f.reshape(f.shape[0], -1)
    return out


def _rows(s):
    """Raw sensitivity rows [stations * raw][parameters]."""
    def rows(st):
        p = _prisms(s, st)
        t = [p[k] for k in ("xx", "xy", "xz", "xy", "yy", "yz", "xz", "yz", "zz")]
        b = (np.cos(s.inc) * np.cos(s.dec), np.cos(s.inc) * np.sin(s.dec), np.sin(s.inc))
        if s.kind == W.SCALAR:
            return [p["gz"]]
        if s.kind == W.TENSOR:
            return t
        if s.kind == W.JOINT:
            return [p["gz"]] + t
        if s.kind == W.MAGNETIC:
            f = s.fs / (4 * np.pi * GRAV)
            return [f * sum(b[j] * t[3 * k + j] for j in range(3)) for k in range(3)]
        if s.kind == W.MAGNETIZATION:
            f = 1e9 * 4e-7 * np.pi / (4 * np.pi * GRAV)
            return [f * np.concatenate([t[3 * k + j] for j in range(3)], axis=1) for k in range(3)]
        f = s.fs * 1e-7 / GRAV
        return [f * (b[0] * p["xz"] + b[1] * p["yz"] + b[2] * p["zz"])]
    J = rows(s.stations)
    if s.kind == W.MAG_GRADIENT:
        J = [J[0] - rows(s.stations + [0.0, 0.0, 1.0])[0]]
    return np.stack(J, axis=1).reshape(-1, J[0].shape[1])


# columns (nx + 1)(ny + 1) around a warp and around a block, nodes per column
# around the pieces of 8 and 64, stations around the stages of 16 and the
# chunks of 64
SHAPES = [(1, 1, 1, 1), (3, 7, 7, 15), (2, 10, 8, 16), (15, 15, 15, 17), (15, 16, 16, 64),
          (4, 5, 63, 65), (6, 4, 64, 33), (5, 5, 130, 129)]


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("kind", KINDS)
def test_kernels_at_tile_edges(ctx, kind, shape):
    for aligned in (False, True):
        s = _survey(kind, *shape, aligned)
        W.setup_context(ctx, s)
        J = _rows(s)
        d = ctx.forward(s.model)
        assert relerr(d, J @ s.model) <= 1e-10
        misfit = np.random.default_rng(3).normal(size=d.size)
        assert relerr(ctx.lqderivative(s.model, misfit), 2.0 * (misfit @ J)) <= 1e-10


@pytest.mark.gpu
@pytest.mark.parametrize("kind", [W.SCALAR, W.TENSOR, W.JOINT])
def test_offsets_left_to_fp64(ctx, oracle_lib, kind):
    """Stations level with the mesh's top on a node plane (two zero offsets), a
    millimetre above an edge's line, and offsets beyond 2^40 m: the nodes that
    the fixed-point terms leave out."""
    s = _survey(kind, 6, 5, 4, 8, False)
    s.stations[:, 2] = -20.0
    s.stations[0] = [s.coords(0)[2] + 3.0, s.coords(1)[0] - 5.0, -1e-3]
    s.stations[1] = [s.coords(0)[0] - 900.0, s.coords(1)[2], -1e-2]
    s.stations[2] = [s.coords(0)[3], s.coords(1)[0] - 40.0, 0.0]
    W.setup_context(ctx, s)
    d, ref = ctx.forward(s.model), oracle_forward(oracle_lib, s)
    assert np.array_equal(np.isnan(d), np.isnan(ref))  # g_z on an edge's line is 0 log 0
    ok = ~np.isnan(ref)
    # values against the sums without cancellation: r + d of the first two
    # stations has no correct digits in the oracle's FP64
    assert relerr(d[ok], (_rows(s) @ s.model)[ok]) <= 1e-10
    far = s.subset([3])
    far.stations = np.array([[3e12, 0.0, -1.0]])
    W.setup_context(ctx, far)
    # the far field's box terms are rounding in FP64 too: finite, and no larger
    # than a few units of the node terms
    assert np.all(np.isfinite(ctx.forward(far.model)))


# rows of one station a multiple of 64, of 16, odd; fewer cells than a tile, not
# a multiple of it; one station, and more than a chunk of eight
@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("shape", [(3, 2, 1, 1), (5, 5, 5, 8), (7, 9, 11, 33), (16, 4, 8, 130)])
def test_stored_pair_at_tile_edges(ctx, kind, shape):
    """The fp16 pair and its transpose, built in one pass: J m of unit models and
    J^T r of unit residuals give the matrix back, column by column and row by
    row, within the 2^-21 of its entries' rows that hi + lo keep."""
    from jif3d_gb300 import capi
    s = _survey(kind, *shape, False)
    W.setup_context(ctx, s)
    J = _rows(s)
    ctx.build_sensitivity(capi.STORE_F16X2)
    rng = np.random.default_rng(5)
    cols = rng.choice(s.nparm, min(s.nparm, 40), replace=False)
    d = ctx.batched_forward(np.eye(s.nparm)[cols])
    bound = 2.0 ** -21 * np.abs(J).max(axis=1)
    # a unit model is centred on its mean, which is added back with J 1
    assert np.all(np.abs(d - J[:, cols].T) <= 2 * bound[None, :])
    rows = rng.choice(J.shape[0], min(J.shape[0], 40), replace=False)
    g = ctx.batched_lqderivative(None, np.eye(J.shape[0])[rows])
    assert np.all(np.abs(g - 2.0 * J[rows]) <= 2 * 2 * bound[rows, None])


@pytest.mark.gpu
@pytest.mark.parametrize("kind", [W.SCALAR, W.TENSOR, W.MAGNETIC, W.MAG_GRADIENT, W.MAGNETIZATION])
@pytest.mark.parametrize("apart", ["none", "some", "all"])
def test_planes_of_given_corners(ctx, oracle_lib, kind, apart):
    """Corners given one by one, lower and upper corners of neighbouring cells
    apart on no axis, on some planes, or on every plane (by a rounding step, by
    a gap and by an overlap): forward, gradient, and the gradients of station
    subsets against the oracle's eight corners per cell."""
    import torch
    s = _survey(kind, 6, 5, 4, 9, False)
    co = [s.coords(a) for a in range(3)]
    rng = np.random.default_rng(17)
    for a in range(3):
        inner = co[a][1:-1]
        shift = np.array([1e-9, 0.3, -0.2])[np.arange(inner.size) % 3]
        take = {"none": np.zeros(inner.size), "all": np.ones(inner.size),
                "some": rng.integers(0, 2, inner.size)}[apart]
        inner += take * shift
    size = (s.xsize, s.ysize, s.zsize)
    W.setup_context(ctx, s)
    ctx.set_mesh(*co, *size)
    p = oracle_lib.Problem(*co, *size, s.stations, kind=kind, inc=s.inc, dec=s.dec, fs=s.fs)
    d = ctx.forward(s.model)
    assert relerr(d, p.forward(s.model)) <= 1e-10
    misfit = rng.normal(size=d.size)
    assert relerr(ctx.lqderivative(s.model, misfit), p.lqderivative(s.model, misfit)) <= 1e-10
    # subsets [0, 3) and [3, 9): their gradients add up to that of all stations
    like = dict(dtype=torch.float64, device="cuda")
    m, r = torch.tensor(s.model, **like), torch.tensor(misfit, **like)
    g = torch.zeros(2, s.nparm, **like)
    torch.cuda.synchronize()
    ctx.subsets_lqderivative_device([np.arange(3), np.arange(3, 9)], m.data_ptr(), r.data_ptr(),
                                    g.data_ptr())
    ctx.synchronize()
    assert relerr(g.sum(0).cpu().numpy(), p.lqderivative(s.model, misfit)) <= 1e-10


# cells around the gradient's tiles of 2 x 4 x 16, station chunks below and
# beyond the 32 that a thread adds up (and the 1024 of 32 groups)
@pytest.mark.gpu
@pytest.mark.parametrize("kind,shape", [(W.SCALAR, (2, 4, 16, 31)), (W.TENSOR, (3, 5, 17, 400)),
                                        (W.MAGNETIZATION, (1, 9, 33, 260)),
                                        (W.SCALAR, (5, 3, 15, 5000))])
@pytest.mark.parametrize("given", [False, True])
def test_gradient_tiles_and_chunk_sums(ctx, kind, shape, given):
    """The gradient of all stations and of uneven subsets of them (one empty, one
    of one station), in one call and in a captured graph; with given corners the
    tile's nodes are planes."""
    import torch
    s = _survey(kind, *shape, False)
    n = s.stations.shape[0]
    W.setup_context(ctx, s)
    if given:  # an upper corner that is not the next lower one, by rounding
        co = [s.coords(a) for a in range(3)]
        co[2][1] = np.nextafter(co[2][1], np.inf)
        ctx.set_mesh(*co, s.xsize, s.ysize, s.zsize)
    J = _rows(s).reshape(n, -1, s.model.size)
    misfit = np.random.default_rng(4).normal(size=(n, J.shape[1]))
    cut = np.array([0, 0, 1, n // 3, n])
    like = dict(dtype=torch.float64, device="cuda")
    m, r = torch.tensor(s.model, **like), torch.tensor(misfit, **like)
    g = torch.full((5, s.model.size), np.nan, **like)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    ctx.set_stream(stream.cuda_stream)
    try:
        subsets = [np.arange(a, b) for a, b in zip(cut[:-1], cut[1:])]

        def run():
            ctx.subsets_lqderivative_device(subsets, m.data_ptr(), r.data_ptr(), g.data_ptr())
            ctx.lqderivative_device(m.data_ptr(), r.data_ptr(), g[4].data_ptr())
        run()
        ctx.synchronize()
        first = g.cpu().numpy()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            run()
        g.fill_(np.nan)
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
    finally:
        ctx.set_stream(0)
    assert np.array_equal(first, g.cpu().numpy())
    for k, (a, b) in enumerate(list(zip(cut[:-1], cut[1:])) + [(0, n)]):
        ref = 2.0 * np.einsum("sr,srp->p", misfit[a:b], J[a:b])
        assert relerr(first[k], ref) <= 1e-10 if b > a else np.all(first[k] == 0.0)


# more nodes to a column than a block takes at a time, and fewer
@pytest.mark.gpu
@pytest.mark.parametrize("kind", [W.TENSOR, W.MAGNETIC, W.JOINT])
@pytest.mark.parametrize("shape", [(6, 5, 9), (3, 2, 70)])
def test_stations_among_the_nodes(ctx, kind, shape):
    """dz of both signs and zero along the columns, where the sum of the three
    angles changes: stations between, on, above and below the mesh's planes, off
    the columns and on them."""
    s = _survey(kind, *shape, 24, False)
    n = s.stations.shape[0]
    z = s.coords(2)
    s.stations[:, 2] = np.concatenate([[z[0] - 5.0, z[-1] + 5.0, z[-1], z[0], z[2]],
                                       np.random.default_rng(8).uniform(z[0], z[-1], n - 5)])
    s.stations[8:, 0] = s.coords(0)[np.arange(n - 8) % (shape[0] + 1)]
    s.stations[16:, 1] = s.coords(1)[np.arange(n - 16) % (shape[1] + 1)]
    W.setup_context(ctx, s)
    J = _rows(s)
    d = ctx.forward(s.model)
    assert relerr(d, J @ s.model) <= 1e-10
    misfit = np.random.default_rng(3).normal(size=d.size)
    assert relerr(ctx.lqderivative(s.model, misfit), 2.0 * (misfit @ J)) <= 1e-10
