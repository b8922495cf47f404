"""Workspaces of the gradients: bounded for any number of station subsets, and
smaller where the device's memory is nearly taken."""
import contextlib

import numpy as np
import pytest

from helpers import relerr
from jif3d_gb300 import capi, workloads as W

pytestmark = pytest.mark.gpu
GB = 1 << 30


def _survey(kind, nmeas):
    """64 x 64 x 32 cells (139,425 nodes, 1.1 MB a chunk of stations)."""
    rng = np.random.default_rng(21)
    n = (64, 64, 32)
    size = [np.full(k, w) for k, w in zip(n, (50.0, 50.0, 25.0))]
    st = rng.uniform(0, 3200, (nmeas, 3))
    st[:, 2] = -rng.uniform(1, 100, nmeas)
    return W.Survey("memory", *size, (0.0, 0.0, 0.0), st, kind, rng.uniform(1, 11, 64 * 64 * 32),
                    bg_thick=np.zeros(0))


@contextlib.contextmanager
def _memory_left(left):
    """All of the device's free memory but `left` bytes held."""
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del held
        torch.cuda.empty_cache()


def test_many_subsets_share_a_bounded_workspace():
    """2000 subsets of one station, a chunk each: 2.2 GB of chunk sums, taken a
    gigabyte at a time."""
    import torch
    s = _survey(W.SCALAR, 2000)
    n = s.stations.shape[0]
    like = dict(dtype=torch.float64, device="cuda")
    ctx = capi.Context(0)
    W.setup_context(ctx, s)
    misfit = np.random.default_rng(2).normal(size=n)
    m, r = torch.tensor(s.model, **like), torch.tensor(misfit, **like)
    g = torch.zeros(n, s.nparm, **like)
    parts = torch.zeros(n, s.nparm, **like)
    subsets = [np.array([k]) for k in range(n)]
    # 500 at a time: 0.56 GB of chunk sums
    for k in range(0, n, 500):
        ctx.subsets_lqderivative_device(subsets[k:k + 500], m.data_ptr(), r[k:].data_ptr(),
                                        parts[k:].data_ptr())
    ctx.synchronize()
    before = torch.cuda.mem_get_info()[0]
    ctx.subsets_lqderivative_device(subsets, m.data_ptr(), r.data_ptr(), g.data_ptr())
    ctx.synchronize()
    assert before - torch.cuda.mem_get_info()[0] <= GB
    # the same chunks of the same stations: bit for bit the same
    assert torch.equal(g, parts)
    ctx.close()


def test_gradient_with_little_memory():
    """14,000 stations: the chunks' sums take 0.98 GB, one chunk's where that
    cannot be had; station subsets likewise.  Bound: a node's chain of n additions of
    misfit times term (up to 3e4 m) is 2^-53 * 0.4 n 3e4 off (random signs), a cell
    takes eight nodes twice, and is itself about 2 * 0.3 m * sqrt(n): 2e-9 of it for
    n = 14,000, and the same for the order it is compared with."""
    import torch
    s = _survey(W.SCALAR, 14000)
    misfit = np.random.default_rng(3).normal(size=14000)
    like = dict(dtype=torch.float64, device="cuda")
    m, r = torch.tensor(s.model, **like), torch.tensor(misfit, **like)
    subsets = [np.arange(0, 9000), np.arange(9000, 9001), np.arange(9001, 14000)]

    def run():
        g = torch.zeros(4, s.nparm, **like)
        ctx = capi.Context(0)
        W.setup_context(ctx, s)
        for _ in range(2):
            ctx.lqderivative_device(m.data_ptr(), r.data_ptr(), g[3].data_ptr())
            ctx.subsets_lqderivative_device(subsets, m.data_ptr(), r.data_ptr(), g.data_ptr())
        ctx.synchronize()
        ctx.close()
        return g.cpu().numpy()
    ref = run()
    with _memory_left(GB * 6 // 10):
        got = run()
    for a, b in zip(got, ref):
        assert relerr(a, b) <= 4e-9


def test_fp32_batch_with_little_memory():
    """Four models on 14 GB of J: 0.9 GB of chunk sums for all of them in one
    pass, a quarter of that one by one, bit for bit the same."""
    s = _survey(W.JOINT, 3930)
    rng = np.random.default_rng(4)
    models = s.model[None, :] * (1 + 0.1 * rng.normal(size=(4, s.nparm)))
    misfits = rng.normal(size=(4, 3930 * s.dpm))
    ctx = capi.Context(0)
    W.setup_context(ctx, s)
    ctx.build_sensitivity(capi.STORE_FP32)
    with _memory_left(GB * 6 // 10):
        got = [ctx.batched_lqderivative(models, misfits) for _ in range(2)]
    ctx.build_sensitivity(capi.STORE_FP32)  # four models a pass again
    ref = ctx.batched_lqderivative(models, misfits)
    ctx.close()
    for g in got:
        assert np.array_equal(g, ref)


def test_given_corners_with_little_memory(oracle_lib):
    """142 x 142 x 142 cells, no corner shared, three model blocks: 0.55 GB of model
    differences on the node planes and as much of chunk sums, 0.2 GB of eight-corner
    rows for the one station where that cannot be had."""
    n = 142
    size = np.full(n, 20.0)
    corner = 21.0 * np.arange(n)  # gaps of a metre
    rng = np.random.default_rng(6)
    s = W.Survey("gaps", size, size, size, (0.0, 0.0, 0.0), np.array([[1500.0, 1400.0, -30.0]]),
                 W.MAGNETIZATION, rng.uniform(1, 11, 3 * n ** 3), bg_thick=np.zeros(0))
    ctx = capi.Context(0)
    W.setup_context(ctx, s)
    ctx.set_mesh(corner, corner, corner, size, size, size)
    p = oracle_lib.Problem(corner, corner, corner, size, size, size, s.stations, kind=s.kind)
    misfit = rng.normal(size=3)
    with _memory_left(GB * 45 // 100):
        got = ctx.forward(s.model), ctx.lqderivative(s.model, misfit)
    ctx.close()
    assert relerr(got[0], p.forward(s.model)) <= 1e-10
    assert relerr(got[1], p.lqderivative(s.model, misfit)) <= 1e-10
