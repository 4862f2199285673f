"""The detector gather's fixed-point walk at the sizes where it can go
wrong: single pixels, lines and cells, lines one past a block of four or a fold
of 32, rows past a multiple of 32 cells, cells much wider and much narrower than
a pixel, cells off the image; every slices-per-thread width.

Tolerance: an overlap is formed from a position good to 2^-24 pixels and a width
good to 2^-23 of itself, a weight adds 3 roundings and at most 2 ulp of a
reciprocal, and sums round by 2^-24 per term within blocks of 32 lines: below
8 * 2^-23 = 9.5e-7 of the result's norm. In fp64 the axis coordinates, up to 1e3
pixels, are rounded by 2^-53: below 4e-13 of a cell of 0.3 pixels, so 1e-12."""

import math

import numpy as np
import pytest
import torch

from ctlib_gb300.workloads import FAN_EA, FAN_ED, fan_options, para_options

pytestmark = pytest.mark.gpu

SIZES = [  # views, dets, width, height, cell width in pixels
    (3, 1, 1, 1, 0.7), (5, 33, 4, 7, 1.1), (4, 3, 9, 5, 7.0), (6, 97, 31, 66, 0.3), (9, 64, 33, 32, 1.0),
    (7, 40, 65, 3, 2.6), (8, 31, 2, 129, 1.6),
]


def _options(scan, V, D, W, H, cell, shift):
    r = 4.0 * max(W, H, D * cell / 2) + 8
    if scan == FAN_ED:
        return fan_options(V, D, W, H, 1.0, 1.6 * cell, 0.2, 2 * math.pi / V, r, 0.6 * r, shift, scan)
    if scan == FAN_EA:
        return fan_options(V, D, W, H, 1.0, cell / r, 0.2, 2 * math.pi / V, r, 0.6 * r, shift / r, scan)
    return para_options(V, D, W, H, 1.0, cell, 0.2, math.pi / V, shift)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("scan", [0, 1, 2])
@pytest.mark.parametrize("size", SIZES)
def test_walk_edges(oracle_mod, scan, size, dtype):
    import ctlib_gb300 as ct
    V, D, W, H, cell = size
    opts = _options(scan, V, D, W, H, cell, 0.35 * cell)
    f32 = dtype == np.float32
    o = torch.tensor(opts, dtype=torch.float64)
    mode, tol = (oracle_mod.MODE_F64_ON_F32, 8 * 2.0 ** -23) if f32 else (oracle_mod.MODE_F64, 1e-12)
    x = np.random.default_rng(V * D + W).uniform(0.5, 1.5, (17, 1, H, W)).astype(dtype)
    xd = torch.from_numpy(x).cuda()
    for op in ("projection", "backprojection_t"):
        f = getattr(ct, op)
        whole = f(xd, o)
        want = oracle_mod.run(op, x, opts, mode)
        assert oracle_mod.rel_l2(whole.cpu().numpy(), want) <= tol, op
        for n in (1, 2, 3, 8):  # other slices per thread: the same bits
            assert torch.equal(f(xd[:n].contiguous(), o), whole[:n]), (op, n)


@pytest.mark.parametrize("scan", [0, 1, 2])
@pytest.mark.parametrize("size", [(300, 200, 96, 80, 0.9), (64, 70, 130, 130, 2.4), (361, 33, 40, 37, 1.2)])
def test_staged_lines_match_global_ones(scan, size):
    """From eight slices per thread on, lines are staged in shared memory where the
    views lie close enough; fewer read global memory. The bits
    agree, also when every wait for a staged slot gives up at once."""
    import ctlib_gb300 as ct
    from ctlib_gb300 import _native as N
    from ctlib_gb300.ops import Plan
    V, D, W, H, cell = size
    opts = _options(scan, V, D, W, H, cell, 0.0)
    o = torch.tensor(opts, dtype=torch.float32)
    g = torch.Generator().manual_seed(7)
    x = torch.randn(21, 1, H, W, generator=g).cuda()
    N.wait_timeouts(0, reset=True)
    for op, name in ((0, "projection"), (3, "backprojection_t")):
        f = getattr(ct, name)
        one = torch.cat([f(x[i:i + 1].contiguous(), o) for i in range(21)])
        for n in (21, 16, 7, 4):
            assert torch.equal(f(x[:n].contiguous(), o), one[:n]), (name, n)
        assert N.wait_timeouts(0) == 0
        plan = Plan(tuple(opts), torch.float32, 0)
        N.check(N.lib().ctgb_plan_set_wait_limit(plan.handle, 0), "wait limit")
        out = torch.empty_like(one)
        plan.run(op, x, out)
        torch.cuda.synchronize()
        assert torch.equal(out, one), name
        N.wait_timeouts(0, reset=True)
