"""The image gather at the sizes where it can go wrong: images of one pixel and
one past a tile of 32 columns or of 8 to 32 rows, cells much wider and much
narrower than a pixel (searches, many cells per pixel), pixels off the detector
on either side, view counts on both sides of a split; every slices-per-thread
width in both precisions.

Tolerance: an overlap is a difference of coordinates good to 2^-38 of themselves,
rounded by a few 2^-24 of the overlap, a weight adds the roundings of its terms and
at most 2 ulp of a reciprocal, and sums round by 2^-24 per term within blocks of 32
views: below 8 * 2^-23 of the result's norm. In fp64 the coordinates, up to 1e3
pixels, carry roundings of 2^-53: below 4e-13 of a cell of 0.3 pixels, so 1e-12."""

import numpy as np
import pytest
import torch

from test_gpu_det_walk import _options

pytestmark = pytest.mark.gpu

SIZES = [  # views, dets, width, height, cell width in pixels, detector shift in cells
    (3, 1, 1, 1, 0.7, 0.2), (90, 70, 33, 40, 0.3, 0.4), (100, 9, 65, 31, 3.0, -0.3), (300, 30, 31, 33, 0.5, 0.0),
    (41, 64, 64, 9, 1.0, 0.5), (170, 25, 20, 129, 1.4, 12.0), (82, 300, 47, 65, 0.22, -80.0),
]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("scan", [0, 1, 2])
@pytest.mark.parametrize("size", SIZES)
def test_gather_edges(oracle_mod, scan, size, dtype):
    import ctlib_gb300 as ct
    V, D, W, H, cell, shift = size
    opts = _options(scan, V, D, W, H, cell, shift * cell)
    o = torch.tensor(opts, dtype=torch.float64)
    f32 = dtype == np.float32
    mode, tol = (oracle_mod.MODE_F64_ON_F32, 8 * 2.0 ** -23) if f32 else (oracle_mod.MODE_F64, 1e-12)
    y = np.random.default_rng(V * D + W).uniform(0.5, 1.5, (17, 1, V, D)).astype(dtype)
    yd = torch.from_numpy(y).cuda()
    for op in ("projection_t", "backprojection"):
        f = getattr(ct, op)
        whole = f(yd, o)
        want = oracle_mod.run(op, y, opts, mode)
        assert np.linalg.norm(want) > 0
        assert oracle_mod.rel_l2(whole.cpu().numpy(), want) <= tol, op
        for n in (1, 2, 3, 8):  # other slices per thread: the same bits
            assert torch.equal(f(yd[:n].contiguous(), o), whole[:n]), (op, n)
