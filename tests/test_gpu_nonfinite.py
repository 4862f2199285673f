"""An infinite or NaN sample reaches every result that overlaps it, whatever the
batch, and none more than two pixels (cells) past it: straight-line steps multiply
samples next to a cell (pixel) by 0. Results beyond keep their bits."""

import math

import numpy as np
import pytest
import torch

from ctlib_gb300.workloads import para_options

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("cell", [0.4, 0.9, 1.3, 2.6])
@pytest.mark.parametrize("batch", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("bad", [math.nan, math.inf])
def test_reach_of_a_nonfinite_sample(dtype, cell, batch, bad):
    import ctlib_gb300 as ct
    H, W = 6, 40
    D = int(1.2 * W / cell)
    # view angle 0: rows are lines, and cell d covers the columns from D edges on
    o = torch.tensor(para_options(1, D, W, H, 1.0, cell, 0.0, math.pi, 0.137), dtype=torch.float64)
    edge = (np.arange(D + 1) - D / 2) * cell + 0.137 + W / 2
    lo, hi = edge[:-1], edge[1:]
    g = torch.Generator().manual_seed(3)
    for op in ("projection", "backprojection_t", "projection_t", "backprojection"):
        f, image = getattr(ct, op), op in ("projection", "backprojection_t")
        shape = (batch, 1, H, W) if image else (batch, 1, 1, D)
        x = torch.randn(shape, generator=g, dtype=torch.float64).to("cuda", dtype)
        clean = f(x, o)
        for at in (0, shape[3] // 2, shape[3] - 1):
            y = x.clone()
            y[:, 0, 0, at] = bad
            out = f(y, o)
            if image:  # gap between cell and pixel, in pixels; negative: overlap
                gap, got, ref = np.maximum(lo - (at + 1), at - hi), out[:, 0, 0], clean[:, 0, 0]
            else:      # between pixel and cell, in cells
                col = np.arange(W)
                gap = np.maximum(col - hi[at], lo[at] - (col + 1)) / cell
                got, ref = out[:, 0].reshape(batch * H, W), clean[:, 0].reshape(batch * H, W)
            near = torch.from_numpy(gap < -1e-3).cuda()
            far = torch.from_numpy(gap > 2.001).cuda()
            assert not torch.isfinite(got[:, near]).any(), (op, at)
            assert torch.equal(got[:, far], ref[:, far]), (op, at)
