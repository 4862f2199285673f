"""Operators with the source close to the image, where cells and pixels differ most
in width between the near and the far side.

Tolerance of the fp32 detector gather, as for a far source (test_gpu_det_walk):
positions good to 2^-24 pixels, widths to 2^-23 of themselves, a weight of 3
roundings and 2 ulp of a reciprocal, sums rounding by 2^-24 per term within blocks
of 32 lines: below 8 * 2^-23. The equal-distance weight is left out: its divisor
1 - n . p cancels towards the source."""

import math

import numpy as np
import pytest
import torch

from ctlib_gb300.workloads import FAN_EA, FAN_ED, fan_options

pytestmark = pytest.mark.gpu


def _options(scan, ratio, size, V, D):
    r = ratio * size
    half = min(0.75, math.asin(min(0.99, 0.71 / ratio)))
    d = 2 * 1.8 * r * math.tan(half) / D if scan == FAN_ED else 2 * half / D
    return fan_options(V, D, size, size, 1.0, d, 0.0, 2 * math.pi / V, r, 0.8 * r, 0.0, scan)


@pytest.mark.parametrize("op,scan", [("projection", FAN_ED), ("projection", FAN_EA), ("backprojection_t", FAN_EA)])
@pytest.mark.parametrize("ratio", [1.2, 0.8, 0.72])
def test_detector_gather(oracle_mod, op, scan, ratio):
    import ctlib_gb300 as ct
    opts = _options(scan, ratio, 256, 144, 368)
    x = np.random.default_rng(3).uniform(0.5, 1.5, (8, 1, 256, 256)).astype(np.float32)
    f, o = getattr(ct, op), torch.tensor(opts, dtype=torch.float64)
    xd = torch.from_numpy(x).cuda()
    got = f(xd, o)
    for n in (1, 4):
        assert torch.equal(f(xd[:n].contiguous(), o), got[:n]), n
    want = oracle_mod.run(op, x, opts, oracle_mod.MODE_F64_ON_F32)
    for v in range(144):  # view by view: only those with the source below or right of the image can fail
        assert oracle_mod.rel_l2(got[:, :, v].cpu().numpy(), want[:, :, v]) <= 8 * 2.0 ** -23, v


@pytest.mark.parametrize("op", ["projection_t", "backprojection", "projection", "backprojection_t"])
@pytest.mark.parametrize("scan", [FAN_ED, FAN_EA])
@pytest.mark.parametrize("ratio", [0.8, 0.72])
def test_double_precision(oracle_mod, op, scan, ratio):
    """Pixels next to the source take more than 52 bits of the image gather's units.
    Axis coordinates of up to 2^8 pixels, off by 4 roundings of 2^-53: 1e-12 of a
    pixel of 0.5 on the far side holds 4 times over."""
    import ctlib_gb300 as ct
    opts = _options(scan, ratio, 256, 24, 368)
    image = op in ("projection", "backprojection_t")
    x = np.random.default_rng(4).standard_normal((3, 1) + ((256, 256) if image else (24, 368)))
    got = getattr(ct, op)(torch.from_numpy(x).cuda(), torch.tensor(opts, dtype=torch.float64)).cpu().numpy()
    assert oracle_mod.rel_l2(got, oracle_mod.run(op, x, opts, oracle_mod.MODE_F64)) <= 1e-12
