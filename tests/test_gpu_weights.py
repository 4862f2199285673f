"""The backprojectors' weights, each alone.

A parallel beam's weight is the one constant 1 / dImg, so its rounding scales the
whole image: it has to be the correctly rounded reciprocal. One cell that covers
the image, holding 1, leaves a single product per pixel, the pixel's length dImg
times the weight, whose bits numpy gives.

A fan at view angle 0 with the source 1024 pixels away weighs line y by 1 / t^2, t =
1 - y / 1024, which is exact in fp32: what is left is the division's rounding."""

import math

import numpy as np
import pytest
import torch

from ctlib_gb300.workloads import FAN_ED, fan_options, para_options

pytestmark = pytest.mark.gpu


def test_parallel_weight_is_the_rounded_reciprocal():
    import ctlib_gb300 as ct
    T = np.float32
    rng = np.random.default_rng(11)
    y = torch.ones(1, 1, 1, 1, device="cuda")
    for h in rng.uniform(0.1, 4.0, 300).astype(T):
        opts = para_options(1, 1, 8, 8, float(h), 64.0 * float(h), 0.0, math.pi, 0.0)
        out = ct.backprojection(y, torch.tensor(opts, dtype=torch.float64)).cpu().numpy()
        assert (out == h * (T(1) / h)).all(), (h, out[0, 0, 0, 0], h * (T(1) / h))


def _fan_one_view(H, W):
    T = np.float32
    t = 1 - (H / 2 - np.arange(H) - 0.5) / 1024
    assert (t == t.astype(T)).all() and (t * t == (t * t).astype(T)).all()
    opts = fan_options(1, 1, W, H, 1.0, 8.0 * W, 0.0, 2 * math.pi, 1024.0, 1024.0, 0.0, FAN_ED)
    return torch.tensor(opts, dtype=torch.float64), (t * t).astype(T), (1 / t).astype(T)


@pytest.mark.parametrize("batch", [1, 2, 4, 8, 16])
def test_fan_overlaps_are_divided_to_the_last_bit(batch):
    """B^T of one pixel of 1 that a wide cell covers: overlap 1 over t^2."""
    import ctlib_gb300 as ct
    H, W = 256, 6
    o, t2, _ = _fan_one_view(H, W)
    for l0 in range(0, H, batch):
        x = torch.zeros(batch, 1, H, W)
        x[torch.arange(batch), 0, l0 + torch.arange(batch), 3] = 1
        got = ct.backprojection_t(x.cuda(), o).cpu().numpy().ravel()
        assert (got == np.float32(1) / t2[l0:l0 + batch]).all(), l0


def test_fan_weights_are_rounded_reciprocals():
    """B of one wide cell of 1: a pixel's length on the axis, 1 / t, times 1 / (t^2 / t)."""
    import ctlib_gb300 as ct
    H, W = 256, 6
    o, t2, length = _fan_one_view(H, W)
    got = ct.backprojection(torch.ones(1, 1, 1, 1, device="cuda"), o).cpu().numpy()[0, 0]
    want = length * (np.float32(1) / (t2 * length))
    assert (got == want[:, None]).all()
