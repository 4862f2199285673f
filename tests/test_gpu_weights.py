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

from ctlib_gb300.workloads import FAN_EA, FAN_ED, fan_options, para_options

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


U64 = 2.0 ** -53


@pytest.mark.parametrize("scan", [FAN_ED, FAN_EA])
@pytest.mark.parametrize("col", range(6))
def test_double_overlaps_are_divided_to_a_few_ulp(scan, col):
    """B^T in fp64 of one pixel of 1 that a wide cell covers, at every place of the
    walk's two straight pixels and its remainder. Roundings: the product of two
    divisors, its reciprocal (one, and below 2^-57 of the method) and the factor
    back, 3; squared, 6, the square and the overlap's product 2: 8 and a little.
    Equal-angle fans: 4 so far, 3 of the distance, 2 of the cell's factor and its
    product, whose table adds up to 5: 14."""
    import ctlib_gb300 as ct
    H, W, r = 256, 6, 1024.0
    L = np.longdouble
    d = 8.0 * W if scan == FAN_ED else 0.05
    opts = fan_options(1, 1, W, H, 1.0, d, 0.0, 2 * math.pi, r, r, 0.0, scan)
    x = torch.zeros(H, 1, H, W, dtype=torch.float64)
    x[torch.arange(H), 0, torch.arange(H), col] = 1
    got = ct.backprojection_t(x.cuda(), torch.tensor(opts, dtype=torch.float64)).cpu().numpy().ravel().astype(L)
    y = H / 2 - np.arange(H).astype(L) - L(0.5)
    if scan == FAN_ED:
        want, tol = 1 / (1 - y / r) ** 2, 9 * U64
    else:
        cbar = np.cos(L(d) / 2)  # both boundaries alike
        want, tol = 1 / ((L(col) + L(0.5) - L(W) / 2) ** 2 + (r - y) ** 2) / cbar, 14 * U64
    assert (np.abs(got / want - 1) <= tol).all(), float(np.abs(got / want - 1).max() / U64)


@pytest.mark.parametrize("scan", [FAN_ED, FAN_EA])
def test_double_weights_are_good_to_a_few_ulp(scan):
    """B in fp64 of one wide cell of 1: the pixel's length, an integer of 2^50 units
    or more (4 U64 at its worst), times the weight (its divisor 4, reciprocal and
    product 3), to the unit and back 1: 12."""
    import ctlib_gb300 as ct
    H, W, r = 256, 6, 1024.0
    L = np.longdouble
    d = 8.0 * W if scan == FAN_ED else 0.05
    opts = fan_options(1, 1, W, H, 1.0, d, 0.0, 2 * math.pi, r, r, 0.0, scan)
    got = ct.backprojection(torch.ones(1, 1, 1, 1, dtype=torch.float64, device="cuda"),
                            torch.tensor(opts, dtype=torch.float64)).cpu().numpy()[0, 0].astype(L)
    y = (H / 2 - np.arange(H).astype(L) - L(0.5))[:, None]
    q = np.arange(W).astype(L) + L(0.5) - L(W) / 2
    want = 1 / (1 - y / r) ** 2 + 0 * q if scan == FAN_ED else 1 / (q ** 2 + (r - y) ** 2)
    assert (np.abs(got / want - 1) <= 12 * U64).all(), float(np.abs(got / want - 1).max() / U64)
