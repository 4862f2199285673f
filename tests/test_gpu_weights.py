"""The backprojectors' weights, each alone.

A parallel beam's weight is the one constant 1 / dImg, so its rounding scales the
whole image: it has to be the correctly rounded reciprocal. One cell that covers
the image, holding 1, leaves a single product per pixel, the pixel's length dImg
times the weight, whose bits numpy gives."""

import math

import numpy as np
import pytest
import torch

from ctlib_gb300.workloads import para_options

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
