"""The detector gather's cell widths with the source close to the image.

A cell's width is linear in the line, and largest on the far side of the image,
so it has to be held from the line nearest the source on: there both of its terms
are positive and each rounds once, by 2^-24 of the width. Held from the far side,
the near lines, which carry the most weight, are left with what cancels."""

import math

import numpy as np
import pytest

from ctlib_gb300.workloads import FAN_EA, FAN_ED, fan_options
from test_geometry_host import _query, native  # noqa: F401


@pytest.mark.parametrize("scan", [FAN_ED, FAN_EA])
@pytest.mark.parametrize("ratio", [4.0, 1.2, 0.8, 0.72])
@pytest.mark.parametrize("size", [(96, 128), (61, 45)])
def test_widths_hold_close_to_the_source(native, scan, ratio, size):  # noqa: F811
    W, H = size
    V, D = 24, 90
    r = ratio * max(W, H)
    half = min(0.75, math.asin(min(0.99, 0.71 / ratio)))
    d = 2 * 1.8 * r * math.tan(half) / D if scan == FAN_ED else 2 * half / D
    opts = fan_options(V, D, W, H, 1.0, d, 0.0, 2 * math.pi / V, r, 0.8 * r, 0.0, scan)
    L = max(W, H)
    flags = _query(native, opts, 0).astype(int)
    db = _query(native, opts, 1).reshape(V, D + 1)
    lp = _query(native, opts, 3).reshape(V, L, 2)
    walk = _query(native, opts, 8).reshape(V, D, 6)
    for v in range(V):
        nl = H if flags[v] & 1 else W
        width = np.diff(db[v])[None] / lp[v, :nl, 1:]
        got = walk[v, :, 2] + walk[v, :, 3] * np.arange(nl)[:, None]
        # (a margin of 2^-28 for the query's and this test's own double arithmetic)
        assert (np.abs(got - width) <= (2.0 ** -24 + 2.0 ** -28) * width).all(), v
