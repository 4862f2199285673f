"""The fp64 image gather's pixel edges are integers in units of 2^-s. The unit has to
be as fine as the rounding of the edges themselves, also on the far side of an
image whose near side lies close to the source, where pixels are projected much
wider: every edge within 2^-53 of its line's extent, as a double holds it, or
within 2^-48 of a pixel."""

import math

import pytest

from ctlib_gb300.workloads import FAN_EA, FAN_ED, fan_options, para_options
from test_geometry_host import _query, native  # noqa: F401


def _fan(scan, ratio, W, H, V=16, D=90):
    r = ratio * max(W, H)
    half = min(0.75, math.asin(min(0.99, 0.71 / ratio)))
    d = 2 * 1.8 * r * math.tan(half) / D if scan == FAN_ED else 2 * half / D
    return fan_options(V, D, W, H, 1.0, d, 0.0, 2 * math.pi / V, r, 0.8 * r, 0.0, scan)


@pytest.mark.parametrize("opts", [_fan(scan, ratio, 96, 96) for scan in (FAN_ED, FAN_EA)
                                  for ratio in (4.0, 1.0, 0.75, 0.72)] + [
    _fan(FAN_ED, 1.0, 1, 1), _fan(FAN_ED, 0.8, 2, 65), _fan(FAN_EA, 30.0, 100, 1),
    para_options(12, 40, 33, 47, 1.0, 1.3, 0.1, math.pi / 12, 0.2), para_options(3, 2, 1, 1, 1.0, 5.0, 0.1, 1.0, 0.0)])
def test_unit_is_as_fine_as_a_double(native, opts):  # noqa: F811
    V, D, W, H = (int(x) for x in opts[:4])
    L = max(W, H)
    flags = _query(native, opts, 0, dtype=1).astype(int)
    lp = _query(native, opts, 3, dtype=1).reshape(V, L, 2)
    q = _query(native, opts, 9, dtype=1).reshape(V, L, 7)
    s = int(q[0, 0, 6])
    for v in range(V):
        nl, K = (H, W) if flags[v] & 1 else (W, H)
        for l in range(nl):
            ah, al, sh, sl, sf, af = (int(x) for x in q[v, l, :6])
            alpha, sigma = (float(x) for x in lp[v, l])
            an, ad = alpha.as_integer_ratio()
            sn, sd = sigma.as_integer_ratio()
            extent = max(abs(alpha), abs(alpha + sigma * K))
            for k in (0, 1, K // 2, K):
                got = (ah << 32) + al + ((sh << 32) + sl) * k + ((af + sf * k) >> 32)
                assert abs(got) <= 2 ** 62
                # got / 2^s - (alpha + sigma k), exactly, then rounded once
                num = got * ad * sd - ((an * sd + sn * k * ad) << s if s >= 0 else 0)
                err = abs(num) / (ad * sd) * 2.0 ** -s
                assert err <= max(2.0 ** -53 * extent, 2.0 ** -48 * sigma), (v, l, k)
