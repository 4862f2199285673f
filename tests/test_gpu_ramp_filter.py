"""fbp's ramp filter at the row lengths where it can go wrong: around a chunk of 16
bins, and up to the longest rows that a CTA's shared memory takes (the layout
without bank padding), with and without even taps.

Bound, pixel by pixel, with u = 2^-24 and Q the convolution of the absolute taps
with the absolute pre-weighted rows: a filtered value is a compensated sum of plain
sums of at most 16 products, so at most 20 u Q from exact; its backprojection adds
16 u of each term (8 * 2^-23, as in the image gather's tests). 40 u times the
backprojection of Q then covers the image, however much the ramp cancels. In fp64
the same with 2^-53, and at least 1e-12 of the image's norm for the coordinates."""

import math

import numpy as np
import pytest
import torch

from ctlib_gb300.workloads import FAN_ED, fan_options, para_options

pytestmark = pytest.mark.gpu


def _options(scan, V, dets, n):
    cell = 1.4 * n / dets
    if scan == 0:
        return fan_options(V, dets, n, n, 1.0, 1.6 * cell, 0.1, 2 * math.pi / V, 120.0, 72.0, 0.0, FAN_ED)
    return para_options(V, dets, n, n, 1.0, cell, 0.1, math.pi / V, 0.0)


def _absolute(y, opts, window):
    """Convolution of |taps| with |pre-weighted rows|."""
    D, scan = int(opts[1]), int(opts[-1])
    d = float(np.float32(opts[5]))
    pre = np.full(D, d)
    if scan == 0:
        d *= float(np.float32(opts[8])) / (float(np.float32(opts[8])) + float(np.float32(opts[9])))
        t = (np.arange(D) + 0.5 - D / 2) * d
        pre = d * opts[8] / np.hypot(opts[8], t)
    n = np.arange(-D, D + 1)
    h = np.where(n % 2 != 0, -1 / np.maximum(1e-300, (math.pi * n * d) ** 2), 0.0)
    h[D] = 1 / (4 * d * d)
    if window == "hann":
        h = 0.25 * np.roll(h, 1) + 0.5 * h + 0.25 * np.roll(h, -1)
    h = np.abs(h[1:-1])
    rows = np.abs(y.astype(np.float64)) * pre
    size = 1 << (3 * D).bit_length()
    q = np.fft.irfft(np.fft.rfft(rows, size) * np.fft.rfft(h, size), size)[..., D - 1:2 * D - 1]
    return np.maximum(q, 0)


@pytest.mark.parametrize("scan", [0, 2])
@pytest.mark.parametrize("dets,batch", [(1, 3), (15, 1), (16, 17), (17, 2), (33, 5), (2870, 16), (3550, 4), (11300, 1)])
@pytest.mark.parametrize("window", ["ram-lak", "hann"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_row_lengths(oracle_mod, scan, dets, batch, window, dtype):
    import ctlib_gb300 as ct
    if dtype == np.float64 and dets > 3550:
        pytest.skip("longer than a CTA takes in fp64")
    V, n = 5, 24
    opts = _options(scan, V, dets, n)
    o = torch.tensor(opts, dtype=torch.float64)
    y = np.random.default_rng(dets).uniform(0.5, 1.5, (batch, 1, V, dets)).astype(dtype)
    yd = torch.from_numpy(y).cuda()
    f32 = dtype == np.float32
    mode = oracle_mod.MODE_F64_ON_F32 if f32 else oracle_mod.MODE_F64
    got = ct.fbp(yd, o, filter=window)
    want = oracle_mod.fbp(y[-2:], opts, mode, filter=window)
    bound = oracle_mod.run("backprojection", _absolute(y[-2:], opts, window), opts, oracle_mod.MODE_F64)
    bound *= 40 * (2.0 ** -24 if f32 else 2.0 ** -53) * opts[7] / 2
    if not f32:
        bound += 1e-12 * np.linalg.norm(want)
    assert (np.abs(got[-2:].cpu().numpy() - want) <= bound).all()
    # one slice per thread, whose rows are laid out otherwise: the same bits
    assert torch.equal(ct.fbp(yd[-1:].contiguous(), o, filter=window), got[-1:])


def test_rows_too_long_are_refused():
    import ctlib_gb300 as ct
    opts = para_options(3, 11400, 24, 24, 1.0, 0.003, 0.1, math.pi / 3, 0.0)
    y = torch.zeros(1, 1, 3, 11400, device="cuda")
    with pytest.raises(RuntimeError, match="ramp filter smem"):
        ct.fbp(y, torch.tensor(opts, dtype=torch.float64))
    assert torch.isfinite(ct.backprojection(y, torch.tensor(opts, dtype=torch.float64))).all()
