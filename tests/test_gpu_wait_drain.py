"""Staged gathers with every wait given up at once. Waits run out, some warps of a
CTA finish on global loads while others still read the ring, and a slot may be
refilled only when those have left it. And where all copies fit the ring, the
producer has issued them before any warp looks: it must wait for them all the
same, or the CTA could end, and its shared memory pass to the next one, with
copies still landing. Every bit stays."""

import math

import pytest
import torch

from ctlib_gb300.workloads import FAN_EA, FAN_ED, fan_options

pytestmark = pytest.mark.gpu

SIZES = [  # views, dets, width, height: lines that fill one slot, two, and a third in part; views of one slot and more
    (400, 96, 7, 8), (400, 96, 14, 16), (400, 96, 19, 15), (3, 96, 200, 190), (9, 64, 128, 96),
    (400, 160, 96, 80),  # several rings
]


def _runs(op, opts, x, shape, times=6):
    """Results at the default limit and at a limit of 0, and the waits that ran out at 0."""
    from ctlib_gb300 import _native as N
    from ctlib_gb300.ops import Plan
    plan = Plan(tuple(opts), torch.float32, 0)
    want = torch.empty(shape, device="cuda")
    torch.cuda.synchronize()
    N.wait_timeouts(0, reset=True)
    try:
        plan.run(op, x, want)
        torch.cuda.synchronize()
        assert N.wait_timeouts(0) == 0
        N.check(N.lib().ctgb_plan_set_wait_limit(plan.handle, 0), "wait limit")
        outs = [torch.full(shape, float("nan"), device="cuda") for _ in range(times)]
        for out in outs:
            plan.run(op, x, out)
        torch.cuda.synchronize()
        for out in outs:
            assert torch.equal(out, want), op
        return N.wait_timeouts(0)
    finally:
        N.wait_timeouts(0, reset=True)


@pytest.mark.parametrize("op", [0, 3])
@pytest.mark.parametrize("batch", [8, 16])
def test_detector_gather_stages_its_lines(op, batch):
    """512 lines through rings of 16 to 24: waits run out at a limit of 0."""
    opts = fan_options(1152, 736, 512, 512, 0.6641, 1.2858, 0.0, 2 * math.pi / 1152, 595.0, 490.6, 0.0, FAN_ED)
    x = torch.randn(batch, 1, 512, 512, generator=torch.Generator().manual_seed(5)).cuda()
    assert _runs(op, opts, x, (batch, 1, 1152, 736), 2) > 0


@pytest.mark.parametrize("scan", [FAN_ED, FAN_EA])
@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("batch", [8, 16])
def test_no_copy_outlives_its_cta(scan, size, batch):
    V, D, W, H = size
    # a detector that covers the image, cells of a pixel or less
    r = 8.0 * max(W, H)
    pitch = 1.5 * max(W, H) / D
    d = pitch / r if scan == FAN_EA else 1.6 * pitch
    opts = fan_options(V, D, W, H, 1.0, d, 0.1, 2 * math.pi / V, r, 0.6 * r, 0.0, scan)
    g = torch.Generator().manual_seed(V + W)
    img = torch.randn(batch, 1, H, W, generator=g).cuda()
    sino = torch.randn(batch, 1, V, D, generator=g).cuda()
    for op in (0, 1, 2, 3, 4):
        det = op in (0, 3)
        _runs(op, opts, img if det else sino, (batch, 1) + ((V, D) if det else (H, W)))
