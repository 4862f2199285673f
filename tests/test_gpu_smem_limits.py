"""A kernel's shared-memory limit is shared by every plan, thread and ragged batch:
calls whose launches need different sizes must not take it from one another."""

import math
import threading

import pytest
import torch

from ctlib_gb300.workloads import FAN_ED, fan_options, para_options

pytestmark = pytest.mark.gpu


def test_a_smaller_ragged_batch_leaves_a_larger_one_its_limit():
    from ctlib_gb300.batched import RaggedBatch

    def batch(D):  # rows of D bins: 88 and 66 KB of taps and inputs
        return RaggedBatch([para_options(4, D, 16, 16, 1.0, 32.0 / D, 0.0, math.pi / 4, 0.0)])

    y = torch.randn(1, 1, 4, 4000, generator=torch.Generator().manual_seed(1)).cuda()
    large = batch(4000)
    (want,) = large.fbp([y])
    small = batch(3000)
    small.fbp([torch.ones(1, 1, 4, 3000, device="cuda")])
    (got,) = large.fbp([y])
    assert torch.equal(got, want)


@pytest.mark.parametrize("op", [0, 1])
def test_threads_with_other_warps_per_cta(op):
    """Both gathers of 8 slices, 8 warps per CTA in one thread and 4 in the other."""
    from ctlib_gb300 import _native as N
    from ctlib_gb300.ops import Plan
    opts = fan_options(16, 32, 16, 16, 1.0, 2.0, 0.0, 2 * math.pi / 16, 120.0, 100.0, 0.0, FAN_ED)
    img, sino = (8, 1, 16, 16), (8, 1, 16, 32)
    x = torch.randn(img if op == 0 else sino, generator=torch.Generator().manual_seed(2)).cuda()
    errors = []

    def work(warps):
        try:
            plan = Plan(tuple(opts), torch.float32, 0)
            N.check(N.lib().ctgb_plan_set_schedule(plan.handle, op, 8, warps), "schedule")
            out = torch.empty(sino if op == 0 else img, device="cuda")
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(4000):
                    plan.run(op, x, out)
        except Exception as e:  # reported by the main thread
            errors.append(f"{warps} warps: {e}")

    threads = [threading.Thread(target=work, args=(w,)) for w in (8, 4, 8, 4)]
    torch.cuda.synchronize()
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors
