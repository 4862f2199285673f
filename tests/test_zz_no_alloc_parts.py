"""ctgb_projection_noalloc on a batch of small images: accepted by the bytes of its
unpadded lines, and run in parts, since with their padding they do not fit the
static array. The same bits as ctgb_projection, whose parts end elsewhere."""

import ctypes
import math

import pytest
import torch

from ctlib_gb300.workloads import FAN_ED, fan_options

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_parts_of_a_batch(dtype):
    import ctlib_gb300 as ct
    from ctlib_gb300 import _native as N
    V, D, W, H = 5, 12, 8, 8
    # unpadded: 2 x 64 pixels a slice, up to 64 MiB; a shorter last part
    batch = (64 << 20) // (2 * 64 * dtype.itemsize) - 16 * 3 - 5
    o = torch.tensor(fan_options(V, D, W, H, 1.0, 1.6, 0.1, 2 * math.pi / V, 64.0, 48.0, 0.2, FAN_ED),
                     dtype=torch.float64)
    x = torch.randn(batch, 1, H, W, generator=torch.Generator().manual_seed(9), dtype=dtype).cuda()
    plan = ct.get_plan(o, dtype, x.device)
    # the array holds 72 MiB: the padded batch takes more
    assert plan.workspace_bytes(N.OP_PROJECTION, batch) > 72 << 20
    out = torch.full((batch, 1, V, D), float("nan"), dtype=dtype, device="cuda")
    rc = N.lib().ctgb_projection_noalloc(plan.handle, ctypes.c_void_p(x.data_ptr()), ctypes.c_void_p(out.data_ptr()),
                                         batch, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == N.OK, N.last_error()
    assert torch.equal(out, ct.projection(x, o))
