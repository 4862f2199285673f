"""What the autotuner times and how its cache is keyed (no GPU needed)."""

import pytest
import torch

from ctlib_gb300 import _native as N
from ctlib_gb300 import tune


@pytest.mark.parametrize("op", range(6))
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("batch", [1, 2, 3, 5, 16, 40])
def test_no_two_schedules_are_the_same_kernel(op, dtype, batch):
    f32, image = dtype == torch.float32, op not in (N.OP_PROJECTION, N.OP_BACKPROJECTION_T)
    got = tune.schedules(dtype, op, batch)
    effective = set()
    for cap, warps, steps in got:
        sb = 1
        while sb < batch and sb < min(cap, 16 if f32 else 4):
            sb *= 2
        built = f32 and image and sb <= 2  # both step counts exist
        assert steps in ((2, 3) if built else (0,))
        effective.add((sb, warps, steps))
    assert len(effective) == len(got) >= 2


def test_cache_entries_of_other_kernels_are_not_used(tmp_path, monkeypatch):
    class Plan:
        device, dtype, values = 0, torch.float32, (1.0, 2.0)

    class Ragged:
        device, dtype, plans = 0, torch.float32, (Plan(),)

    src = tmp_path / "kernels.cu"
    src.write_text("one")
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda d: "GPU")
    monkeypatch.setattr(N, "SOURCES", [str(src)])
    monkeypatch.setattr(N, "HEADERS", [])
    keys = []
    for text in ("one", "one", "two"):
        src.write_text(text)
        tune._kernels.cache_clear()
        keys.append((tune._key(Plan(), 0, 4), tune._ragged_key(Ragged(), ("fbp",))))
    tune._kernels.cache_clear()
    assert keys[0] == keys[1]
    assert keys[0][0] != keys[2][0] and keys[0][1] != keys[2][1]
