"""GPU tests of what the native half of the tensor entry points accepts, refuses and raises."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from dsa_multi_layer_indexer_b200 import _lib, ops as _ops

    yield _ops
    _lib.check_device_status()


def test_an_allocation_that_does_not_fit_raises_torchs_own_error(ops):
    """What serving loops catch to retry with a smaller batch; nothing is launched."""
    R, n = 65535, 1 << 20  # 275 GB of logits
    q = torch.zeros(R, 1, 16, device="cuda")
    k = torch.zeros(1, n, 16, device="cuda")
    with pytest.raises(torch.cuda.OutOfMemoryError):
        ops.indexer_scan_f32(q, torch.zeros(R, 1, device="cuda"), k, rows_per_seq=R)


def test_torchs_argument_errors_keep_their_class(ops):
    scalar = torch.zeros((), device="cuda")
    with pytest.raises(IndexError):
        ops.rmsnorm(scalar, torch.ones(1, device="cuda"), 1e-6)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_rows_without_elements_are_refused(ops, dtype):
    """An error, not a division by zero in the process."""
    import dsa_multi_layer_indexer_b200 as D

    refused = pytest.raises((ValueError, RuntimeError, ZeroDivisionError))
    x, w = torch.zeros(3, 0, device="cuda", dtype=dtype), torch.zeros(0, device="cuda", dtype=dtype)
    with refused:
        ops.rmsnorm(x, w, 1e-6)
    with refused:
        ops.add_rmsnorm(x, x, w, 1e-6)
    model = D.DSAModel(D.SMALL_CONFIG).eval().cuda()
    layer = model.layers[0]
    for b, s in ((1, 0), (0, 5)):
        empty = torch.zeros(b, s, D.SMALL_CONFIG.hidden_size, device="cuda")
        rope = model._build_rope(s, "cuda", torch.float32)
        with torch.no_grad():
            with refused:
                layer.indexer_indices(empty, rope)
            with refused:
                model(empty, D.ScheduleMode.BASELINE)
