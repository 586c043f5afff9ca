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
