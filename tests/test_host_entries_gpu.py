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


def test_what_int_converts_is_taken(ops):
    """The arguments that the entry points convert themselves: floats and one-element tensors of whole numbers."""
    torch.manual_seed(0)
    iq, _ = ops.quantize_e4m3_rowwise(torch.randn(2, 16, 128, device="cuda"))
    ik, ks = ops.quantize_e4m3_rowwise(torch.randn(2, 96, 128, device="cuda"))
    iw = torch.randn(2, 16, device="cuda")
    want = ops.indexer_scan_fp8(iq, iw, ik, ks, ctx=64)
    for ctx in (64.0, torch.tensor(64), torch.tensor(64.0)):
        assert torch.equal(ops.indexer_scan_fp8(iq, iw, ik, ks, ctx=ctx), want)
    out = torch.empty(2, 8, dtype=torch.int32, device="cuda")
    ref = ops.topk_select(want, 8, torch.tensor([3, 64], dtype=torch.int32, device="cuda"), pad_value=-7, index_offset=5)
    got = ops.topk_select(want, 8.0, torch.tensor([3, 64], dtype=torch.int32, device="cuda"), pad_value=-7.0, index_offset=5.0, out_idx=out)
    assert torch.equal(got, ref)
    q, kv = torch.randn(2, 16, 576, device="cuda").bfloat16(), torch.randn(2, 96, 576, device="cuda").bfloat16()
    assert torch.equal(ops.sparse_mla_decode(q, kv, None, 0.1, dense_keys=64.0), ops.sparse_mla_decode(q, kv, None, 0.1, dense_keys=64))
    for bad in ("x", object(), [64]):
        with pytest.raises((TypeError, ValueError)):
            ops.topk_select(want, 8, index_offset=bad)


def test_fp32_entries_take_buffers_of_more_rows(ops):
    """Buffers sized for the largest batch: only the rows of this call are read and written."""
    torch.manual_seed(1)
    q, w, k = torch.randn(3, 4, 20, device="cuda"), torch.randn(7, 4, device="cuda"), torch.randn(3, 50, 20, device="cuda")
    out = torch.full((5, 52), 9.0, device="cuda")
    got = ops.indexer_scan_f32(q, w, k, out=out)
    assert got.shape == (5, 50) and torch.equal(got[:3], ops.indexer_scan_f32(q, w[:3].contiguous(), k)) and bool((out[3:] == 9).all())
    a, kv = torch.randn(3, 4, 20, device="cuda"), torch.randn(3, 50, 20, device="cuda")
    idx = torch.randint(0, 50, (6, 11), dtype=torch.int32, device="cuda")
    assert torch.equal(ops.sparse_mla_f32(a, kv, idx, 16, 0.1), ops.sparse_mla_f32(a, kv, idx[:3].contiguous(), 16, 0.1))
    with pytest.raises(ValueError):
        ops.sparse_mla_f32(a, kv, idx[:2].contiguous(), 16, 0.1)
