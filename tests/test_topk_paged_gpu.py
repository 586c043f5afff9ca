"""GPU tests of the top-k that emits cache slots of 64-token pages (dsa_topk_select_paged): exactly the
positions of dsa_topk_select, mapped through the page table, for rows that take one CTA, a cluster of
eight and a cluster of sixteen, short and ragged ones and rows with -inf among the selected."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,topk,rows", [(64, 16, 2), (1000, 2048, 3), (16384, 512, 2), (16448, 2048, 5), (131072, 2048, 2),
                                         (200000, 2048, 1)])
def test_slots_equal_mapped_positions(n, topk, rows):
    from dsa_multi_layer_indexer_b200 import _lib, ops

    torch.manual_seed(n)
    pages = (n + 63) // 64 + 1
    iq, _ = ops.quantize_e4m3_rowwise(torch.randn(rows, 16, 128, device="cuda"))
    ik, ks = ops.quantize_e4m3_rowwise(torch.randn(rows, n, 128, device="cuda"))
    iw = torch.randn(rows, 16, device="cuda") / 8
    lens = torch.tensor([max(1, n - 37 * r * r) for r in range(rows)], dtype=torch.int32, device="cuda")
    ks[0, 3] = float("inf")  # a key whose logit is -inf or inf, whichever sign its sum has
    table = torch.randperm(rows * pages, device="cuda").int().view(rows, pages)
    hist = torch.zeros(rows, ops.HIST_BINS, dtype=torch.int32, device="cuda")
    logits = ops.indexer_scan_fp8(iq, iw, ik, ks, lens, hist=hist)
    kept = hist.clone()
    pos = ops.topk_select(logits, topk, lens, hist=hist)
    assert int(hist.abs().sum()) == 0
    hist.copy_(kept)
    slots = torch.full((rows, topk), -7, dtype=torch.int32, device="cuda")
    ops.topk_select_paged(logits, topk, lens, hist, table, slots)
    assert int(hist.abs().sum()) == 0  # re-armed
    safe = pos.clamp(min=0).long()
    want = torch.where(pos >= 0, table.gather(1, safe >> 6) * 64 + (pos & 63), pos)
    assert torch.equal(slots, want)
    _lib.check_device_status()


def test_rows_without_workspace_take_none_and_errors_are_raised():
    from dsa_multi_layer_indexer_b200 import ops

    x = torch.randn(2, 300, device="cuda")
    hist = torch.zeros(2, ops.HIST_BINS, dtype=torch.int32, device="cuda")
    out = torch.empty(2, 8, dtype=torch.int32, device="cuda")
    with pytest.raises(ValueError, match="cover"):
        ops.topk_select_paged(x, 8, None, hist, torch.zeros(2, 4, dtype=torch.int32, device="cuda"), out)
    with pytest.raises(ValueError, match="out_idx"):
        ops.topk_select_paged(x, 9, None, hist, torch.zeros(2, 5, dtype=torch.int32, device="cuda"), out)
    with pytest.raises(TypeError):
        ops.topk_select_paged(x, 8, None, "hist", torch.zeros(2, 5, dtype=torch.int32, device="cuda"), out)
    big = torch.randn(1, 300000, device="cuda")  # longer rows still get their scratch
    idx, val = ops.topk_select(big, 5, return_values=True)
    assert torch.equal(val.sort().values[0], big[0].topk(5).values.sort().values)
    assert torch.equal(idx[0].long(), big[0].topk(5).indices.sort().values)
