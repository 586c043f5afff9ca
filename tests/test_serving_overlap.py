"""When two contiguous tensors share memory, as the serving entry asks before it reorders its launches (CPU)."""

from __future__ import annotations

import torch

from dsa_multi_layer_indexer_b200 import serving


def test_overlap():
    whole = torch.zeros(8, 16, dtype=torch.int32)
    other = torch.zeros(8, 16, dtype=torch.int32)
    assert serving._overlap(whole, whole) and serving._overlap(whole[2:5], whole[4:])
    assert serving._overlap(whole[3:4], whole) and serving._overlap(whole.view(torch.uint8), whole[7:])
    assert not serving._overlap(whole[:4], whole[4:]) and not serving._overlap(whole[4:], whole[:4])
    assert not serving._overlap(whole, other)
