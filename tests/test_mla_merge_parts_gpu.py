"""The merge of split partials: the same bits whether four, two or one CTA take a (row, head) pair's columns."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsplit", [2, 3, 4, 9, 33])
def test_one_row_has_the_same_bits_among_any_number_of_rows(nsplit):
    from dsa_multi_layer_indexer_b200 import _lib, ops

    # (1 and 2 rows: four CTAs a pair, 3: two, 4 and 9: one; 10, more pairs than SMs: one of its other form, up to 16 splits
    # a kernel that sums in another order)
    heads, most = 16, 10
    g = torch.Generator().manual_seed(nsplit)
    acc = torch.randn(most, nsplit, heads, 512, generator=g)
    m = 4 * torch.randn(most, nsplit, heads, generator=g)
    l = 1 + 60 * torch.rand(most, nsplit, heads, generator=g)
    m[:, nsplit - 1, ::3] = float("-inf")  # splits without a visible key
    m[0, :, 5] = float("-inf")             # a head without any
    acc[m == float("-inf")] = 0
    l[m == float("-inf")] = 0
    w = torch.exp2(m.double() - m.double().amax(1, keepdim=True)).nan_to_num(0)
    ref = (w[..., None] * acc.double()).sum(1) / (w * l.double()).sum(1).clamp(min=1e-300)[..., None]
    idx = torch.zeros(most, 64, dtype=torch.int32, device="cuda")
    q, kv = (torch.zeros(most, n, 576, dtype=torch.bfloat16, device="cuda") for n in (heads, 64))
    got = {}
    for rows in (1, 2, 3, 4, 9) + ((10,) if nsplit > 16 else ()):
        s = ops.MlaScratch(rows, heads, nsplit, "cuda")
        for buf, src in ((s.acc, acc), (s.m, m), (s.l, l)):
            buf.copy_(src[:rows])
        got[rows] = ops.sparse_mla_decode(q[:rows], kv[:rows], idx[:rows], 1.0, scratch=s, stage="combine").cpu()
        # fp32 sums of at most 33 terms, then one rounding to bf16
        assert (got[rows].double() - ref[:rows]).abs().max() < 2 ** -8 * ref.abs().max()
        assert torch.equal(got[rows][:1], got[1])
    assert torch.equal(got[3], got[9][:3]) and (10 not in got or torch.equal(got[10][:9], got[9]))
    assert not got[1][0, 5].any()
    _lib.check_device_status()
