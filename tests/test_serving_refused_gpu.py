"""A serving call whose attention refuses its operands raises before anything is launched: the selection that the
call before it returned stays, and the next call is right."""

from __future__ import annotations

import pytest
import torch

from test_serving_gpu import build_case, call

pytestmark = pytest.mark.gpu


def _misaligned(t):
    raw = torch.zeros(t.numel() * t.element_size() + 16, dtype=torch.uint8, device="cuda")
    v = raw[8:8 + t.numel() * t.element_size()]
    v.copy_(t.cuda().contiguous().view(torch.uint8).view(-1))
    return v.view(t.dtype).view(t.shape)


@pytest.mark.parametrize("what", ["strided pool", "misaligned pool", "empty pool", "fp16 queries", "no scale"])
def test_refused_call_leaves_the_selection(what):
    from dsa_multi_layer_indexer_b200 import _lib, serving

    serving.clear_scratch()
    c = build_case(True, heads=16)
    nxt = call(c)[1]
    before = nxt.clone()
    other = {**c, "iq8": c["iq8"].flip(0).contiguous(), "wp": c["wp"].flip(0).contiguous()}  # (another selection)
    scale = 192 ** -0.5
    pool = c["kv_pool"].cuda()
    q = c["q"].cuda()
    if what == "strided pool":
        wide = torch.zeros(pool.shape[0], 1312, dtype=torch.uint8, device="cuda")
        wide[:, :656] = pool
        pool = wide[:, :656]
    elif what == "misaligned pool":
        pool = _misaligned(pool)
    elif what == "empty pool":
        pool = pool[:0]
    elif what == "fp16 queries":
        q = q.half()
    elif what == "no scale":
        scale = None
    d = lambda t: t.cuda().contiguous()
    with pytest.raises(Exception):
        serving.fused_hide_decode_paged(q, pool, d(c["inc"]), d(other["iq8"]), d(other["wp"]), d(c["pages"]), d(c["pt"]),
                                        d(torch.tensor(c["lens"], dtype=torch.int32)), c["cap"], scale, d(c["pos2slot"]))
    torch.cuda.synchronize()
    assert torch.equal(nxt, before)
    want = call(c, mode="attn_only").clone()
    attn, again = call(c)
    assert torch.equal(attn, want) and torch.equal(again, before)
    _lib.check_device_status()
