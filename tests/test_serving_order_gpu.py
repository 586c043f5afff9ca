"""The serving entry runs its attention behind scan and top-k, beside the top-k, unless the incumbents are the very
buffer that the selection is written to: then in front of them. The results are those of the separate modes."""

from __future__ import annotations

import pytest
import torch

from test_serving_gpu import build_case, call

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,topk,cap,fp8", [(16, 512, 2048, False), (64, 512, 2048, True), (128, 2048, 4096, False)])
@pytest.mark.parametrize("mapped", [False, True])
def test_incumbents_that_are_the_selection_buffer(heads, topk, cap, fp8, mapped, monkeypatch):
    from dsa_multi_layer_indexer_b200 import _lib, ops, serving

    order = []

    def noted(name, fn):
        def f(*a, **kw):
            order.append((name, kw.get("beside_previous", False)))
            return fn(*a, **kw)
        return f

    for name, what in (("sparse_mla_decode", "attention"), ("indexer_scan_fp8_paged", "scan"), ("topk_select", "select"),
                       ("topk_select_paged", "select")):
        monkeypatch.setattr(ops, name, noted(what, getattr(ops, name)))
    serving.clear_scratch()
    c = build_case(fp8, cap=cap, heads=heads, topk=topk, lens=[cap, cap - 300, cap - 7])
    kw = {} if mapped else {"pool_map": None}
    old = c["inc"].cuda()
    attn, nxt = call(c, **kw)  # (plan buffers)
    selected = nxt.clone()
    assert not torch.equal(old, selected)
    want = call(c, mode="attn_only", **kw).clone()
    over_selected = call({**c, "inc": selected}, mode="attn_only", **kw).clone()
    assert not torch.equal(want, over_selected)
    for _ in range(3):
        for aliased in (True, False):
            nxt.copy_(old)
            attn.fill_(float("nan"))
            order.clear()
            got, again = call({**c, "inc": nxt if aliased else old.clone()}, **kw)
            assert again.data_ptr() == nxt.data_ptr() and got.data_ptr() == attn.data_ptr()
            assert torch.equal(got, want) and torch.equal(again, selected)
            assert order == ([("attention", False), ("scan", False), ("select", False)] if aliased else
                             [("scan", False), ("select", False), ("attention", True)])
    _lib.check_device_status()


def test_attention_goes_first_where_the_lists_share_memory():
    from dsa_multi_layer_indexer_b200 import ops

    q, kv = (torch.zeros(n, 16, 576, dtype=torch.bfloat16, device="cuda") for n in (8, 1))
    last = lambda a, b: ops.attention_last(q, kv[0], a, 1.0, b, None, 64)
    whole, other = (torch.zeros(8, 16, dtype=torch.int32, device="cuda") for _ in range(2))
    assert not last(whole, whole) and not last(whole[2:5], whole[4:]) and not last(whole[4:], whole[2:5])
    assert not last(whole[3:4], whole) and not last(whole, whole[7:])
    assert last(whole[:4], whole[4:]) and last(whole[4:], whole[:4]) and last(whole, other)
