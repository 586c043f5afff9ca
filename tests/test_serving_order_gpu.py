"""The serving entry runs its attention beside the top-k where that is safe: the results are those of the
separate modes, also where the incumbents are the very buffer that the selection is written to."""

from __future__ import annotations

import pytest
import torch

from test_serving_gpu import build_case, call

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,topk,cap,fp8", [(16, 512, 2048, False), (64, 512, 2048, True), (128, 2048, 4096, False)])
@pytest.mark.parametrize("mapped", [False, True])
def test_incumbents_that_are_the_selection_buffer(heads, topk, cap, fp8, mapped):
    from dsa_multi_layer_indexer_b200 import _lib, serving

    serving.clear_scratch()
    c = build_case(fp8, cap=cap, heads=heads, topk=topk, lens=[cap, cap - 300, cap - 7])
    kw = {} if mapped else {"pool_map": None}
    attn, nxt = call(c, **kw)
    assert torch.equal(attn, call(c, mode="attn_only", **kw))
    for _ in range(3):
        attn, nxt = call(c, **kw)
        own = {**c, "inc": nxt.clone()}
        want = call(own, mode="attn_only", **kw).clone()
        selected = nxt.clone()
        attn, again = call({**c, "inc": nxt}, **kw)  # reads and writes one buffer
        assert again.data_ptr() == nxt.data_ptr()
        assert torch.equal(attn, want) and torch.equal(again, selected)
        attn, again = call(own, **kw)
        assert torch.equal(attn, want) and torch.equal(again, selected)
    _lib.check_device_status()
