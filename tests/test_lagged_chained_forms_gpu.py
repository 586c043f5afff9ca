"""The attention enqueued behind scan and top-k and running beside the top-k, in each of the forms that a launch's size
selects: bit for bit what it returns when nothing runs beside it, and that within the kernel's tolerance of the oracle."""

from __future__ import annotations

import pytest
import torch

from conftest import rel_err
from oracle import dsa_oracle as O

pytestmark = pytest.mark.gpu

ATTN_TOL = 2e-2
SM = 192 ** -0.5


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("rows,heads,ctx,topk,nsplit,forms", [  # (forms: over bf16 rows and fp8 rows)
    (1, 128, 20000, 2048, None, (0, 2)),  # one tile per split: 16 heads per CTA, fp8 rows 32
    (10, 32, 6000, 2048, None, (1, 1)),   # 32 heads per CTA, three tiles per split
    (80, 32, 3000, 256, 1, (1, 1)),       # the same without partials, four tiles
    (80, 32, 3000, 64, 1, (0, 2)),        # one tile
    (10, 48, 6000, 2048, None, (0, 0)),   # 16 heads per CTA, two CTAs on an SM
    (4, 128, 6000, 2048, None, (3, 3)),   # tcgen05
    (80, 64, 3000, 256, 1, (3, 3)),       # tcgen05 without partials
    (14, 128, 6000, 2048, None, (4, 3)),  # pairs of CTAs, bf16 rows
    (80, 128, 3000, 256, 1, (4, 3)),      # the same without partials, two rows for some pairs
    (40, 128, 3000, 256, 2, (4, 3)),      # the same, splits of one tile
])
def test_beside_the_topk_equals_alone(rows, heads, ctx, topk, nsplit, forms, fp8):
    from dsa_multi_layer_indexer_b200 import _lib, ops
    from dsa_multi_layer_indexer_b200.decode import HotPathState, LayerCache

    g = torch.Generator(device="cuda").manual_seed(rows + heads + topk)
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=g)
    st = HotPathState(rows, heads, 64, ctx, topk, "cuda", nsplit=nsplit)
    beside = 1 | 2 | 8  # a list, lengths, beside the kernel in front
    assert _lib.lib().dsa_sparse_mla_form(rows, 1, heads, topk, st.nsplit, SM, ctx, fp8, beside) == forms[fp8]
    k8, ks = ops.quantize_e4m3_rowwise(rand(rows, ctx, 128))
    lat = rand(rows * ctx, 576)
    kv = O.pack_fp8_latent(lat.cpu()).cuda() if fp8 else lat.to(torch.bfloat16)
    kv_ref = O.unpack_fp8_latent(kv.cpu()) if fp8 else kv.cpu()
    cache = LayerCache(k8.view(torch.uint8), ks, kv.view(rows, ctx, -1))
    q8, sq = ops.quantize_e4m3_rowwise(rand(rows, 64, 128))
    st.index_q.copy_(q8.view(torch.uint8))
    st.index_w.copy_(sq * rand(rows, 64) / 8)
    st.q.copy_(rand(rows, heads, 576).to(torch.bfloat16))
    st.seq_lens.copy_(torch.randint(topk, ctx + 1, (rows,), device="cuda", generator=g).int())
    attend = torch.stack([torch.randperm(ctx, device="cuda", generator=g)[:topk] for _ in range(rows)]).int()
    selected = st.run_indexer(cache).clone()
    want = st.run_attention(cache, attend, SM).clone()
    for r in (0, rows - 1):
        ref = O.sparse_mla_decode(st.q[r:r + 1].cpu(), kv_ref.view(rows, ctx, 576)[r], attend[r:r + 1].cpu(), [int(st.seq_lens[r])], SM)
        assert rel_err(want[r:r + 1].float().cpu(), ref) < ATTN_TOL

    def check():
        assert torch.equal(st.indices, selected) and torch.equal(st.out, want)

    for _ in range(3):
        st.indices.fill_(-1)
        st.out.fill_(float("nan"))
        st.run_lagged_chained(cache, attend, SM)
        check()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(3):
            st.run_lagged_chained(cache, attend, SM)
    st.indices.fill_(-1)
    st.out.fill_(float("nan"))
    graph.replay()
    check()
    _lib.check_device_status()
