"""GPU tests of the single-split attention that writes its result without partials, and of the tile
count that stops at a list's last visible key: both must give bit for bit what the partials + merge
launches give (the merge of one split multiplies by 2^0 and divides by the same sum)."""

from __future__ import annotations

import pytest
import torch

from conftest import rel_err
from oracle import dsa_oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from dsa_multi_layer_indexer_b200 import _lib, ops as _ops

    _lib.lib()
    yield _ops
    _lib.check_device_status()


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("H,rows", [(16, 3), (48, 2), (64, 130), (128, 66)])  # mma.sync kernel, tcgen05 kernel
def test_one_split_equals_partials_and_merge(ops, H, rows, fp8):
    torch.manual_seed(H + rows)
    n, topk, sm = 700, 200, 192 ** -0.5
    q = torch.randn(rows, H, 576, device="cuda").to(torch.bfloat16)
    kvf = torch.randn(n, 576)
    kv = (O.pack_fp8_latent(kvf) if fp8 else kvf.to(torch.bfloat16)).cuda().unsqueeze(0).contiguous()
    idx = torch.stack([torch.randperm(n)[:topk] for _ in range(rows)]).int()
    for r in range(rows):  # lists that end at every place of a tile, and holes in the middle
        idx[r, (r * 7) % (topk + 1):] = -1 if r % 2 else n + 3
        idx[r, 3::11] = -1
    lens = torch.tensor([n if r % 3 else n // 2 for r in range(rows)], dtype=torch.int32, device="cuda")
    idx = idx.cuda()
    one = ops.sparse_mla_decode(q, kv, idx, sm, lens, rows_per_seq=rows, nsplit=1)
    scratch = ops.MlaScratch(rows, H, 1, "cuda")
    ops.sparse_mla_decode(q, kv, idx, sm, lens, rows_per_seq=rows, nsplit=1, scratch=scratch, stage="partials")
    two = ops.sparse_mla_decode(q, kv, idx, sm, lens, rows_per_seq=rows, nsplit=1, scratch=scratch, stage="combine")
    assert torch.equal(one, two)
    assert float(one[0].float().abs().max()) == 0.0  # an all-padding list
    split = ops.sparse_mla_decode(q, kv, idx, sm, lens, rows_per_seq=rows, nsplit=4)
    assert rel_err(one.float().cpu(), split.float().cpu()) < 2e-2
    ref_kv = O.unpack_fp8_latent(kv[0].cpu()) if fp8 else kv[0].cpu()
    for r in (1, rows - 1):
        ref = O.sparse_mla_decode(q[r:r + 1].cpu(), ref_kv, idx[r:r + 1].cpu(), [int(lens[r])], sm)
        assert rel_err(one[r:r + 1].float().cpu(), ref) < 2e-2


@pytest.mark.parametrize("H", [16, 64])
def test_one_split_dense_rows_of_a_prompt(ops, H):
    torch.manual_seed(3)
    s, sm = 150, 0.07
    q = torch.randn(s, H, 576, device="cuda").to(torch.bfloat16)
    kv = torch.randn(1, s + 9, 576, device="cuda").to(torch.bfloat16)
    lens = torch.arange(1, s + 1, dtype=torch.int32, device="cuda")
    got = ops.sparse_mla_decode(q, kv, None, sm, lens, rows_per_seq=s, dense_keys=s, nsplit=1)
    for r in (0, 63, 64, s - 1):
        ref = O.dense_mla_decode(q[r:r + 1].cpu(), kv[0].cpu(), [r + 1], sm)
        assert rel_err(got[r:r + 1].float().cpu(), ref) < 2e-2


@pytest.mark.parametrize("H,rows", [(16, 3), (64, 130)])  # mma.sync kernel, tcgen05 kernel
@pytest.mark.parametrize("beside", [False, True])
def test_partials_that_a_caller_hands_over_are_written(ops, H, rows, beside):
    """One split writes its result at once only where there is nothing else to write."""
    from dsa_multi_layer_indexer_b200 import kernels_ext

    torch.manual_seed(H)
    n, topk, sm = 300, 128, 192 ** -0.5
    q = torch.randn(rows, H, 576, device="cuda").to(torch.bfloat16)
    kv = torch.randn(1, n, 576, device="cuda").to(torch.bfloat16)
    idx = torch.stack([torch.randperm(n)[:topk] for _ in range(rows)]).int().cuda()
    want, got = (ops.MlaScratch(rows, H, 1, "cuda") for _ in range(2))
    ops.sparse_mla_decode(q, kv, idx, sm, rows_per_seq=rows, nsplit=1, scratch=want, stage="partials")
    for s in (got.acc, got.m, got.l):
        s.fill_(float("nan"))
    out = ops.sparse_mla_decode(q, kv, idx, sm, rows_per_seq=rows, nsplit=1, scratch=got, beside_previous=beside)
    for a, b in ((got.acc, want.acc), (got.m, want.m), (got.l, want.l)):
        assert torch.equal(a, b)
    assert torch.equal(out, ops.sparse_mla_decode(q, kv, idx, sm, rows_per_seq=rows, nsplit=1))
    acc, m, l = kernels_ext.alloc_part(rows, H, 1, "cuda")  # the extension's own output arguments
    kernels_ext.build().launch_fused_sparse_splitk(q, kv[0], idx, None, None, None, None, acc, m, l, None, None, out, rows, n, H, 16, topk,
                                                   1, sm, 0, 1, 0)
    assert float(l.min()) > 0 and float(acc.abs().sum()) > 0
