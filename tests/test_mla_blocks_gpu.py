"""The mma.sync attention's forms for few and for many CTAs (16 heads, or 32 with the next tile on its way) give the
same partials, those of a batch's rows bit for bit what the rows launched alone leave; the merged result (whose
kernels differ in the order of their sums) agrees with the oracle within the kernel's tolerance."""

from __future__ import annotations

import pytest
import torch

from conftest import rel_err
from oracle import dsa_oracle as O

pytestmark = pytest.mark.gpu

ATTN_TOL = 2e-2


# (a launch of more than 148 CTAs of 16 heads takes the 32-head form where H allows it)
@pytest.mark.parametrize("rows,H,topk,nsplit", [
    (10, 32, 1000, 8),   # two tiles per split, the last one short
    (10, 48, 1000, 8),   # heads of no whole 32-head blocks
    (3, 96, 700, 9),     # 96-key splits
    (19, 32, 64, 4),     # 16 keys per split
    (75, 32, 130, 1),    # one split, no partials; three tiles
    (75, 32, 64, 1),     # one tile
    (75, 32, 260, 1),    # five tiles: both buffers are refilled, the last tile is short
    (75, 32, 330, 1),    # six
    (75, 32, 420, 1),    # seven
    (5, 32, 330, 2),     # five heads' CTAs, merges of two splits
])
@pytest.mark.parametrize("fp8", [False, True])
def test_batch_leaves_the_rows_partials(rows, H, topk, nsplit, fp8):
    from dsa_multi_layer_indexer_b200 import _lib, ops

    g = torch.Generator().manual_seed(rows * H + topk)
    n = 1500
    q = torch.randn(rows, H, 576, generator=g).to(torch.bfloat16)
    lat = torch.randn(n, 576, generator=g)
    kv = O.pack_fp8_latent(lat) if fp8 else lat.to(torch.bfloat16)
    kv_ref = O.unpack_fp8_latent(kv) if fp8 else kv
    idx = torch.stack([torch.randperm(n, generator=g)[:topk] for _ in range(rows)]).int()
    idx[:, 3::17] = -1
    idx[0, topk // 3:] = -1  # splits and tiles without a visible key
    lens = torch.full((rows,), n, dtype=torch.int32)
    lens[-1] = 11
    dev = [t.cuda() for t in (q, kv, idx, lens)]
    sm = 192 ** -0.5
    many = ops.MlaScratch(rows, H, nsplit, "cuda")
    both = ops.sparse_mla_decode(dev[0], dev[1], dev[2], sm, dev[3], rows_per_seq=rows, nsplit=nsplit, scratch=many).cpu()
    direct = ops.sparse_mla_decode(dev[0], dev[1], dev[2], sm, dev[3], rows_per_seq=rows, nsplit=nsplit).cpu()
    assert rel_err(direct.float(), both.float()) < 1e-5  # (one split: written without partials, else the same launches)
    for r in sorted({0, 1, rows // 2, rows - 1}):
        few = ops.MlaScratch(1, H, nsplit, "cuda")
        one = ops.sparse_mla_decode(dev[0][r:r + 1], dev[1], dev[2][r:r + 1].contiguous(), sm, dev[3][r:r + 1], nsplit=nsplit,
                                    scratch=few).cpu()
        assert torch.equal(few.acc[0], many.acc[r]) and torch.equal(few.m[0], many.m[r]) and torch.equal(few.l[0], many.l[r])
        ref = O.sparse_mla_decode(q[r:r + 1], kv_ref, idx[r:r + 1], [int(lens[r])], sm)
        for got in (both[r:r + 1], one):
            assert rel_err(got.float(), ref) < ATTN_TOL
    _lib.check_device_status()
