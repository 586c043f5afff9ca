"""GPU parity tests of the tcgen05 sparse MLA decode kernel (64-head CTAs, S and
O^T in tensor memory) against the CPU oracle and against the mma.sync kernel on
the same inputs. A launch runs on it by its size (128 tiles of 64 heads x 64 keys
or more, and not on pairs of CTAs); each test asserts that its launches do, and
gets the mma.sync kernel's result from launches of one row and 16 heads.
Tolerance: attention output <= 2e-2 relative (bf16)."""

from __future__ import annotations

import pytest
import torch

from conftest import corr_diff, rel_err
from oracle import dsa_oracle as O

pytestmark = pytest.mark.gpu

ATTN_TOL = 2e-2
MMA_SYNC, TC = 0, 3  # dsa_mla_form


@pytest.fixture(scope="module")
def ops():
    from dsa_multi_layer_indexer_b200 import _lib, ops as _ops

    _lib.lib()  # fail loudly if the library is missing
    yield _ops
    _lib.check_device_status()


def dev(t: torch.Tensor) -> torch.Tensor:
    return t.cuda().contiguous()


def decode(ops, form, q, kv, idx, sm, seq=None, nsplit=None, dense_keys=None):
    """One launch of independent sequences (or of rows over one cache), which runs on the kernel ``form``."""
    from dsa_multi_layer_indexer_b200 import _lib

    R, H, _ = q.shape
    rows_per_seq = 1 if kv.dim() == 3 else R
    topk = idx.shape[1] if idx is not None else dense_keys
    nsplit = nsplit or ops.default_nsplit(R, H, topk)
    flags = (1 if idx is not None else 0) | (2 if seq is not None else 0) | (4 if nsplit == 1 else 0)
    assert _lib.lib().dsa_sparse_mla_form(R, rows_per_seq, H, topk, nsplit, sm, kv.shape[-2], kv.dtype == torch.uint8, flags) == form
    out = ops.sparse_mla_decode(q, kv, idx, sm, seq, rows_per_seq=rows_per_seq, nsplit=nsplit, dense_keys=dense_keys).float().cpu()
    _lib.check_device_status()
    return out


def decode_mma_sync(ops, q, kv, idx, sm, seq=None, nsplit=4):
    R, H, _ = q.shape
    rows = []
    for r in range(R):
        mine = kv if kv.dim() == 2 else kv[r]
        rows.append(torch.cat([decode(ops, MMA_SYNC, q[r:r + 1, h:h + 16].contiguous(), mine, idx[r:r + 1].contiguous(), sm,
                                      None if seq is None else seq[r:r + 1].contiguous(), nsplit) for h in range(0, H, 16)], dim=1))
    return torch.cat(rows)


@pytest.mark.parametrize("R,H,topk,n,nsplit", [(128, 64, 64, 300, 1), (64, 64, 128, 4096, 1), (32, 64, 200, 1000, 3),
                                               (4, 128, 2048, 8192, 8), (4, 128, 2048, 3000, 5), (64, 64, 80, 100, 2),
                                               (6, 192, 512, 2000, 4), (74, 128, 65, 300, 1)])
def test_tc_matches_oracle_and_mma_sync(ops, R, H, topk, n, nsplit):
    torch.manual_seed(H + topk + nsplit)
    q = torch.randn(R, H, 576).to(torch.bfloat16)
    kv = torch.randn(n, 576).to(torch.bfloat16)
    idx = torch.full((R, topk), -1, dtype=torch.int32)
    take = min(topk, n)
    for r in range(R):
        idx[r, :take] = torch.randperm(n)[:take].int()
    idx[:, ::17] = n + 5  # entries beyond the sequence are skipped
    idx[:, 3::29] = -1    # and so is padding
    sm = 192 ** -0.5
    tc = decode(ops, TC, dev(q), dev(kv), dev(idx), sm, nsplit=nsplit)
    some = sorted({0, 1, R // 2, R - 1})
    legacy = decode_mma_sync(ops, dev(q[some]), dev(kv), dev(idx[some]), sm)
    for i, r in enumerate(some):
        ref = O.sparse_mla_decode(q[r:r + 1], kv, idx[r:r + 1], [n], sm)
        assert rel_err(tc[r:r + 1], ref) < ATTN_TOL
        assert corr_diff(tc[r:r + 1], ref) < 1e-3
        assert rel_err(tc[r:r + 1], legacy[i:i + 1]) < ATTN_TOL


def test_tc_ragged_batch_and_empty_rows(ops):
    torch.manual_seed(21)
    B, H, n, topk = 8, 64, 2500, 1024
    q = torch.randn(B, H, 576).to(torch.bfloat16)
    kv = torch.randn(B, n, 576).to(torch.bfloat16)
    lens = [2500, 1, 1300, 0, 64, 2499, 65, 700]
    idx = torch.stack([torch.randperm(n)[:topk] for _ in range(B)]).int()
    idx[4] = -1  # a row whose selection is all padding
    seq = dev(torch.tensor(lens, dtype=torch.int32))
    sm = 576 ** -0.5
    both = decode(ops, TC, dev(q), dev(kv), dev(idx), sm, seq, nsplit=4)
    assert torch.isfinite(both).all()
    assert float(both[3].abs().max()) == 0.0 and float(both[4].abs().max()) == 0.0
    for b in range(B):
        one = decode(ops, TC, *(dev(t[b:b + 1].expand(B, *t.shape[1:])) for t in (q, kv, idx)), sm, dev(seq[b:b + 1].expand(B)),
                     nsplit=4)
        assert torch.equal(one[0], both[b])  # a row does not depend on its batch
        if lens[b] > 0 and b != 4:
            ref = O.sparse_mla_decode(q[b:b + 1], kv[b], idx[b:b + 1], [lens[b]], sm)
            assert rel_err(both[b:b + 1], ref) < ATTN_TOL


@pytest.mark.parametrize("nsplit", [1, 3])
def test_tc_dense_mode(ops, nsplit):
    torch.manual_seed(22)
    B, H, n = 12, 64, 700
    q = torch.randn(B, H, 576).to(torch.bfloat16)
    kv = torch.randn(B, n, 576).to(torch.bfloat16)
    lens = [650, 700, 1, 63, 64, 65, 128, 400, 699, 300, 449, 511]
    seq = dev(torch.tensor(lens, dtype=torch.int32))
    got = decode(ops, TC, dev(q), dev(kv), None, 0.07, seq, nsplit=nsplit, dense_keys=n)
    for b in range(B):
        ref = O.dense_mla_decode(q[b:b + 1], kv[b], [lens[b]], 0.07)
        assert rel_err(got[b:b + 1], ref) < ATTN_TOL


def test_tc_fp8_latent_rows(ops):
    torch.manual_seed(23)
    H, n, topk = 128, 3000, 2048
    q = torch.randn(2, H, 576).to(torch.bfloat16)
    rows = O.pack_fp8_latent(torch.randn(n, 576))
    idx = torch.stack([torch.randperm(n)[:topk] for _ in range(2)]).int()
    idx[:, ::13] = -1
    sm = 192 ** -0.5
    seq = dev(torch.tensor([n, n - 700], dtype=torch.int32))
    kv = dev(rows).unsqueeze(0).expand(2, -1, -1).contiguous()
    got = decode(ops, TC, dev(q), kv, dev(idx), sm, seq, nsplit=4)
    legacy = decode_mma_sync(ops, dev(q), kv, dev(idx), sm, seq)
    for b, ln in enumerate((n, n - 700)):
        ref = O.sparse_mla_decode(q[b:b + 1], O.unpack_fp8_latent(rows), idx[b:b + 1], [ln], sm)
        assert rel_err(got[b:b + 1], ref) < ATTN_TOL
        assert corr_diff(got[b:b + 1], ref) < 1e-3
    assert rel_err(got, legacy) < ATTN_TOL


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("nsplit", [1, 2])
@pytest.mark.parametrize("mult", [20.0, 80.0])
def test_tc_runaway_maximum_rescales(ops, mult, nsplit, fp8):
    """Keys late in the list have logits far above the first tile's maximum, which
    the kernel keeps as its softmax reference: the rescale of O^T must kick in."""
    torch.manual_seed(24)
    B, H, n, topk = 8, 64, 4096, 1024
    q = torch.randn(B, H, 576).to(torch.bfloat16)
    kvf = torch.randn(2, n, 576)
    kvf[:, n // 2:] *= mult
    kv = torch.stack([O.pack_fp8_latent(k) for k in kvf]) if fp8 else kvf.to(torch.bfloat16)
    plain = [O.unpack_fp8_latent(k) for k in kv] if fp8 else kv
    kv = kv.repeat(B // 2, 1, 1)
    idx = torch.stack([torch.sort(torch.randperm(n)[:topk]).values for _ in range(B)]).int()
    first, late = plain[0][idx[0, :64].long()].double(), plain[0][idx[0].long()].double()
    ahead = ((q[0].double() @ late.T).amax(1) - (q[0].double() @ first.T).amax(1)) * 0.07 * 1.4427
    assert float(ahead.max()) > 40  # (powers of two: what the kernel lets a score run ahead)
    got = decode(ops, TC, dev(q), dev(kv), dev(idx), 0.07, nsplit=nsplit)
    for b in range(B):
        ref = O.sparse_mla_decode(q[b:b + 1], plain[b % 2], idx[b:b + 1], [n], 0.07)
        assert torch.isfinite(got[b]).all()
        assert rel_err(got[b:b + 1], ref) < ATTN_TOL


def test_size_based_dispatch_matches(ops):
    """Eight rows of 128 heads x 2048 keys cross the tile threshold and run on the
    tcgen05 kernel by themselves; the result agrees with the mma.sync kernel."""
    torch.manual_seed(25)
    B, H, n, topk = 8, 128, 6000, 2048
    q = torch.randn(B, H, 576).to(torch.bfloat16)
    kv = torch.randn(B, n, 576).to(torch.bfloat16)
    idx = torch.stack([torch.randperm(n)[:topk] for _ in range(B)]).int()
    sm = 192 ** -0.5
    auto = decode(ops, TC, dev(q), dev(kv), dev(idx), sm)
    legacy = decode_mma_sync(ops, dev(q), dev(kv), dev(idx), sm)
    assert rel_err(auto, legacy) < ATTN_TOL
