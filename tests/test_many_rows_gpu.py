"""GPU tests of the kernels for many short rows (full-sequence layers): the one-CTA-per-row top-k
against a stable sort, the fp32 scan and the fp32 attention that share keys between heads against
plain fp32 arithmetic (1e-5: sums of at most a few hundred fp32 products in another order)."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

ROWS = 160  # more rows than SMs: the row kernel


@pytest.fixture(scope="module")
def ops():
    from dsa_multi_layer_indexer_b200 import _lib, ops as _ops

    yield _ops
    _lib.check_device_status()


def expected(x, lens, k, pad):
    out = torch.full((x.shape[0], k), pad, dtype=torch.int32)
    for r in range(x.shape[0]):
        n = min(max(int(lens[r]), 0), x.shape[1])
        order = torch.sort(x[r, :n], descending=True, stable=True).indices[:k]
        order = order.sort().values
        order = torch.where(torch.isinf(x[r, order]) & (x[r, order] < 0), torch.tensor(pad), order)
        out[r, :order.numel()] = order.int()
    return out


@pytest.mark.parametrize("n,k", [(1, 1), (31, 16), (500, 16), (2048, 2048), (2049, 64), (4096, 512), (4099, 2048), (8192, 2048),
                                 (8193, 2048), (16384, 300)])
@pytest.mark.parametrize("kind", ["random", "ties", "equal", "inf"])
def test_row_topk_matches_a_stable_sort(ops, n, k, kind):
    torch.manual_seed(n + k)
    x = torch.randn(ROWS, n)
    if kind == "ties":
        x = (x * 2).round() / 2
        x[::2][x[::2] == 0] = -0.0
    elif kind == "equal":
        x[:] = 1.25
    elif kind == "inf":
        x[torch.rand_like(x) < 0.9] = float("-inf")
        x[3, : n // 2] = float("inf")
    lens = torch.randint(0, n + 1, (ROWS,), dtype=torch.int32)
    lens[0], lens[1], lens[2] = n, 0, n + 5
    got = ops.topk_select(x.cuda(), k, lens.cuda(), pad_value=-3).cpu()
    assert torch.equal(got, expected(x, lens, k, -3))


def test_row_topk_values_map_offset_and_strided_slab(ops):
    torch.manual_seed(1)
    n, k = 700, 64
    slab = torch.randn(ROWS, n + 9, device="cuda")
    x = slab[:, :n]
    idx, val = ops.topk_select(x, k, return_values=True, index_offset=1000)
    ref = expected(x.cpu(), [n] * ROWS, k, -1)
    assert torch.equal(idx.cpu(), ref + 1000)
    assert torch.equal(val, x.gather(1, ref.long().cuda()))
    m = torch.randint(0, 1 << 20, (ROWS, n), dtype=torch.int32, device="cuda")
    mapped = ops.topk_select(x, k, index_map=m)
    assert torch.equal(mapped, m.gather(1, ref.long().cuda()))
    nan = x.clone()
    nan[5, 10:] = float("nan")
    assert ops.topk_select(nan, k)[5].shape == (k,)  # terminates; the other rows are untouched
    assert torch.equal(ops.topk_select(nan, k)[6].cpu(), ref[6])


@pytest.mark.parametrize("rps,n_seq,heads,dim,ctx", [(1, 3, 64, 128, 100), (20, 2, 8, 16, 33), (9, 1, 5, 7, 64), (17, 2, 33, 130, 65),
                                                     (3, 1, 70, 300, 31)])
def test_f32_scan_matches_plain_arithmetic(ops, rps, n_seq, heads, dim, ctx):
    torch.manual_seed(heads + dim)
    R, cap = rps * n_seq, ctx + 5
    q, w = torch.randn(R, heads, dim, device="cuda"), torch.randn(R, heads, device="cuda") / 8
    k = torch.randn(n_seq, cap, dim, device="cuda")
    lens = torch.randint(0, ctx + 1, (R,), dtype=torch.int32, device="cuda")
    lens[0] = ctx
    got = ops.indexer_scan_f32(q, w, k, lens, rows_per_seq=rps, ctx=ctx)
    kk = k[:, :ctx].double().repeat_interleave(rps, 0)
    dots = torch.einsum("rhd,rsd->rhs", q.double(), kk).clamp(min=0)
    ref = (dots * w.double().unsqueeze(-1)).sum(1)
    dead = torch.arange(ctx, device="cuda")[None, :] >= lens[:, None]
    assert torch.isneginf(got[dead]).all() and torch.isfinite(got[~dead]).all()
    scale = float((dots * w.double().abs().unsqueeze(-1)).sum(1).max())
    assert float((got.double() - ref)[~dead].abs().max()) < 1e-5 * scale


@pytest.mark.parametrize("H,qk,v,topk", [(8, 80, 64, 16), (3, 20, 20, 40), (17, 576, 512, 33), (8, 84, 70, None)])
def test_f32_attention_rows_match_plain_arithmetic(ops, H, qk, v, topk):
    torch.manual_seed(H + qk)
    rps, n_seq, ctx = 90, 2, 120
    R = rps * n_seq
    q, kv = torch.randn(R, H, qk, device="cuda"), torch.randn(n_seq, ctx, qk, device="cuda")
    lens = torch.arange(1, rps + 1, dtype=torch.int32, device="cuda").repeat(n_seq)
    idx = None
    if topk is not None:
        idx = torch.stack([torch.randperm(ctx)[:topk] for _ in range(R)]).int().cuda()
        idx[1] = -1
    got = ops.sparse_mla_f32(q, kv, idx, v, 0.1, lens, rows_per_seq=rps)
    keep = torch.zeros(R, ctx, dtype=torch.bool, device="cuda")
    if idx is None:
        keep[:] = True
    else:
        keep.scatter_(1, idx.clamp(min=0).long(), idx >= 0)
    keep &= torch.arange(ctx, device="cuda")[None, :] < lens[:, None]
    kk = kv.double().repeat_interleave(rps, 0)
    s = torch.einsum("rhd,rsd->rhs", q.double(), kk) * 0.1
    p = torch.softmax(s.masked_fill(~keep[:, None], float("-inf")), -1).nan_to_num(0.0)
    ref = torch.einsum("rhs,rsd->rhd", p, kk[..., :v])
    assert float((got.double() - ref).abs().max()) < 1e-5 * float(ref.abs().max())


def test_f32_residual_norm_and_silu(ops):
    torch.manual_seed(4)
    x, d, w = torch.randn(5, 300, device="cuda"), torch.randn(5, 300, device="cuda"), torch.randn(300, device="cuda")
    s, n = ops.add_rmsnorm(x, d, w, 1e-6)
    assert torch.equal(s, x + d)
    ref = (x + d).double()
    ref = ref * torch.rsqrt(ref.pow(2).mean(-1, keepdim=True) + 1e-6) * w.double()
    assert float((n.double() - ref).abs().max()) < 1e-5 * float(ref.abs().max())
    y = ops.silu_mul(x, d)
    ref = torch.nn.functional.silu(x.double()) * d.double()
    assert float((y.double() - ref).abs().max()) < 1e-6 * float(ref.abs().max())


@pytest.mark.parametrize("m,k,ns", [(1, 4, (1,)), (64, 16, (32, 32, 32)), (65, 20, (33, 1, 70)), (1024, 256, (96, 80, 16)), (7, 300, (5, 9))])
def test_small_f32_linears_match_fp64(m, k, ns):
    """dsa_linear_f32 at the edges of its 64 x 32 tiles, 64 deep; 1e-5 per term of products of N(0, 1) numbers (a sum of k
    fp32 products in another order; of magnitudes: test_small_f32_swiglu_matches_fp64)."""
    from dsa_multi_layer_indexer_b200 import _lib

    torch.manual_seed(m + k)
    x = torch.randn(m, k, device="cuda")
    ws = [torch.randn(n, k, device="cuda") for n in ns]
    ys = [torch.full((m, n), 7.0, device="cuda") for n in ns]
    args = []
    for i in range(3):
        args += [ws[i].data_ptr(), ns[i], ys[i].data_ptr()] if i < len(ns) else [None, 0, None]
    st = torch.cuda.current_stream().cuda_stream
    _lib.check(_lib.lib().dsa_linear_f32(x.data_ptr(), m, k, *args, 0, st))
    bound = 1e-6 * k
    for w, y in zip(ws, ys):
        assert float((y.double() - x.double() @ w.double().T).abs().max()) < bound * 10
    if len(ns) == 1 or ns[0] == ns[1]:
        up = torch.randn(ns[0], k, device="cuda")
        _lib.check(_lib.lib().dsa_linear_f32(x.data_ptr(), m, k, ws[0].data_ptr(), ns[0], ys[0].data_ptr(), up.data_ptr(), ns[0], None,
                                             None, 0, None, 1, st))
        g, u = x.double() @ ws[0].double().T, x.double() @ up.double().T
        ref = torch.nn.functional.silu(g) * u
        assert float((ys[0].double() - ref).abs().max()) < bound * 10 * max(1.0, float(u.abs().max()))


def test_hooked_or_replaced_projections_keep_the_module_path():
    import dsa_multi_layer_indexer_b200 as D

    torch.manual_seed(9)
    model = D.DSAModel(D.named_config("small")).eval().cuda()
    x = torch.randn(1, 40, 256, device="cuda")
    mode, cold = D.ScheduleMode.LAGGED_FUSED, D.ColdStartPolicy.EAGER
    seen = []
    with torch.no_grad():
        plain = model(x, mode, cold)
        handle = model.layers[2].gate_proj.register_forward_hook(lambda m, a, o: seen.append(o.shape))
        hooked = model(x, mode, cold)
        handle.remove()
    assert seen == [torch.Size([1, 40, 512])]
    assert float((plain - hooked).abs().max()) < 1e-4 * float(plain.abs().max())


def scan_histogram(x, lens):
    """What the scan leaves for the top-k: counts of the top 12 bits of the order-preserving key."""
    bits = (x + 0.0).view(torch.int32)
    key = torch.where(bits < 0, ~bits, bits ^ -(1 << 31)).long() & 0xFFFFFFFF
    hist = torch.zeros(x.shape[0], 4096, dtype=torch.int32)
    for r in range(x.shape[0]):
        n = min(max(int(lens[r]), 0), x.shape[1])
        hist[r] = torch.bincount(key[r, :n] >> 20, minlength=4096).int()
    return hist


@pytest.mark.parametrize("n,k", [(1, 4), (60, 16), (2048, 512), (2049, 2048), (4096, 2048), (4097, 64), (8192, 2048), (8193, 2048),
                                 (16384, 2048)])
@pytest.mark.parametrize("kind", ["random", "ties", "equal", "inf", "close"])
def test_solo_topk_with_the_scans_histogram(ops, n, k, kind):
    """Rows with a histogram (up to 4096 logits: register kernel), at the edges of its sizes, with
    more equal logits than it ranks by comparison, and with logits that share their top 19 bits."""
    torch.manual_seed(n + k)
    rows = 5
    x = torch.randn(rows, n)
    if kind == "ties":
        x = (x * 2).round() / 2
        x[::2][x[::2] == 0] = -0.0
    elif kind == "equal":
        x[:] = -2.5
    elif kind == "inf":
        x[torch.rand_like(x) < 0.9] = float("-inf")
        x[3, : n // 2] = float("inf")
    elif kind == "close":
        x = 1.0 + torch.randint(0, 1 << 9, (rows, n)) * 2.0 ** -23
    lens = torch.tensor([n, 0, n + 5, max(1, n - 3), n // 2], dtype=torch.int32)
    hist = scan_histogram(x, lens).cuda()
    got = ops.topk_select(x.cuda(), k, lens.cuda(), hist=hist, pad_value=-3, index_offset=7).cpu()
    ref = expected(x, lens, k, -10)
    assert torch.equal(got, torch.where(ref == -10, torch.tensor(-3, dtype=torch.int32), ref + 7))
    assert int(hist.abs().sum()) == 0  # re-armed for the next scan


@pytest.mark.parametrize("n,k", [(60, 16), (60, 100), (512, 64), (2048, 300), (4096, 2048), (4096, 5000), (6000, 64)])
def test_nans_are_ranked_and_not_selected_by_any_kernel(ops, n, k):
    """Rows with NaNs by the three kernels that a row of this size can take (one CTA without a histogram, one with
    the scan's, the cluster kernel): the same positions. A NaN takes a rank and is not selected."""
    torch.manual_seed(n + k)
    x = torch.randn(ROWS, n)
    x[:, ::7] = float("-inf")
    for r, share in enumerate((0.0, 0.01, 0.2, 0.9, 1.0)):
        x[r][torch.rand(n) < share] = float("nan")
    x[1, 0] = -float("nan")
    lens = torch.full((ROWS,), n, dtype=torch.int32)
    lens[5:8] = torch.tensor([0, n // 2, min(k, n)], dtype=torch.int32)
    x[6, : n // 4] = float("nan")
    x[7, 1::3] = float("nan")
    few = 8
    cluster = ops.topk_select(x[:few].cuda(), k, lens[:few].cuda(), pad_value=-3, index_offset=5).cpu()
    for r in range(few):  # the rule itself
        row = x[r, : int(lens[r])]
        nans = int(row.isnan().sum())
        kept = row.numel() if k >= row.numel() else max(0, k - nans)
        numbers = torch.sort(row[~row.isnan()], descending=True, stable=True).indices[:kept]
        pos = torch.nonzero(~row.isnan()).flatten()[numbers].sort().values
        want = torch.full((k,), -3, dtype=torch.int32)
        want[: pos.numel()] = torch.where(torch.isneginf(row[pos]), torch.tensor(-3), pos.int() + 5).int()
        assert torch.equal(cluster[r], want), r
    rows = ops.topk_select(x.cuda(), k, lens.cuda(), pad_value=-3, index_offset=5).cpu()
    assert torch.equal(rows[:few], cluster)
    hist = torch.zeros(few, 4096, dtype=torch.int32)
    for r in range(few):  # (the scan counts a NaN in the last bin, whatever its sign)
        row = x[r, : int(lens[r])]
        bits = (row[~row.isnan()] + 0.0).view(torch.int32)
        key = torch.where(bits < 0, ~bits, bits ^ -(1 << 31)).long() & 0xFFFFFFFF
        hist[r] = torch.bincount(key >> 20, minlength=4096).int()
        hist[r, 4095] += int(row.isnan().sum())
    solo = ops.topk_select(x[:few].cuda(), k, lens[:few].cuda(), hist=hist.cuda(), pad_value=-3, index_offset=5).cpu()
    assert torch.equal(solo, cluster)


@pytest.mark.parametrize("n", [6144, 6145, 8192, 8193])
@pytest.mark.parametrize("rows", [149, 296, 297])
def test_row_topk_around_the_line_to_the_cluster_kernel(ops, rows, n):
    """Longer rows change kernel at two rows per SM (148 of them here) and at 8192 logits."""
    torch.manual_seed(rows + n)
    x = (torch.randn(rows, n) * 4).round() / 4
    lens = torch.randint(n - 700, n + 1, (rows,), dtype=torch.int32)
    got = ops.topk_select(x.cuda(), 700, lens.cuda(), pad_value=-3).cpu()
    some = [0, 1, rows // 2, rows - 1]
    assert torch.equal(got[some], expected(x[some], lens[some], 700, -3))
    values = torch.where(torch.arange(n)[None] < lens[:, None], x, torch.tensor(float("-inf"))).topk(700, -1).values
    assert torch.equal(x.gather(1, got.long()).sort(-1, descending=True).values, values)


# on both sides of the line between the kernels: a warp per key (few CTAs, wide keys), rows or heads of a CTA staged
@pytest.mark.parametrize("rps,n_seq,heads,dim,ctx", [(8, 1, 64, 128, 130), (8, 1, 16, 64, 4700), (8, 1, 16, 64, 9001), (1, 1, 8, 32, 70),
                                                     (1, 4, 8, 16, 70), (1, 2, 4, 256, 300), (8, 2, 3, 129, 600), (64, 4, 4, 130, 3000),
                                                     (1, 1, 300, 200, 40), (2, 1, 400, 128, 33)])
def test_f32_scan_kernels_agree_with_plain_arithmetic(ops, rps, n_seq, heads, dim, ctx):
    test_f32_scan_matches_plain_arithmetic(ops, rps, n_seq, heads, dim, ctx)


# one and two heads: a CTA per head unless the list is short, or there are more rows than SMs
@pytest.mark.parametrize("H,topk", [(1, 64), (1, 65), (2, 70), (1, None)])
def test_f32_attention_of_few_heads(ops, H, topk):
    test_f32_attention_rows_match_plain_arithmetic(ops, H, 80, 64, topk)


# one, two and several 64-deep slices, a part of one, both groups of threads, partial row and column tiles
@pytest.mark.parametrize("m,n,k", [(1, 1, 4), (64, 32, 16), (65, 33, 20), (1024, 96, 256), (7, 5, 300), (65, 31, 64), (63, 65, 68), (130, 40, 1028)])
def test_small_f32_swiglu_matches_fp64(m, n, k):
    """Both matrices' sums, their fold over the thread groups and the slices' ring: 2^-24 per term and step of the
    order, bounded by (k / 16 + 4) 2^-23 of the sum of magnitudes of each factor, and |silu'| < 1.1."""
    from dsa_multi_layer_indexer_b200 import _lib

    torch.manual_seed(m + n + k)
    x, wg, wu = (torch.randn(r, k, device="cuda") for r in (m, n, n))
    y = torch.full((m, n), 7.0, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    _lib.check(_lib.lib().dsa_linear_f32(x.data_ptr(), m, k, wg.data_ptr(), n, y.data_ptr(), wu.data_ptr(), n, None, None, 0, None, 1, st))
    x, wg, wu = x.double(), wg.double(), wu.double()
    g, u = x @ wg.T, x @ wu.T
    step = (k / 16 + 4) * 2.0 ** -23
    dg, du = x.abs() @ wg.abs().T * step, x.abs() @ wu.abs().T * step
    silu = torch.nn.functional.silu(g)
    err = 1.1 * dg * (u.abs() + du) + silu.abs() * du + (silu * u).abs() * 2.0 ** -20  # (expf, the division, the product)
    assert float(((y.double() - silu * u).abs() - err).max()) <= 0.0
