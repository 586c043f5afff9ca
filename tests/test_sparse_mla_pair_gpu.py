"""GPU tests of the sparse MLA kernel that runs 128 heads on a pair of CTAs (bf16 rows), at the sizes where it can go wrong:
a tile's last keys, one tile, several triples per pair, splits of unequal length, masked entries at either end of the list,
scores that run away from the softmax reference.

Tolerance, relative 2-norm against the same computation in 64 bits: probabilities and results are rounded to bf16, at most
2^-9 each, and their errors add up like the values themselves: 2 x 2^-9 = 3.9e-3, and 5e-3 with what the 32-bit sums add.
"""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = 5e-3
SM = 192 ** -0.5


@pytest.fixture(scope="module")
def ops():
    from dsa_multi_layer_indexer_b200 import _lib, ops as _ops

    _lib.lib()
    yield _ops
    _lib.check_device_status()


def reference(q, kv, idx, lens, rows_per_seq):
    out = torch.zeros(*q.shape[:2], 512, dtype=torch.float64, device=q.device)
    for r in range(q.shape[0]):
        i = idx[r].long()
        i = i[(i >= 0) & (i < int(lens[r]))]
        if i.numel():
            k = kv[r // rows_per_seq][i].double()
            out[r] = torch.softmax(q[r].double() @ k.T * SM, -1) @ k[:, :512]
    return out


def operands(R, H, n, topk, rows_per_seq=1, seed=0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    q = torch.randn(R, H, 576, device="cuda", generator=gen).bfloat16()
    kv = torch.randn(R // rows_per_seq, n, 576, device="cuda", generator=gen).bfloat16()
    idx = torch.full((R, topk), -1, dtype=torch.int32, device="cuda")
    take = min(n, topk)
    for r in range(R):
        idx[r, :take] = torch.randperm(n, device="cuda", generator=gen)[:take].sort().values.int()
    return q, kv, idx, torch.full((R,), n, dtype=torch.int32, device="cuda")


def check(ops, q, kv, idx, lens, rows_per_seq, nsplit, **kw):
    from dsa_multi_layer_indexer_b200 import _lib

    got = ops.sparse_mla_decode(q, kv, idx, SM, lens, rows_per_seq=rows_per_seq, nsplit=nsplit, **kw)
    _lib.check_device_status()
    want = reference(q, kv, idx, lens, rows_per_seq)
    assert torch.isfinite(got).all()
    for r in range(q.shape[0]):
        norm = float(want[r].norm())
        assert float((got[r].double() - want[r]).norm()) <= TOL * norm, r
        if norm == 0.0:
            assert float(got[r].abs().max()) == 0.0


# (rows, heads, keys, list, splits): one split of 4 tiles, with a last tile of 1, 64, 65 and 127 keys; one tile of few keys
# and two in which more triples than pairs exist; splits of which the last is short; several head blocks; several triples
# a pair of very different length
@pytest.mark.parametrize("R,H,n,topk,nsplit,rows_per_seq", [
    (8, 128, 3000, 512, 1, 1), (8, 128, 700, 513, 1, 2), (8, 128, 600, 576, 1, 8), (4, 256, 900, 577, 1, 4), (8, 128, 700, 639, 1, 1),
    (150, 128, 40, 40, 1, 150), (76, 128, 300, 64, 1, 76), (150, 128, 40, 70, 1, 150), (76, 128, 300, 65, 1, 76),
    (100, 128, 300, 129, 1, 100), (20, 512, 300, 200, 1, 1), (33, 128, 300, 256, 1, 1),
    (3, 128, 5000, 2048, 3, 1), (40, 128, 500, 129, 2, 1), (6, 384, 3000, 1100, 2, 3), (160, 128, 2100, 2048, 1, 160)])
def test_against_64_bits(ops, R, H, n, topk, nsplit, rows_per_seq):
    q, kv, idx, lens = operands(R, H, n, topk, rows_per_seq, seed=R + topk)
    check(ops, q, kv, idx, lens, rows_per_seq, nsplit)


@pytest.mark.parametrize("nsplit", [1, 3])
def test_masked_entries_and_rows(ops, nsplit):
    R, n, topk = 90, 2500, 1600
    q, kv, idx, lens = operands(R, 128, n, topk, seed=5)
    idx[:, ::17] = n + 5           # beyond the sequence
    idx[:, 3::29] = -1
    lens[1], lens[2] = 0, 1
    idx[3] = -1
    idx[4, :-3] = -1               # only the list's end
    idx[5, 1:] = -1                # only its start
    idx[6, :64] = -1               # the reference comes from the tile's other half,
    idx[7, :130] = -1              # from the next tile
    idx[8, 200:1400] = -1          # tiles without a key in between
    for r in range(9, 40):         # lengths as those of a prompt
        idx[r, 40 * (r - 8):] = -1
    check(ops, q, kv, idx, lens, 1, nsplit)


@pytest.mark.parametrize("topk,nsplit", [(2048, 1), (2050, 1), (2048, 4), (3100, 2)])
def test_where_a_list_ends(ops, topk, nsplit):
    """The plan looks for the last visible key 32 entries, then 1024 at a time from the end of a split's part of the list."""
    part = (-(-topk // nsplit) + 127) // 128 * 128
    ends = {min(max(end, 0), topk - 1) for k1 in range(0, topk + part, part) for end in
            [min(k1, topk) - back for back in (1, 2, 31, 32, 33, 34, 1055, 1056, 1057, 1058, 2047, 2048)]}
    ends = sorted(ends)
    R, n = 80, 3200
    q, kv, idx, lens = operands(R, 128, n, topk, rows_per_seq=R, seed=topk)
    for r in range(R):
        idx[r, ends[r % len(ends)] + 1:] = -1
        if r >= len(ends):
            idx[r, :ends[r % len(ends)]] = n  # nothing in front of it either
    check(ops, q, kv, idx, lens, R, nsplit)


def test_short_rows_in_long_lists_take_no_longer_than_in_short_ones(ops):
    def us(topk):
        q, kv, idx, _ = operands(40, 128, 3000, topk, rows_per_seq=40)
        idx[:, 40:] = -1
        lens = torch.full((40,), 40, dtype=torch.int32, device="cuda")
        idx[:, :40] = torch.arange(40, dtype=torch.int32, device="cuda")
        run = lambda: ops.sparse_mla_decode(q, kv, idx, SM, lens, rows_per_seq=40, nsplit=1)
        run()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for _ in range(20):
                run()
        graph.replay()
        times = []
        for _ in range(10):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            graph.replay()
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return min(times) / 20 * 1e3

    # (11.1 and 11.8 us; entries requested one by one: 12.6 and 22.8)
    assert us(2048) < 1.35 * us(256)


def test_scores_that_run_away(ops):
    R, n, topk = 8, 2048, 2048
    q, kv, idx, lens = operands(R, 128, n, topk, seed=9)
    grow = torch.linspace(0.01, 3, n, device="cuda")[None, :, None]
    q = (q.float() * 60).bfloat16()
    kv = (kv.float() * grow).bfloat16()
    kv[3] = kv[3].flip(0)          # largest first
    kv[4, :64] *= 0.001            # the first half of the first tile is far below the second
    check(ops, q, kv, idx, lens, 1, 1)
    check(ops, q, kv, idx, lens, 1, 2)


def test_no_list_attends_every_key(ops):
    from dsa_multi_layer_indexer_b200 import _lib

    q, kv, _, _ = operands(8, 128, 1000, 8, seed=3)
    lens = torch.tensor([1000, 999, 513, 1, 0, 128, 129, 700], dtype=torch.int32, device="cuda")
    got = ops.sparse_mla_decode(q, kv, None, SM, lens, nsplit=1, dense_keys=1000)
    _lib.check_device_status()
    every = torch.arange(1000, dtype=torch.int32, device="cuda").expand(8, -1)
    want = reference(q, kv, every, lens, 1)
    assert float((got.double() - want).norm()) <= TOL * float(want.norm())
    assert float(got[4].abs().max()) == 0.0


def test_agrees_with_one_cta_per_64_heads(ops):
    """64 heads at a time run on the other kernel: the same reference, the same rounded probabilities and products added in
    the same order, so only the row sums' order can round a result the other way."""
    q, kv, idx, lens = operands(40, 128, 3000, 2048, seed=7)
    both = ops.sparse_mla_decode(q, kv, idx, SM, lens, nsplit=1)
    for h in (0, 64):
        half = ops.sparse_mla_decode(q[:, h:h + 64].contiguous(), kv, idx, SM, lens, nsplit=1)
        same = both[:, h:h + 64]
        assert float((same != half).float().mean()) < 0.01
        assert float((same.float() - half.float()).norm()) <= 2.0 ** -9 * float(half.float().norm())


def test_several_launches_in_a_graph_and_on_two_streams(ops):
    from dsa_multi_layer_indexer_b200 import _lib

    a = operands(90, 128, 900, 600, 90, seed=1)
    b = operands(90, 128, 900, 600, 90, seed=2)
    run = lambda o: ops.sparse_mla_decode(*o[:3], SM, o[3], rows_per_seq=90, nsplit=1)
    want = [run(a), run(b)]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = [run(a), run(b), run(a)]
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]) and torch.equal(got[2], want[0])
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        other = run(b)
    mine = run(a)
    torch.cuda.synchronize()
    assert torch.equal(mine, want[0]) and torch.equal(other, want[1])
    _lib.check_device_status()


# ---- 64 heads: two rows of a prompt on a pair, where the second row sees what the first one sees and one key more
def prompt(batch, n, topk, seed=0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    q = torch.randn(batch * n, 64, 576, device="cuda", generator=gen).bfloat16()
    kv = torch.randn(batch, n, 576, device="cuda", generator=gen).bfloat16()
    pos = torch.arange(topk, dtype=torch.int32, device="cuda")
    row = torch.arange(n, dtype=torch.int32, device="cuda")
    idx = torch.where(pos[None] <= row[:, None], pos[None], -1).repeat(batch, 1).contiguous()
    return q, kv, idx, (row + 1).repeat(batch)


@pytest.mark.parametrize("batch,n,topk", [(1, 256, 256), (1, 257, 300), (2, 193, 193), (3, 200, 256), (1, 385, 385), (1, 700, 703)])
def test_two_rows_of_a_prompt(ops, batch, n, topk):
    check(ops, *prompt(batch, n, topk, seed=n), n, 1)


def test_two_rows_without_a_list(ops):
    n = 259
    q, kv, idx, lens = prompt(1, n, n, seed=11)
    got = ops.sparse_mla_decode(q, kv, None, SM, lens, rows_per_seq=n, nsplit=1, dense_keys=n)
    want = ops.sparse_mla_decode(q, kv, idx, SM, lens, rows_per_seq=n, nsplit=1)
    assert torch.equal(got, want)


@pytest.mark.parametrize("n,topk", [(257, 256), (400, 256), (700, 301)])
def test_a_prompt_longer_than_its_lists(ops, n, topk):
    """The rows that the list has room for go two by two, the others one by one beside them."""
    q, kv, _, lens = prompt(1, n, n, seed=n)
    gen = torch.Generator(device="cuda").manual_seed(topk)
    idx = torch.full((n, topk), -1, dtype=torch.int32, device="cuda")
    for r in range(n):
        k = min(r + 1, topk)
        idx[r, :k] = torch.randperm(r + 1, device="cuda", generator=gen)[:k].sort().values.int()
    check(ops, q, kv, idx, lens, n, 1, prompt=True)
    check(ops, q, kv, idx, lens, n, 1)


def test_what_is_called_a_prompt_and_is_none(ops):
    """Rows behind a context, lists that do not nest: the caller's word changes the launch, not the result."""
    q, kv, idx, lens = operands(400, 64, 900, 256, 400, seed=13)
    check(ops, q, kv, idx, lens, 400, 1, prompt=True)


def test_a_prefill_says_that_its_rows_are_a_prompt(ops, monkeypatch):
    import dataclasses

    import dsa_multi_layer_indexer_b200 as dsa

    said, decode = [], ops.sparse_mla_decode
    monkeypatch.setattr(ops, "sparse_mla_decode", lambda *a, **kw: said.append(kw.get("prompt", False)) or decode(*a, **kw))
    cfg = dataclasses.replace(dsa.named_config("glm5"), num_hidden_layers=1, first_k_dense_replace=0)
    torch.manual_seed(0)
    with torch.device("cuda"):
        model = dsa.DSAModel(cfg).to(torch.bfloat16).eval()
    model.prefill(model.init_decode(1, 128), torch.randn(1, 70, cfg.hidden_size, device="cuda").bfloat16())
    assert said == [True]


def rows_that_differ(n):
    """Lists that do not nest, rows of which one or both see nothing, lengths that shrink."""
    q, kv, idx, lens = prompt(1, n, 400, seed=4)
    gen = torch.Generator(device="cuda").manual_seed(5)
    for r in range(20, 60):                                    # unrelated lists
        idx[r] = -1
        idx[r, :100] = torch.randperm(n, device="cuda", generator=gen)[:100].int()
        lens[r] = n
    idx[60, :3] = torch.tensor([2, 0, 1], dtype=torch.int32)   # the second row's list in another order
    idx[70] = -1
    idx[73] = -1
    idx[74:76] = -1
    lens[80] = 0
    lens[83] = 5                                               # shorter than the row before it
    idx[85, 84:90] = torch.tensor([84, 85, 86, 87, 88, 89], dtype=torch.int32)  # more than one key more
    lens[85] = n
    idx[90, 10] = -1                                           # the first row misses one in the middle,
    idx[93, 10] = -1                                           # the second one does
    return q, kv, idx, lens


def test_two_rows_that_differ(ops):
    check(ops, *rows_that_differ(260), 260, 1)


@pytest.mark.parametrize("operands_of", [lambda: (*prompt(1, 257, 300, seed=3), 257), lambda: (*prompt(2, 193, 193, seed=4), 193),
                                         lambda: (*rows_that_differ(260), 260), lambda: (*rows_that_differ(261), 261)])
def test_two_rows_into_partials(ops, operands_of):
    """The two-row form with a caller's scratch: of one split, the merge makes the same result of it bit for bit."""
    from dsa_multi_layer_indexer_b200 import _lib

    q, kv, idx, lens, rows_per_seq = operands_of()
    R, cap = q.shape[0], kv.shape[1]
    assert _lib.lib().dsa_sparse_mla_form(R, rows_per_seq, 64, idx.shape[1], 1, SM, cap, 0, 1 | 2) == 5
    want = ops.sparse_mla_decode(q, kv, idx, SM, lens, rows_per_seq=rows_per_seq, nsplit=1)
    scratch = ops.MlaScratch(R + 1, 64, 1, "cuda")
    for t in (scratch.acc, scratch.m, scratch.l):
        t.fill_(float("nan"))
    kw = dict(rows_per_seq=rows_per_seq, nsplit=1, scratch=scratch)
    ops.sparse_mla_decode(q, kv, idx, SM, lens, stage="partials", **kw)
    _lib.check_device_status()
    assert torch.isfinite(scratch.acc[:R]).all() and not torch.isnan(scratch.m[:R]).any() and torch.isfinite(scratch.l[:R]).all()
    assert torch.isnan(scratch.acc[R]).all() and torch.isnan(scratch.m[R]).all() and torch.isnan(scratch.l[R]).all()
    assert torch.equal(ops.sparse_mla_decode(q, kv, idx, SM, lens, stage="combine", **kw), want)
    assert torch.equal(ops.sparse_mla_decode(q, kv, idx, SM, lens, **kw), want)


def test_a_long_prompt_right_behind_its_selection(ops):
    """Both launches of a prompt longer than its lists read what the kernel in front of them writes: the second one starts
    without a wait of its own, behind the first one's. Replayed over changing logits."""
    from dsa_multi_layer_indexer_b200 import _lib

    n, topk = 900, 300
    q, kv, _, lens = prompt(1, n, n, seed=21)
    gen = torch.Generator(device="cuda").manual_seed(22)
    logits = torch.zeros(n, n, device="cuda")
    lists = torch.empty(n, topk, dtype=torch.int32, device="cuda")
    out = torch.empty(n, 64, 512, dtype=torch.bfloat16, device="cuda")

    def both():
        ops.topk_select(logits, topk, lens, out_idx=lists)
        ops.sparse_mla_decode(q, kv, lists, SM, lens, rows_per_seq=n, nsplit=1, out=out, prompt=True)

    assert _lib.lib().dsa_sparse_mla_form(n, n, 64, topk, 1, SM, n, 0, 1 | 2 | 4 | 16) == 6
    both()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(2):
            both()
    for _ in range(4):
        logits.copy_(torch.randn(n, n, device="cuda", generator=gen))
        ops.topk_select(logits, topk, lens, out_idx=lists)
        torch.cuda.synchronize()
        want = ops.sparse_mla_decode(q, kv, lists, SM, lens, rows_per_seq=n, nsplit=1, prompt=True)
        torch.cuda.synchronize()
        lists.fill_(-1)
        out.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    _lib.check_device_status()
    check(ops, q, kv, lists, lens, n, 1, prompt=True)


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("dim", [0, 511, 512])
def test_a_key_that_is_not_finite_stays_out_of_the_rows_before_it(ops, bad, dim):
    n, at = 256, 101  # the second row of its pair
    q, kv, idx, lens = prompt(1, n, n, seed=6)
    clean = ops.sparse_mla_decode(q, kv, idx, SM, lens, rows_per_seq=n, nsplit=1).clone()
    kv[0, at, dim] = bad
    got = ops.sparse_mla_decode(q, kv, idx, SM, lens, rows_per_seq=n, nsplit=1)
    assert torch.equal(got[:at], clean[:at])
    # from there on what 64 bits make of it: a bad value dim spoils that dim (and, through the scores, every dim of the heads
    # whose scores it reaches), a bad score dim every dim
    for r in range(at, n):
        k = kv[0, :r + 1].double()
        s = q[r].double() @ k.T * SM
        p = torch.softmax(s, -1)
        want = torch.isfinite(p @ k[:, :512])
        assert not want.all() and torch.equal(torch.isfinite(got[r]), want), r


def test_two_rows_agree_with_one_at_a_time(ops):
    n = 640
    q, kv, idx, lens = prompt(1, n, n, seed=8)
    both = ops.sparse_mla_decode(q, kv, idx, SM, lens, rows_per_seq=n, nsplit=1)
    for r in range(0, n, 80):  # (fewer rows run on the other kernel)
        some = slice(r, r + 80)
        alone = ops.sparse_mla_decode(q[some].contiguous(), kv, idx[some].contiguous(), SM, lens[some].contiguous(), rows_per_seq=80, nsplit=1)
        assert float((both[some] != alone).float().mean()) < 0.01
        assert float((both[some].float() - alone.float()).norm()) <= 2.0 ** -9 * float(alone.float().norm())
