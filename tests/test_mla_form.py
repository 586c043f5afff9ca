"""Which kernel a sparse MLA launch runs on, by its sizes (no GPU needed)."""

from __future__ import annotations

import pytest

HEADS_16, HEADS_32, HEADS_32_ONE_TILE, TC, PAIR, TWO_ROWS, FIRST_ROWS = range(7)
LIST, LENGTHS, DIRECT, BESIDE, PROMPT = 1, 2, 4, 8, 16


def form(R, rows_per_seq, H, topk, nsplit, cap, flags=LIST | LENGTHS | DIRECT, fp8=0, scale=0.07):
    from dsa_multi_layer_indexer_b200 import _lib

    return _lib.lib().dsa_sparse_mla_form(R, rows_per_seq, H, topk, nsplit, scale, cap, fp8, flags)


@pytest.mark.parametrize("R,rows_per_seq,topk,cap", [
    (256, 256, 2048, 8192), (1024, 1024, 2048, 32768), (2048, 2048, 2048, 32768), (300, 300, 300, 4096), (900, 300, 300, 556),
    (2500, 2500, 2048, 32768), (4000, 4000, 2048, 4000)])
def test_rows_behind_a_context_do_not_share_a_pair(R, rows_per_seq, topk, cap):
    """Lists that are selections from more keys than they have room for hardly ever nest."""
    assert form(R, rows_per_seq, 64, topk, 1, cap) == TC
    assert form(R, rows_per_seq, 64, topk, 1, cap, LIST | LENGTHS) == TC


@pytest.mark.parametrize("R,rows_per_seq,topk,cap,with_prompt,without", [
    (700, 700, 2048, 956, TWO_ROWS, TWO_ROWS), (700, 700, 700, 956, TWO_ROWS, TC), (600, 200, 200, 456, TWO_ROWS, TC),
    (256, 256, 256, 256, TWO_ROWS, TWO_ROWS), (2048, 2048, 2048, 2304, TWO_ROWS, TC), (255, 255, 255, 255, TC, TC),
    (382, 191, 191, 191, TC, TC), (2049, 2049, 2048, 2305, FIRST_ROWS, TC), (4002, 2001, 2000, 4096, TC, TC), (700, 700, 255, 700, TC, TC)])
def test_rows_of_a_prompt(R, rows_per_seq, topk, cap, with_prompt, without):
    every = LIST | LENGTHS | DIRECT
    assert form(R, rows_per_seq, 64, topk, 1, cap, every | PROMPT) == with_prompt
    assert form(R, rows_per_seq, 64, topk, 1, cap, every) == without
    # not without lengths, in several splits, over fp8 rows, beside the top-k or with another head count; the first rows of a
    # longer prompt not into partials either
    assert form(R, rows_per_seq, 64, topk, 1, cap, LIST | DIRECT | PROMPT) == TC
    assert form(R, rows_per_seq, 64, topk, 2, cap, LIST | LENGTHS | PROMPT) == TC
    assert form(R, rows_per_seq, 64, topk, 1, cap, every | PROMPT, fp8=1) == TC
    assert form(R, rows_per_seq, 64, topk, 1, cap, every | BESIDE) == TC
    assert form(R, rows_per_seq, 192, topk, 1, cap, every | PROMPT) == TC
    assert form(R, rows_per_seq, 64, topk, 1, cap, LIST | LENGTHS | PROMPT) == (TC if with_prompt == FIRST_ROWS else with_prompt)


@pytest.mark.parametrize("R,H,topk,nsplit,want", [
    (75, 128, 64, 1, TC), (148, 128, 40, 1, TC), (149, 128, 64, 1, PAIR), (512, 128, 64, 1, PAIR), (38, 256, 64, 1, TC), (16, 128, 512, 8, TC),
    (19, 128, 512, 8, PAIR), (19, 128, 256, 4, PAIR), (18, 128, 256, 4, TC), (38, 128, 128, 2, PAIR), (75, 128, 65, 1, PAIR),
    (74, 128, 65, 1, TC), (76, 128, 128, 1, PAIR), (38, 256, 128, 1, PAIR), (16, 128, 640, 8, PAIR)])
def test_half_tiles_on_pairs(R, H, topk, nsplit, want):
    for rows_per_seq in (1, R):
        assert form(R, rows_per_seq, H, topk, nsplit, 4096) == want


@pytest.mark.parametrize("batch,n,H,want", [(1, 75, 128, TC), (1, 128, 128, TC), (1, 149, 128, PAIR), (2, 74, 128, TC), (2, 75, 128, PAIR),
                                            (1, 74, 256, TC), (1, 75, 256, PAIR), (1, 700, 128, PAIR)])
def test_short_prompts_are_half_tiles(batch, n, H, want):
    assert form(batch * n, n, H, n, 1, n + 256, LIST | LENGTHS | DIRECT | PROMPT) == want


@pytest.mark.parametrize("R,H,topk,nsplit,cap,want", [
    (16, 128, 2048, 4, 16384, TC), (15, 128, 2048, 4, 8192, TC), (14, 128, 2048, 4, 16384, PAIR), (17, 128, 2048, 4, 16384, PAIR),
    (11, 128, 2048, 4, 40000, PAIR), (7, 256, 2048, 4, 40000, PAIR), (12, 128, 2048, 4, 40000, TC), (10, 128, 2048, 4, 40000, PAIR), (13, 128, 2048, 4, 40000, PAIR),
    (28, 128, 1024, 2, 8192, TC), (28, 128, 2048, 2, 16384, PAIR), (16, 256, 1024, 2, 8192, TC), (9, 256, 2048, 4, 8192, PAIR),
    (75, 128, 2048, 1, 16384, PAIR), (200, 128, 512, 1, 16384, PAIR), (16, 128, 2048, 4, 4096, PAIR), (16, 128, 2048, 4, 4097, TC)])
def test_pairs_beside_the_topk_need_room(R, H, topk, nsplit, cap, want):
    for rows_per_seq, stride in ((1, cap), (R, cap * R)):  # a cache each, one pool
        assert form(R, rows_per_seq, H, topk, nsplit, stride) == PAIR
        assert form(R, rows_per_seq, H, topk, nsplit, stride, LIST | LENGTHS | BESIDE) == want
