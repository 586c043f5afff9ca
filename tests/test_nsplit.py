"""The split count that plans are made with and the one that a launch takes by itself are one function; its
values over rows, heads and list lengths, against the rule written out (no GPU needed)."""

from __future__ import annotations

import math

import pytest


def rule(rows, heads, topk, sms=148):
    tiles = max(1, math.ceil(topk / 64))
    if heads % 64 == 0 and rows * (heads // 64) * tiles >= 128:  # tcgen05: CTAs of 64 heads, one per SM
        want = max(1, min(sms // max(1, rows * (heads // 64)), 16, tiles))
        while tiles % want:
            want -= 1
        return want
    want = max(1, 2 * sms // max(1, rows * (heads // 16)))  # mma.sync: CTAs of 16 heads, two per SM
    if rows * heads > sms:
        want = min(want, 16)
    return max(1, min(want, tiles))


@pytest.mark.parametrize("sms", [148, 132, 1])
def test_split_counts(sms):
    from dsa_multi_layer_indexer_b200 import ops

    for rows in (1, 2, 3, 4, 7, 8, 16, 31, 32, 64, 75, 149, 4099):
        for heads in (16, 32, 48, 64, 80, 128):
            for topk in (1, 63, 64, 65, 512, 1000, 2048, 8192):
                got = ops.default_nsplit(rows, heads, topk, sms)
                assert got == rule(rows, heads, topk, sms), (rows, heads, topk)
                assert 1 <= got <= math.ceil(topk / 64)
    assert ops.default_nsplit(1, 16, 2048) == rule(1, 16, 2048)
