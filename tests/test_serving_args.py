"""Argument checks of the serving entry point that need no GPU."""

from __future__ import annotations

import pytest

from dsa_multi_layer_indexer_b200 import serving


@pytest.mark.parametrize("select", [1, 0, 1.0, None, "Exact", ["exact"], ("prod",)])
def test_unknown_selections_are_refused(select):
    """Only True, False and the named selections: 1 and 0 equal the former, a list has no hash."""
    with pytest.raises(ValueError, match="select"):
        serving.fused_hide_decode_paged(*[None] * 9, 0.1, None, select=select)


def test_unknown_modes_are_refused():
    with pytest.raises(ValueError, match="mode"):
        serving.fused_hide_decode_paged(*[None] * 9, 0.1, None, mode="half")
