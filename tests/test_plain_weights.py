"""What makes a projection's weight one that the native chain may multiply by itself (no GPU needed)."""

from __future__ import annotations

import sys

import pytest
import torch

import dsa_multi_layer_indexer_b200 as D
from dsa_multi_layer_indexer_b200.dsa_layer import _PROJECTIONS, _plain_weights


@pytest.fixture
def layer():
    return D.DSAModel(D.SMALL_CONFIG).layers[0]


def plain(layer, dtype=torch.float32):
    return _plain_weights(layer._modules, _PROJECTIONS, dtype)


def test_plain_projections_give_their_parameters(layer):
    weights = plain(layer)
    assert [w is getattr(layer, n).weight for w, n in zip(weights, _PROJECTIONS)] == [True] * len(_PROJECTIONS)
    assert plain(layer, torch.bfloat16) is None and plain(layer.to(torch.bfloat16), torch.bfloat16) is not None


def test_one_projection_that_is_not_plain_is_enough(layer):
    class Other(torch.nn.Parameter):
        pass

    m, kept = layer.up_proj, layer.up_proj.weight
    handle = m.register_forward_hook(lambda *a: None)
    assert plain(layer) is None
    handle.remove()
    handle = m.register_forward_pre_hook(lambda *a: None)
    assert plain(layer) is None
    handle.remove()
    m.forward = lambda t: t
    assert plain(layer) is None
    del m.forward
    m.bias = torch.nn.Parameter(torch.zeros(m.out_features))
    assert plain(layer) is None
    m.bias = None
    m.weight = Other(kept.detach())
    assert type(m.weight) is Other and plain(layer) is None
    m.weight = torch.nn.Parameter(kept.detach().double())
    assert plain(layer) is None
    m.weight = kept
    assert plain(layer) is not None
    layer.up_proj = torch.nn.Identity()
    assert plain(layer) is None
    layer.up_proj = m
    torch.nn.utils.parametrizations.weight_norm(layer.down_proj)
    assert plain(layer) is None


def test_looking_keeps_no_references(layer):
    w, d = layer.q_a_proj.weight, layer.q_a_proj.__dict__
    before = sys.getrefcount(w), sys.getrefcount(d)
    for _ in range(50):
        plain(layer)
        _plain_weights(layer._modules, ("q_a_proj", "attn_norm"), torch.float32)
    assert (sys.getrefcount(w), sys.getrefcount(d)) == before
