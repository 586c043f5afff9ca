"""GPU tests of a decode step over the batch sizes and module forms that take different launches: each
sequence must come out as it does alone, up to the roundings of bf16 activations by other kernels."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def D():
    import dsa_multi_layer_indexer_b200 as pkg
    from dsa_multi_layer_indexer_b200 import _lib

    _lib.lib()
    yield pkg
    _lib.check_device_status()


def make_model(D, layers=2, **kw):
    cfg = D.DSAConfig(hidden_size=256, num_hidden_layers=layers, num_attention_heads=16, q_lora_rank=96, index_n_heads=32,
                      index_topk=64, intermediate_size=256, first_k_dense_replace=0, **kw)  # (64: every key of these contexts)
    torch.manual_seed(5)
    return D.DSAModel(cfg).eval().cuda().to(torch.bfloat16)


def decode(model, prompt, toks, mode, cold, **kw):
    state = model.init_decode(prompt.shape[0], 64)
    model.prefill(state, prompt, mode, cold)
    return torch.stack([model.decode_step(state, t, mode, cold, **kw) for t in toks])


def rel(a, b):
    return float((a.float() - b.float()).norm() / b.float().norm())


# one launch for up to eight tokens, GEMMs and a separate preparation beyond
@pytest.mark.parametrize("batch", [2, 3, 4, 5, 8, 9, 16, 33])
@pytest.mark.parametrize("mode_name", ["BASELINE", "LAGGED_FUSED"])
def test_batches_decode_as_their_sequences_alone(D, batch, mode_name):
    mode, cold = D.ScheduleMode[mode_name], D.ColdStartPolicy.EAGER
    model = make_model(D)
    prompt = torch.randn(batch, 20, 256, device="cuda").to(torch.bfloat16)
    toks = torch.randn(3, batch, 256, device="cuda").to(torch.bfloat16)
    got = decode(model, prompt, toks, mode, cold)
    for i in (0, batch - 1):
        alone = decode(model, prompt[i:i + 1], toks[:, i:i + 1], mode, cold)
        assert rel(got[:, i:i + 1], alone) < 2e-2  # a few bf16 roundings (2^-9 each) per layer


@pytest.mark.parametrize("batch", [1, 3, 9])
def test_norm_weights_in_fp32(D, batch):
    """A bf16 model whose norms stay in fp32 decodes as one with the same numbers in bf16."""
    mode, cold = D.ScheduleMode.LAGGED_FUSED, D.ColdStartPolicy.EAGER
    model = make_model(D)
    norms = [m for m in model.modules() if type(m).__name__ == "RMSNorm"]
    with torch.no_grad():
        for m in norms:
            m.weight.copy_(1.0 + torch.randint(-32, 33, m.weight.shape) / 64.0)
    prompt = torch.randn(batch, 20, 256, device="cuda").to(torch.bfloat16)
    toks = torch.randn(3, batch, 256, device="cuda").to(torch.bfloat16)
    want = decode(model, prompt, toks, mode, cold)
    for m in norms:
        m.float()
    assert rel(decode(model, prompt, toks, mode, cold), want) < 2e-2  # (bf16 roundings of norms by other kernels)
