"""GPU parity of the fused full-sequence preparation (dsa_prefill_latents / dsa_prefill_queries) with
the chain of separate operations it replaces (src/lagged_indexer_dsa/dsa_layer.py:87-143), which the
layer still runs when autograd is on. The rotary embeddings and the quantisation are the same
operations with the same roundings, so they agree exactly; the two norms add their squares in another
order, so a normed value may move by one unit in the last place of its type, and what is computed
from it by that much again (bf16: 2^-7 relative to the row's largest value; fp32: 1e-5)."""

from __future__ import annotations

import dataclasses

import pytest
import torch

pytestmark = pytest.mark.gpu


def _layer(dtype, interleave, heads, production=True):
    import dsa_multi_layer_indexer_b200 as D

    if production:
        cfg = D.DSAConfig(hidden_size=192, num_hidden_layers=1, num_attention_heads=heads, q_lora_rank=96,
                          index_n_heads=32, index_topk=64, intermediate_size=256, first_k_dense_replace=0,
                          indexer_rope_interleave=interleave)
    else:
        cfg = dataclasses.replace(D.named_config("small"), num_attention_heads=heads, indexer_rope_interleave=interleave)
    torch.manual_seed(5)
    model = D.DSAModel(dataclasses.replace(cfg, num_hidden_layers=1, first_k_dense_replace=0)).eval().cuda().to(dtype)
    return D, cfg, model


def _close(a, b, tol):
    a, b = a.float(), b.float()
    assert float((a - b).abs().max()) <= tol * float(b.abs().max())


@pytest.mark.parametrize("dtype,interleave,heads,production", [
    (torch.bfloat16, False, 16, True), (torch.bfloat16, True, 5, True), (torch.float32, False, 8, False),
    (torch.float32, True, 3, False), (torch.float32, False, 16, True)])
@pytest.mark.parametrize("b,s,cap", [(1, 1, 1), (2, 37, 64), (1, 200, 200)])
def test_fused_full_operands_match_the_separate_chain(dtype, interleave, heads, production, b, s, cap):
    D, cfg, model = _layer(dtype, interleave, heads, production)
    layer = model.layers[0]
    fp8 = dtype == torch.bfloat16
    state = model.init_decode(b, cap, fp8=fp8)  # (stacks the projections of the bf16 model)
    rope = D.RopeCaches(*(t[:s] for t in (state.rope.mla_cos, state.rope.mla_sin, state.rope.idx_cos, state.rope.idx_sin)))
    x = torch.randn(b, s, cfg.hidden_size, device="cuda").to(dtype)
    cache = state.caches[0]
    with torch.no_grad():
        op = layer.full_operands(x, rope, cache=cache)
        part_a = layer.full_operands(x, rope, attention=False)
        part_q = layer.full_operands(x, rope, indexer=False)
    assert op.fused and part_a.fused and part_q.fused
    ref = layer.full_operands(x, rope)  # autograd is on: the separate chain
    assert not ref.fused
    tol = 2.0 ** -7 if fp8 else 1e-5
    with torch.no_grad():
        _close(op.q, ref.q, tol)
        _close(op.kv[:, :s], ref.kv, tol)
        assert torch.equal(part_q.q, op.q) or float((part_q.q.float() - op.q.float()).abs().max()) <= tol * float(op.q.float().abs().max())
        _close(part_q.kv, op.kv[:, :s], tol)
        if fp8:
            from dsa_multi_layer_indexer_b200 import ops
            k8, ks = ops.quantize_e4m3_rowwise(ref.ik.float().contiguous())
            deq = k8.float() * ks.unsqueeze(-1)
            got = op.ik[:, :s].view(torch.float8_e4m3fn).float() * op.ik_scale[:, :s].unsqueeze(-1)
            _close(got, deq, 2.0 ** -4 + tol)  # (one e4m3 step where the bf16 value moved)
            q8, qs = ops.quantize_e4m3_rowwise(ref.iq.float().contiguous())
            _close(op.iq.view(torch.float8_e4m3fn).float() * (op.iw / ref.iw.float()).unsqueeze(-1),
                   q8.float() * qs.unsqueeze(-1), 2.0 ** -4 + 4 * tol)
            assert torch.equal(cache.index_k[:, :s], op.ik[:, :s])
            assert part_a.ik.shape == (b, s, 128) and part_a.q is None
        else:
            _close(op.ik[:, :s], ref.ik, tol)
            _close(op.iq, ref.iq, tol)
            _close(op.iw, ref.iw, tol)
            _close(part_a.iq, ref.iq, tol)


@pytest.mark.parametrize("interleave", [False, True])
def test_prefill_queries_and_latents_are_exact_on_given_operands(interleave):
    """The kernels alone on given inputs: rotary embedding and e4m3 bytes bit for bit."""
    from dsa_multi_layer_indexer_b200 import ops
    from dsa_multi_layer_indexer_b200.dsa_layer import RopeCaches
    from dsa_multi_layer_indexer_b200.rope import apply_rotary, build_rope_cache

    torch.manual_seed(6)
    b, s, H, Hidx, nope = 2, 33, 6, 16, 128
    mc, ms = build_rope_cache(s, 64, 1e4, "cuda", torch.bfloat16)
    ic, is_ = build_rope_cache(s, 128, 1e4, "cuda", torch.bfloat16, interleave=interleave)
    rope = RopeCaches(mc, ms, ic, is_)
    stacked = torch.randn(b * s, H * (nope + 64) + Hidx * 128 + Hidx, device="cuda").to(torch.bfloat16)
    q, iq, w = stacked.split([H * (nope + 64), Hidx * 128, Hidx], dim=1)
    q = q.unflatten(1, (H, nope + 64))
    q_full = torch.zeros(b * s, H, 576, dtype=torch.bfloat16, device="cuda")
    iq8 = torch.zeros(b * s, Hidx, 128, dtype=torch.uint8, device="cuda")
    iw = torch.zeros(b * s, Hidx, device="cuda")
    ops.prefill_queries(q, nope, iq, w, rope, q_full, iq8, iw, s, interleave)
    qr = apply_rotary(q[..., nope:].reshape(b, s, H, 64).transpose(1, 2), mc, ms).transpose(1, 2).reshape(b * s, H, 64)
    assert torch.equal(q_full[..., 512:], qr) and float(q_full[..., :512].float().abs().max()) == 0.0
    iqr = apply_rotary(iq.reshape(b, s, Hidx, 128).transpose(1, 2), ic, is_, interleave=interleave).transpose(1, 2)
    want, scale = ops.quantize_e4m3_rowwise(iqr.reshape(b * s, Hidx, 128).float().contiguous())
    assert torch.equal(iq8, want.view(torch.uint8))
    assert torch.equal(iw, scale * w.float())
    ik = torch.randn(b * s, 128, device="cuda").to(torch.bfloat16)
    ik_out = torch.zeros(b, s + 5, 128, dtype=torch.uint8, device="cuda")
    ik_scale = torch.zeros(b, s + 5, device="cuda")
    ops.prefill_latents(None, None, ik, None, None, rope, None, None, ik_out, ik_scale, s, interleave, 1e-6)
    ikr = apply_rotary(ik.view(b, 1, s, 128), ic, is_, interleave=interleave).view(b, s, 128)
    want, scale = ops.quantize_e4m3_rowwise(ikr.float().contiguous())
    assert torch.equal(ik_out[:, :s], want.view(torch.uint8)) and torch.equal(ik_scale[:, :s], scale)
    assert int(ik_out[:, s:].sum()) == 0
