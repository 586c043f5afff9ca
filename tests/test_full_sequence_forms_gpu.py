"""GPU tests of full-sequence layers in the forms that the fused native chain does not take: whatever a
module of the layer has been made into (other weight types, hooks, replacements), forward and prefill must
give what calling the modules one after the other gives. That path still runs when autograd is on, so it is
the reference here, bit for bit."""

from __future__ import annotations

import dataclasses

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


def make_model(D, dtype, layers=1, **kw):
    """Small layers whose norm weights are not ones (but numbers of every type used here)."""
    if dtype == torch.bfloat16:
        cfg = D.DSAConfig(hidden_size=192, num_hidden_layers=layers, num_attention_heads=16, q_lora_rank=96, index_n_heads=32,
                          index_topk=64, intermediate_size=256, first_k_dense_replace=0, **kw)
    else:
        cfg = dataclasses.replace(D.named_config("small"), num_hidden_layers=layers, first_k_dense_replace=0, **kw)
    torch.manual_seed(5)
    model = D.DSAModel(cfg).eval()
    with torch.no_grad():
        for m in norms_of(model):
            m.weight.copy_(1.0 + torch.randint(-32, 33, m.weight.shape) / 64.0)
    return model.cuda().to(dtype)


def norms_of(model):
    return [m for m in model.modules() if type(m).__name__ == "RMSNorm"]


def tokens(model, b, s):
    torch.manual_seed(6)
    return torch.randn(b, s, model.config.hidden_size, device="cuda").to(model.layers[0].q_a_proj.weight.dtype)


def operands(model, x, cache=None):
    """(q, kv, ik, iq, iw) of layer 0 as computed, whatever the path."""
    op = model.layers[0].full_operands(x, model._build_rope(x.shape[1], x.device, x.dtype), cache=cache)
    return op, [t.detach() for t in (op.q, op.kv, op.ik, op.iq, op.iw)]


def check_against_modules(model, x):
    """full_operands without gradients must be the modules' own results."""
    with torch.no_grad():
        op, got = operands(model, x)
    ref_op, want = operands(model, x)  # autograd is on: the modules one by one
    assert not op.fused and not ref_op.fused
    assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("dtype,other", [(torch.bfloat16, torch.float32), (torch.float32, torch.bfloat16)])
@pytest.mark.parametrize("which", ["all", "q_a_layernorm", "kv_a_layernorm"])
def test_norm_weights_of_another_type(D, dtype, other, which):
    mode, cold = D.ScheduleMode.LAGGED_FUSED, D.ColdStartPolicy.DENSE  # (no selection, whose cutoff rounding moves)
    model = make_model(D, dtype)
    x = tokens(model, 2, 70)
    with torch.no_grad():
        same_type = model(x, mode, cold)
    for m in norms_of(model) if which == "all" else [getattr(model.layers[0], which)]:
        m.to(other)
    check_against_modules(model, x)
    with torch.no_grad():
        got = model(x, mode, cold)
    filled = model.prefill(model.init_decode(2, 80, fp8=dtype == torch.bfloat16), x, mode, cold)
    # the same numbers as with weights of the activations' type, by other kernels: a handful of bf16 roundings
    # (2^-8 each); fp32 sums in another order
    tol = 3e-2 if dtype == torch.bfloat16 else 1e-4
    for y in (got, filled):
        assert float((y.float() - same_type.float()).norm()) <= tol * float(same_type.float().norm())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("name,row", [("q_a_layernorm", 0), ("kv_a_layernorm", 1)])
@pytest.mark.parametrize("change", ["hook", "pre_hook", "subclass", "forward", "eps"])
def test_changed_latent_norms_are_honoured(D, dtype, name, row, change):
    model = make_model(D, dtype)
    x = tokens(model, 1, 33)
    with torch.no_grad():
        plain = operands(model, x)[1]
    m = getattr(model.layers[0], name)
    if change == "hook":
        m.register_forward_hook(lambda mod, a, o: o * 2)
    elif change == "pre_hook":
        m.register_forward_pre_hook(lambda mod, a: (a[0].sin(),))
    elif change == "subclass":
        class Doubled(type(m)):
            def forward(self, t):
                return super().forward(t) * 2

        m.__class__ = Doubled
    elif change == "forward":
        inner = m.forward
        m.forward = lambda t: inner(t) * 2
    else:
        m.eps = 0.5
    check_against_modules(model, x)
    with torch.no_grad():
        changed = operands(model, x)[1]
    assert not torch.allclose(changed[row].float(), plain[row].float(), rtol=2e-2, atol=1e-3)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_gradients_after_a_pass_in_inference_mode(D, dtype):
    """The rotary tables that one pass leaves for the next serve every mode."""
    mode, cold = D.ScheduleMode.BASELINE, D.ColdStartPolicy.EAGER
    model = make_model(D, dtype)
    x = tokens(model, 1, 40)
    with torch.inference_mode():
        first = model(x, mode, cold)
    x = x.clone().requires_grad_(True)
    model(x, mode, cold)  # (apply_rotary saves its tables for the backward pass)
    shorter = model(x[:, :17], mode, cold)
    assert shorter.shape == (1, 17, model.config.hidden_size) and not model._rope_kept[1].mla_cos.is_inference()
    with torch.inference_mode():
        assert torch.equal(model(x, mode, cold), first)


@pytest.mark.parametrize("name", ["q_a_proj", "kv_a_proj", "index_k_proj", "q_b_proj", "index_q_proj", "index_weights_proj", "kv_b_proj",
                                  "o_proj", "gate_proj", "up_proj", "down_proj", "q_a_layernorm", "kv_a_layernorm"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_weights_on_another_device_are_refused(D, dtype, name):
    """Never read by a kernel: torch's own error, or that of the argument checks."""
    model = make_model(D, dtype)
    x = tokens(model, 1, 33)
    getattr(model.layers[0], name).cpu()
    with torch.no_grad(), pytest.raises((RuntimeError, ValueError)):
        model(x, D.ScheduleMode.BASELINE, D.ColdStartPolicy.EAGER)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_operands_of_other_widths_are_refused(D, dtype):
    model = make_model(D, dtype)
    layer, hidden = model.layers[0], model.config.hidden_size
    x = tokens(model, 1, 33)
    rope = model._build_rope(33, x.device, dtype)
    refused = pytest.raises((RuntimeError, ValueError))
    with torch.no_grad():
        for width in (hidden - 4, hidden + 4, 2 * hidden):
            with refused:
                layer.full_operands(torch.zeros(1, 33, width, device="cuda", dtype=dtype), rope)
            with refused:
                layer.mlp(torch.zeros(1, 33, width, device="cuda", dtype=dtype))
        c_q = layer.q_latent(x)
        for bad in (c_q.cpu(), c_q[..., :-4], c_q.double()):
            with refused:
                layer.full_operands(x, rope, c_q=bad)
        for field in ("mla_cos", "mla_sin", "idx_cos", "idx_sin"):
            narrow = dataclasses.replace(rope, **{field: getattr(rope, field)[:, :-2].contiguous()})
            with refused:
                layer.full_operands(x, narrow)
        wide = torch.nn.Linear(model.config.q_lora_rank, model.config.index_n_heads * model.config.index_head_dim - 4, bias=False)
        layer.index_q_proj = wide.cuda().to(dtype)
        with refused:
            layer.full_operands(x, rope)


@pytest.mark.parametrize("nope", [30, 33, 36])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_query_heads_of_any_width(D, dtype, nope):
    """Heads whose rotary part does not start on 8 bytes (bf16) take the modules, the others the fused chain."""
    model = make_model(D, dtype, qk_nope_head_dim=nope)
    x = tokens(model, 2, 41)
    mode, cold = D.ScheduleMode.LAGGED_FUSED, D.ColdStartPolicy.DENSE
    state = model.init_decode(2, 48, fp8=dtype == torch.bfloat16)  # (bf16: stacked projections)
    filled = model.prefill(state, x, mode, cold)
    with torch.no_grad():
        got = model(x, mode, cold)
    want = model(x, mode, cold).detach()  # autograd is on: the modules
    tol = 3e-2 if dtype == torch.bfloat16 else 1e-4
    for y in (got, filled):
        assert float((y.float() - want.float()).norm()) <= tol * float(want.float().norm())


def _as(cache, change):
    """A cache of another form than new_cache's, same contents after a fill."""
    def strided(t):
        return torch.zeros(t.shape[0], t.shape[1], 2, *t.shape[2:], dtype=t.dtype, device=t.device)[:, :, 1]

    def wide(t):  # one prompt for three sequences
        return torch.zeros(3, *t.shape[1:], dtype=t.dtype, device=t.device)

    if change == "fp32 rows":
        return dataclasses.replace(cache, kv=cache.kv.float())
    if change == "bf16 rows":
        return dataclasses.replace(cache, kv=cache.kv.to(torch.bfloat16))
    make = {"broadcast": wide, "host": lambda t: torch.zeros_like(t, device="cpu"), "strided": strided}[change]
    return type(cache)(make(cache.index_k), None if cache.k_scale is None else make(cache.k_scale), make(cache.kv))


@pytest.mark.parametrize("dtype,change", [(torch.bfloat16, c) for c in ("broadcast", "host", "strided", "fp32 rows")] + [
    (torch.float32, c) for c in ("broadcast", "host", "strided", "bf16 rows")])
def test_caches_of_other_forms_are_filled(D, dtype, change):
    model = make_model(D, dtype)
    layer, x = model.layers[0], tokens(model, 1, 37)
    rope = model._build_rope(37, x.device, dtype)
    plain = layer.new_cache(1, 40, x.device, fp8=dtype == torch.bfloat16)
    other = _as(plain, change)
    with torch.no_grad():
        layer.fill_cache(plain, x, rope)
        layer.fill_cache(other, x, rope)
    # (by other kernels: a unit in the last place of the type that is stored)
    for a, b, scale in ((plain.kv, other.kv, None), (plain.index_k, other.index_k, (plain.k_scale, other.k_scale))):
        a, b = a[:, :37], b[:, :37]
        if scale and scale[0] is not None:
            a, b = (t.view(torch.float8_e4m3fn).float() * s[:, :37, None] for t, s in ((a, scale[0]), (b.contiguous(), scale[1])))
        tol = 2.0 ** -4 if scale and scale[0] is not None else 2.0 ** -7 if torch.bfloat16 in (a.dtype, b.dtype) else 1e-5
        a, b = a.float().cpu().expand(b.shape), b.float().cpu()
        assert float((a - b).abs().max()) <= tol * float(a.abs().max()) and float(b.abs().max()) > 0
    short = type(plain)(plain.index_k[:, :30], None if plain.k_scale is None else plain.k_scale[:, :30], plain.kv[:, :30])
    with torch.no_grad(), pytest.raises((RuntimeError, ValueError)):
        layer.fill_cache(short, x, rope)


def test_schedules_and_policies_are_members_not_their_names(D):
    """"baseline" and "eager" equal the members they name; taken by equality in one place and by identity in the
    next they would run the other schedule."""
    model = make_model(D, torch.float32, layers=2)
    x = tokens(model, 1, 24)
    with torch.no_grad():
        for mode, cold in (("baseline", D.ColdStartPolicy.EAGER), ("unknown", D.ColdStartPolicy.EAGER),
                           (D.ScheduleMode.LAGGED_FUSED, "eager"), (D.ScheduleMode.LAGGED_FUSED, "unknown")):
            with pytest.raises(ValueError):
                model(x, mode, cold)
        want = model(x, D.ScheduleMode.LAGGED_FUSED, D.ColdStartPolicy.EAGER)
        assert torch.equal(model(x, "lagged_fused", D.ColdStartPolicy.EAGER), want)
    state = model.init_decode(1, 32, fp8=False)
    assert torch.equal(model.prefill(state, x, "lagged", D.ColdStartPolicy.EAGER), want)  # (prefill: all but BASELINE lag)


def test_a_model_without_layers_is_its_final_norm(D):
    model = make_model(D, torch.float32, layers=0)
    x = torch.randn(2, 9, model.config.hidden_size, device="cuda")
    with torch.no_grad():
        assert torch.equal(model(x, D.ScheduleMode.BASELINE), model.final_norm(x))


class ScaledNorm(torch.nn.Module):
    """A norm that is no RMSNorm and knows nothing of residuals."""

    def forward(self, t):
        return (t.float() * torch.rsqrt(t.float().pow(2).mean(-1, keepdim=True) + 1e-6) * 1.5).to(t.dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("change", ["hook", "replaced", "global hook"])
def test_residual_norms_are_called_as_modules(D, dtype, change):
    """attn_norm, ffn_norm and final_norm: hooks see every call, replacements take their place."""
    model = make_model(D, dtype, layers=2)
    x = tokens(model, 2, 24)
    mode, cold = D.ScheduleMode.BASELINE, D.ColdStartPolicy.DENSE
    places = [(l, n) for l in model.layers for n in ("attn_norm", "ffn_norm")] + [(model, "final_norm")]
    seen = []
    if change == "replaced":
        for owner, name in places:
            setattr(owner, name, ScaledNorm())
    elif change == "hook":
        for owner, name in places:
            getattr(owner, name).register_forward_hook(lambda m, a, o: seen.append(m) or o * 1.5)
    else:
        norms = [getattr(owner, name) for owner, name in places]
        handle = torch.nn.modules.module.register_module_forward_hook(
            lambda m, a, o: seen.append(m) if any(m is n for n in norms) else None)
    try:
        with torch.no_grad():
            got = model(x, mode, cold)
        calls = list(seen)
        state = model.init_decode(2, 32, fp8=dtype == torch.bfloat16)
        filled = model.prefill(state, x[:, :23], mode, cold)
        seen.clear()
        step = model.decode_step(state, x[:, 23], mode, cold)
        if change != "replaced":
            in_order = [getattr(owner, name) for owner, name in places]
            assert [id(m) for m in calls] == [id(m) for m in in_order] == [id(m) for m in seen]
        want = model(x, mode, cold).detach()  # autograd is on: the modules one by one
    finally:
        if change == "global hook":
            handle.remove()
    tol = 3e-2 if dtype == torch.bfloat16 else 1e-3  # (topk keys of a cutoff within rounding may change places)
    for a, b in ((got, want), (filled, want[:, :23]), (step, want[:, 23])):
        assert float((a.float() - b.float()).norm()) <= tol * float(b.float().norm())


class ScaledWeight(torch.nn.Parameter):
    """A weight with a product of its own, as quantised weights have: F.linear through __torch_function__."""

    @classmethod
    def __torch_function__(cls, func, types, args=(), kwargs=None):
        with torch._C.DisableTorchFunctionSubclass():
            if func is torch.nn.functional.linear:
                return func(args[0], args[1].as_subclass(torch.Tensor) * 1.5)
            return func(*args, **(kwargs or {}))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("change", ["forward", "weight", "global hook"])
@pytest.mark.parametrize("name", ["o_proj", "gate_proj", "up_proj", "down_proj"])
def test_changed_projections_are_honoured(D, dtype, change, name):
    """A patched forward (as offloading and adapter libraries do), a weight of another tensor class, hooks of
    every module: forward without gradients, prefill and the decode step against the module path."""
    model = make_model(D, dtype)
    x = tokens(model, 2, 24)
    mode, cold = D.ScheduleMode.LAGGED_FUSED, D.ColdStartPolicy.DENSE
    with torch.no_grad():
        plain = model(x, mode, cold)
    layer, fp8 = model.layers[0], dtype == torch.bfloat16
    m = getattr(layer, name)
    if change == "forward":
        inner = m.forward
        m.forward = lambda t: inner(t) * 1.5
    elif change == "weight":
        m.weight = ScaledWeight(m.weight.detach())
    else:
        handle = torch.nn.modules.module.register_module_forward_hook(lambda mod, a, o: o * 1.5 if mod is m else None)
    try:
        with torch.no_grad():
            got = model(x, mode, cold)
        state = model.init_decode(2, 32, fp8=fp8)
        outs = [(got, slice(None)), (model.prefill(state, x[:, :23], mode, cold), slice(0, 23))]
        if name in ("o_proj", "down_proj"):  # (the decode step reads the weights of gate and up itself)
            outs.append((model.decode_step(state, x[:, 23], mode, cold)[:, None], slice(23, 24)))
        want = model(x, mode, cold).detach()  # autograd is on: the modules one by one
    finally:
        if change == "global hook":
            handle.remove()
    tol = 3e-2 if dtype == torch.bfloat16 else 1e-3
    for y, rows in outs:
        ref = want[:, rows].float()
        assert float((y.float() - ref).norm()) <= tol * float(ref.norm())
    assert float((want.float() - plain.float()).norm()) > 5e-2 * float(plain.float().norm())


@pytest.mark.parametrize("name", ["q_a_proj", "kv_a_proj", "index_k_proj", "q_b_proj", "index_q_proj", "index_weights_proj"])
@pytest.mark.parametrize("how", ["parameter", "data"])
def test_a_weight_replaced_after_stacking_is_the_one_that_runs(D, name, how):
    """init_decode stacks three weights each; prompts and decode steps must notice that one of them (the middle
    one too) has been given other memory."""
    model = make_model(D, torch.bfloat16)
    state = model.init_decode(1, 40)
    layer, x = model.layers[0], tokens(model, 1, 24)
    m = getattr(layer, name)
    new = torch.randn_like(m.weight) * 0.2
    if how == "parameter":
        m.weight = torch.nn.Parameter(new)
    else:
        m.weight.data = new
    rope = model._build_rope(24, x.device, x.dtype)
    with torch.no_grad():
        op = layer.full_operands(x, rope)
        q, iq, iw = layer.decode_project(x[:, 5], state.rope, torch.full((1,), 5, device="cuda"), state.caches[0], state.batch_index)
    want = layer.full_operands(x, rope)  # autograd is on: the modules
    assert op.fused and not want.fused
    f8 = lambda t: t.view(torch.float8_e4m3fn).float()

    def near(a, b, tol=3e-2):
        assert float((a.float() - b.detach().float()).norm()) <= tol * float(b.detach().float().norm())

    # (a bf16 rounding apart; e4m3 bytes against the unquantised keys: half a step of 2^-3 at most)
    near(op.q, want.q)
    near(op.kv, want.kv)
    near(f8(op.ik) * op.ik_scale[..., None], want.ik, 6e-2)
    near(f8(op.iq) * op.iw[..., None], want.iq * want.iw[..., None], 6e-2)
    near(q[0], want.q[5])
    near(f8(iq[0]) * iw[0, :, None], want.iq[5] * want.iw[5, :, None], 6e-2)
    near(state.caches[0].kv[0, 5], want.kv[0, 5])
    near(f8(state.caches[0].index_k[0, 5]) * state.caches[0].k_scale[0, 5], want.ik[0, 5], 6e-2)
