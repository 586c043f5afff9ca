"""Performance cases of the DSA decode hot path and of the layers and models around it.

Each case is one call (or one short sequence of calls) that a program built on this package makes,
through the package's public entry points:

* ``step``     one layer's decode hot path (``decode.HotPathState``): indexer scan, top-k, sparse MLA
* ``host``     the same step with the operands and the result in host memory (``decode.HostDecoder``)
* ``serve``    the serving form over paged caches (``serving.forward_hide_operands``,
               ``ops.latent_append``, ``serving.fused_hide_decode_paged``)
* ``verify``   several query tokens of one sequence through the extension-style launch
               (``kernels_ext``) and the selection that follows it
* ``prefill``  ``DSAModel.prefill`` of a prompt: full-sequence layers, caches filled on the way
* ``decode``   one token per sequence through a stack of layers, replayed from a CUDA graph
               (``DSAModel.capture_decode``)
* ``forward``  ``DSAModel.forward`` of the small fp32 preset
"""

from __future__ import annotations

import dataclasses
import math

import torch

import dsa_multi_layer_indexer_b200 as dsa
from dsa_multi_layer_indexer_b200 import kernels_ext, ops, serving
from dsa_multi_layer_indexer_b200.decode import HostDecoder, HotPathState, LayerCache

SM_SCALE = 192 ** -0.5
PAGE = ops.PAGE_TOKENS
DEV = "cuda"


# --------------------------------------------------------------------------- the cases
def listed():
    return [
        # The smallest step: one request at a 4K context, 16 MLA heads (one rank's share of 128 heads
        # over eight GPUs); the step is replayed from a graph, so launches and latency are all there is.
        dict(name="step_4k", kind="step", rows=1, heads=16, index_heads=64, ctx=4096, topk=2048, fp8=False, graph=True),
        # The headline step: batch 1 at 128K, 128 heads.
        dict(name="step_128k", kind="step", rows=1, heads=128, index_heads=64, ctx=131072, topk=2048, fp8=False,
             graph=True),
        # The long-context step: 256K keys, 64 heads and 32 indexer heads (the glm5 preset's counts).
        dict(name="step_256k", kind="step", rows=1, heads=64, index_heads=32, ctx=262144, topk=2048, fp8=False,
             graph=True),
        # A small ragged batch called without a graph, odd capacity.
        dict(name="step_batch8_eager", kind="step", rows=8, heads=64, index_heads=32, ctx=20011, topk=2048, fp8=False,
             graph=False),
        # A host-side caller: operands in pinned host memory, result back there, every step.
        dict(name="host_128k", kind="host", heads=128, index_heads=64, ctx=131072, topk=2048),
        # Batched serving: 32 ragged requests of 16K to 64K tokens, paged FP8 index keys, fp8 latent pool.
        dict(name="serve_32_fp8", kind="serve", rows=32, heads=128, index_heads=64, ctx=65536, topk=2048, fp8=True),
        # A lightly loaded server: 3 requests, bf16 latent pool, table of an odd number of pages.
        dict(name="serve_3_bf16", kind="serve", rows=3, heads=64, index_heads=32, ctx=9152, topk=2048, fp8=False),
        # Multi-token decode of one sequence (4 drafted tokens checked at once) at 32K.
        dict(name="verify_4x32k", kind="verify", rows=4, heads=128, index_heads=64, ctx=32768, topk=2048),
        # A short prompt (no row is longer than top-k): two layers of the glm5 preset, each layer
        # attending its own selection.
        dict(name="prefill_glm5_700", kind="prefill", config="glm5", layers=2, batch=1, seq=700, lagged=False),
        # A long prompt: two layers of the deepseek preset under the lagged schedule, odd length.
        dict(name="prefill_deepseek_4099", kind="prefill", config="deepseek", layers=2, batch=1, seq=4099, lagged=True),
        # The 8-layer stack at 128K, one token, lagged schedule, one graph per step.
        dict(name="decode_stack_128k", kind="decode", config="deepseek", layers=8, batch=1, ctx=131072, lagged=True,
             overlap="chained"),
        # The small fp32 preset, full sequence: what a developer runs to compare schedules.
        dict(name="forward_small_fp32", kind="forward", batch=2, seq=512, lagged=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["step", "host", "serve", "verify", "prefill", "decode", "forward"],
                       [30, 6, 18, 8, 18, 12, 8])[0]
    heads, index_heads = rng.choice([(16, 64), (32, 64), (64, 32), (64, 64), (128, 64)])
    topk = rng.choice([512, 1024, 2048, 2048, 2048])
    if kind == "step":
        rows = rng.choice([1, 1, 1, 2, 3, 4, 7, 8, 16])
        ctx = _log(rng, 2048, min(262144, 524288 // rows))
        return dict(kind=kind, rows=rows, heads=heads, index_heads=index_heads, ctx=ctx, topk=topk,
                    fp8=rng.random() < 0.3, graph=rng.random() < 0.6)
    if kind == "host":
        return dict(kind=kind, heads=heads, index_heads=index_heads, ctx=_log(rng, 4096, 262144), topk=topk)
    if kind == "serve":
        rows = _log(rng, 1, 32)
        ctx = _log(rng, 4096, min(131072, 2097152 // rows)) // PAGE * PAGE
        return dict(kind=kind, rows=rows, heads=heads, index_heads=index_heads, ctx=ctx, topk=topk,
                    fp8=rng.random() < 0.6)
    if kind == "verify":
        return dict(kind=kind, rows=rng.randint(2, 8), heads=heads, index_heads=index_heads,
                    ctx=_log(rng, 4096, 131072), topk=topk)
    if kind == "prefill":
        batch = rng.choice([1, 1, 1, 2, 3])
        return dict(kind=kind, config=rng.choice(["deepseek", "glm5"]), layers=rng.choice([1, 2]), batch=batch,
                    seq=_log(rng, 128, 4000 // batch), lagged=rng.random() < 0.5)
    if kind == "decode":
        batch = rng.choice([1, 1, 2, 3, 4, 8])
        return dict(kind=kind, config=rng.choice(["deepseek", "glm5"]), layers=rng.randint(2, 6), batch=batch,
                    ctx=_log(rng, 32768, 131072), lagged=rng.random() < 0.7,
                    overlap=rng.choice(["chained", "streams"]))
    return dict(kind=kind, batch=rng.randint(1, 4), seq=_log(rng, 48, 700), lagged=rng.random() < 0.6)


# --------------------------------------------------------------------------- inputs
def _ragged(rows, ctx, gen):
    """Lengths spread evenly over [ctx / 4, ctx], in a random order (their sum is known without the
    seed); a single row is full."""
    lens = torch.tensor(_length_list(rows, ctx), dtype=torch.int32, device=DEV)
    return lens[torch.randperm(rows, generator=gen, device=DEV)].contiguous()


def _length_list(rows, ctx):
    if rows == 1:
        return [ctx]
    return [ctx // 4 + (ctx - ctx // 4) * i // (rows - 1) for i in range(rows)]


def _randn(gen, *shape):
    return torch.randn(*shape, device=DEV, generator=gen)


def _index_operands(gen, rows, index_heads):
    """e4m3 queries and head weights with the query scale folded in."""
    q8, sq = ops.quantize_e4m3_rowwise(_randn(gen, rows, index_heads, 128))
    return q8, (sq * _randn(gen, rows, index_heads) / 8).contiguous()


def _index_keys(gen, n_seq, cap):
    k8, scale = ops.quantize_e4m3_rowwise(_randn(gen, n_seq, cap, 128))
    return k8.view(torch.uint8), scale


def _rope_tables(cap):
    inv = 10000.0 ** (-torch.arange(32, device=DEV, dtype=torch.float32) / 32)
    ang = torch.arange(cap, device=DEV, dtype=torch.float32)[:, None] * inv[None, :]
    return torch.cos(ang).contiguous(), torch.sin(ang).contiguous()


def _latent_rows(gen, n, fp8):
    """``n`` cached latent rows: bf16 ``[n, 576]``, or the 656-byte fp8-packed rows."""
    kv_a = torch.empty(n, 576, dtype=torch.bfloat16, device=DEV)
    for i in range(0, n, 1 << 18):
        kv_a[i:i + (1 << 18)] = _randn(gen, min(1 << 18, n - i), 576).to(torch.bfloat16)
    if not fp8:
        return kv_a
    pool = torch.zeros(n, 656, dtype=torch.uint8, device=DEV)
    cos, sin = _rope_tables(1)
    ones, slots = torch.ones(512, device=DEV), torch.arange(n, device=DEV)
    ops.latent_append(kv_a, ones, 1e-6, cos, sin, torch.zeros(n, dtype=torch.int64, device=DEV), slots, pool)
    return pool


def _hot_path(case, gen, rows, fp8):
    state = HotPathState(rows, case["heads"], case["index_heads"], case["ctx"], case["topk"], DEV)
    index_k, k_scale = _index_keys(gen, rows, case["ctx"])
    kv = _latent_rows(gen, rows * case["ctx"], fp8)
    cache = LayerCache(index_k, k_scale, kv.view(rows, case["ctx"], -1))
    q8, w = _index_operands(gen, rows, case["index_heads"])
    state.index_q.copy_(q8.view(torch.uint8))
    state.index_w.copy_(w)
    state.q.copy_(_randn(gen, rows, case["heads"], 576).to(torch.bfloat16))
    state.seq_lens.copy_(_ragged(rows, case["ctx"], gen))
    return state, cache


def _model(name, layers, seed, dtype):
    cfg = dataclasses.replace(dsa.named_config(name), num_hidden_layers=layers, first_k_dense_replace=0)
    torch.manual_seed(seed)
    with torch.device(DEV):
        return dsa.DSAModel(cfg).to(dtype).eval()


def prepare(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "step":
        s["state"], s["cache"] = _hot_path(case, gen, case["rows"], case["fp8"])
        s["graph"] = s["state"].capture(s["cache"], SM_SCALE) if case["graph"] else None
    elif kind == "host":
        state, cache = _hot_path(case, gen, 1, False)
        dec = s["decoder"] = HostDecoder(state, cache, SM_SCALE)
        q8, w = _index_operands(gen, 1, case["index_heads"])
        dec.h_index_q.copy_(q8.view(torch.uint8))
        dec.h_index_w.copy_(w)
        dec.h_q.copy_(_randn(gen, 1, case["heads"], 576).to(torch.bfloat16))
    elif kind == "serve":
        rows, ctx = case["rows"], case["ctx"]
        per_row = ctx // PAGE
        table = torch.randperm(rows * per_row, generator=gen, device=DEV).int().view(rows, per_row)
        pages = torch.empty(rows * per_row, ops.INDEX_PAGE_BYTES, dtype=torch.uint8, device=DEV)
        for r in range(rows):
            k8, scale = _index_keys(gen, 1, ctx)
            mine = table[r].long()
            pages[mine, :PAGE * 128] = k8.view(per_row, PAGE * 128)
            pages[mine, PAGE * 128:] = scale.view(torch.uint8).view(per_row, PAGE * 4)
        lens = _ragged(rows, ctx, gen)
        cos, sin = _rope_tables(ctx)
        k = min(case["topk"], ctx // 4)
        incumbent = torch.full((rows, case["topk"]), -1, dtype=torch.int32, device=DEV)
        for r in range(rows):  # the previous layer's selection, as slot numbers in ascending position
            pos = torch.randperm(int(lens[r]), generator=gen, device=DEV)[:k].sort().values
            incumbent[r, :k] = table[r][pos // PAGE] * PAGE + (pos % PAGE).int()
        last = lens.long() - 1
        s.update(
            q_proj=_randn(gen, rows, case["index_heads"], 128).to(torch.bfloat16),
            k_proj=_randn(gen, rows, 128).to(torch.bfloat16), gates=_randn(gen, rows, case["index_heads"]),
            norm_w=torch.ones(128, device=DEV), norm_b=torch.zeros(128, device=DEV), cos=cos, sin=sin,
            positions=last, pages=pages, table=table, lens=lens, incumbent=incumbent,
            slots=table.gather(1, (last // PAGE)[:, None])[:, 0].long() * PAGE + last % PAGE,
            kv_a=_randn(gen, rows, 576).to(torch.bfloat16), kv_norm_w=torch.ones(512, device=DEV),
            pool=_latent_rows(gen, rows * ctx, case["fp8"]), fmt="fp8" if case["fp8"] else "bf16",
            q=_randn(gen, 1, rows, case["heads"], 576).to(torch.bfloat16))
    elif kind == "verify":
        rows, ctx, topk = case["rows"], case["ctx"], case["topk"]
        nsplit = ops.default_nsplit(rows, case["heads"], topk)
        index_k, k_scale = _index_keys(gen, 1, ctx)
        iq, iw = _index_operands(gen, rows, case["index_heads"])
        k = min(topk, ctx - rows)
        idx = torch.stack([torch.randperm(ctx - rows, generator=gen, device=DEV)[:k].sort().values
                           for _ in range(rows)]).int()
        attend = torch.full((rows, topk), -1, dtype=torch.int32, device=DEV)
        attend[:, :k] = idx
        s.update(
            ext=kernels_ext.build(), shape=(rows, ctx, case["heads"], case["index_heads"], topk, nsplit),
            q=_randn(gen, rows, case["heads"], 576).to(torch.bfloat16), kv=_latent_rows(gen, ctx, False),
            attend=attend, index_q=iq.view(torch.uint8), index_w=iw, index_k=index_k[0], k_scale=k_scale[0],
            part=kernels_ext.alloc_part(rows, case["heads"], nsplit, DEV),
            slab=torch.empty(rows, ctx, device=DEV), hist=torch.zeros(rows, ops.HIST_BINS, dtype=torch.int32, device=DEV),
            out=torch.empty(rows, case["heads"], 512, dtype=torch.bfloat16, device=DEV),
            lens=torch.arange(ctx - rows + 1, ctx + 1, dtype=torch.int32, device=DEV),
            selected=torch.empty(rows, topk, dtype=torch.int32, device=DEV), ws=ops.topk_workspace(rows, ctx, DEV))
    elif kind == "prefill":
        model = s["model"] = _model(case["config"], case["layers"], seed, torch.bfloat16)
        s["state"] = model.init_decode(case["batch"], case["seq"] + 256)
        s["x"] = _randn(gen, case["batch"], case["seq"], model.config.hidden_size).to(torch.bfloat16)
        s["mode"] = dsa.ScheduleMode.LAGGED_FUSED if case["lagged"] else dsa.ScheduleMode.BASELINE
    elif kind == "decode":
        model = s["model"] = _model(case["config"], case["layers"], seed, torch.bfloat16)
        state = s["state"] = model.init_decode(case["batch"], case["ctx"])
        for c in state.caches:  # a prefix of three quarters of the capacity, as a prefill would leave it
            index_k, scale = _index_keys(gen, case["batch"], case["ctx"])
            c.index_k.copy_(index_k)
            c.k_scale.copy_(scale)
            c.kv.copy_(_latent_rows(gen, case["batch"] * case["ctx"], False).view(c.kv.shape))
        state.positions.fill_(_start(case))
        state.seq_lens.fill_(_start(case))
        mode = dsa.ScheduleMode.LAGGED_FUSED if case["lagged"] else dsa.ScheduleMode.BASELINE
        s["graph"], s["x_in"], s["x_out"] = model.capture_decode(
            state, mode, dsa.ColdStartPolicy.EAGER, "chained" if case["overlap"] == "chained" else True)
        s["x"] = _randn(gen, case["batch"], model.config.hidden_size).to(torch.bfloat16)
    elif kind == "forward":
        torch.manual_seed(seed)
        with torch.device(DEV):
            s["model"] = dsa.DSAModel(dsa.named_config("small")).eval()
        s["x"] = _randn(gen, case["batch"], case["seq"], s["model"].config.hidden_size)
        s["mode"] = dsa.ScheduleMode.LAGGED_FUSED if case["lagged"] else dsa.ScheduleMode.BASELINE
    else:
        raise ValueError(kind)
    return s


def _start(case):
    return case["ctx"] * 3 // 4


# --------------------------------------------------------------------------- one pass
def run(s):
    kind = s["kind"]
    if kind == "step":
        state = s["state"]
        if s["graph"] is not None:
            s["graph"].replay()
        else:
            state.run(s["cache"], SM_SCALE)
        return state.out, state.indices
    if kind == "host":
        out = s["decoder"].step()
        return out, s["decoder"].h_indices
    if kind == "serve":
        iq, iw, pages, table, lens, cap = serving.forward_hide_operands(
            s["q_proj"], s["k_proj"], s["gates"], s["norm_w"], s["norm_b"], 1e-6, s["cos"], s["sin"], s["positions"],
            s["pages"], s["table"], s["lens"])
        ops.latent_append(s["kv_a"], s["kv_norm_w"], 1e-6, s["cos"], s["sin"], s["positions"], s["slots"], s["pool"],
                          fmt=s["fmt"])
        attn, nxt = serving.fused_hide_decode_paged(
            s["q"], s["pool"], s["incumbent"], iq, iw, pages, table, lens, cap, SM_SCALE, None)
        return attn, nxt, iq, iw, s["pages"], s["pool"]
    if kind == "verify":
        rows, ctx, heads, index_heads, topk, nsplit = s["shape"]
        acc, m, l = s["part"]
        s["ext"].launch_fused_sparse_splitk(
            s["q"], s["kv"], s["attend"], s["index_q"], s["index_k"], s["index_w"], s["k_scale"], acc, m, l, s["slab"],
            s["hist"], s["out"], rows, ctx, heads, index_heads, topk, nsplit, SM_SCALE, 2, 1, 0)
        ops.topk_select(s["slab"], topk, s["lens"], hist=s["hist"], out_idx=s["selected"], workspace=s["ws"])
        return s["out"], s["selected"]
    if kind == "prefill":
        state = s["state"]
        hidden = s["model"].prefill(state, s["x"], s["mode"], dsa.ColdStartPolicy.EAGER)
        return hidden, _caches(state)
    if kind == "decode":
        s["x_in"].copy_(s["x"])
        s["graph"].replay()
        return s["x_out"], _caches(s["state"])
    with torch.no_grad():
        return s["model"](s["x"], s["mode"], dsa.ColdStartPolicy.EAGER)


def _caches(state):
    """The updated caches; the index keys as the e4m3 numbers that their bytes are."""
    return [(c.index_k.view(torch.float8_e4m3fn), c.k_scale, c.kv) for c in state.caches]


# --------------------------------------------------------------------------- what a pass cannot do without
def _attention(keys, heads, row_bytes, distinct=None):
    """``keys``: attended keys summed over the query rows; ``distinct``: latent rows read."""
    distinct = keys if distinct is None else distinct
    return distinct * row_bytes, keys * heads * 2 * (576 + 512)


def _params(cfg):
    h = cfg.num_attention_heads
    return (cfg.hidden_size * (cfg.q_lora_rank + 576 + cfg.index_head_dim + 3 * cfg.intermediate_size)
            + cfg.q_lora_rank * (h * (cfg.qk_nope_head_dim + 64) + cfg.index_n_heads * (cfg.index_head_dim + 1))
            + 512 * h * (cfg.qk_nope_head_dim + cfg.v_head_dim) + h * cfg.v_head_dim * cfg.hidden_size)


def work(case):
    kind = case["kind"]
    if kind in ("step", "host", "serve", "verify"):
        rows = case.get("rows", 1)
        ctx, heads, ih, topk = case["ctx"], case["heads"], case["index_heads"], case["topk"]
        if kind == "verify":
            lens, distinct = [ctx - rows + 1 + i for i in range(rows)], min(ctx, rows * topk)
            scanned = ctx
        else:
            lens, distinct = _length_list(rows, ctx), None
            scanned = sum(lens)
        keys = sum(min(n, topk) for n in lens)
        if kind == "serve":
            keys = rows * min(topk, ctx // 4)
        kv_bytes, flops = _attention(keys, heads, 656 if case.get("fp8") else 1152, distinct)
        io = rows * (heads * (576 + 512) * 2 + topk * 4 * (1 if kind in ("step", "host") else 2) + ih * 132)
        return {"bytes": scanned * 132 + kv_bytes + io, "flops": flops + sum(lens) * ih * 128 * 2}
    if kind == "forward":
        cfg, b, n = dsa.named_config("small"), case["batch"], case["seq"]
        h, qk = cfg.num_attention_heads, cfg.kv_lora_rank + cfg.qk_rope_head_dim
        params = (cfg.hidden_size * (cfg.q_lora_rank + qk + cfg.index_head_dim + 3 * cfg.intermediate_size)
                  + cfg.q_lora_rank * (h * (cfg.qk_nope_head_dim + cfg.qk_rope_head_dim)
                                       + cfg.index_n_heads * (cfg.index_head_dim + 1))
                  + cfg.kv_lora_rank * h * (cfg.qk_nope_head_dim + cfg.v_head_dim) + h * cfg.v_head_dim * cfg.hidden_size)
        keys = b * sum(min(i + 1, cfg.index_topk) for i in range(n))
        scanned = b * n * (n + 1) // 2
        return {"bytes": cfg.num_hidden_layers * params * 4 + 2 * b * n * cfg.hidden_size * 4,
                "flops": cfg.num_hidden_layers * (2 * params * b * n + keys * h * 2 * (qk + cfg.kv_lora_rank)
                                                  + scanned * cfg.index_n_heads * cfg.index_head_dim * 2)}
    cfg, b, layers = dsa.named_config(case["config"]), case["batch"], case["layers"]
    heads, ih, topk, params = cfg.num_attention_heads, cfg.index_n_heads, cfg.index_topk, _params(cfg)
    if kind == "prefill":
        n = case["seq"]
        keys, scanned = b * sum(min(i + 1, topk) for i in range(n)), b * n * (n + 1) // 2
        return {"bytes": layers * (params * 2 + b * n * (132 + 1152)) + 2 * b * n * cfg.hidden_size * 2,
                "flops": layers * (2 * params * b * n + keys * heads * 2 * (576 + 512) + scanned * ih * 128 * 2)}
    n = _start(case)
    kv_bytes, attn = _attention(b * topk, heads, 1152)
    return {"bytes": layers * (params * 2 + kv_bytes + b * n * 132),
            "flops": layers * (2 * params * b + attn + b * n * ih * 128 * 2)}


def tolerance(case):
    if case["kind"] == "forward":
        # fp32 sums; a key whose logit lies within rounding of the cutoff may change places with its
        # neighbour, which moves one row of many
        return {"rel": 1e-4, "max": 0.05}
    if case["kind"] in ("prefill", "decode"):
        return {"rel": 1e-2}
    # bf16 attention; positions are ascending, so one exchanged key shifts those between the two
    return {"rel": 1e-2, "differ": 0.005}
