"""Serving-shaped entry of the hot path: one call per layer for a batch of decode
rows over the PAGED caches, graph-capturable, every buffer static-shaped.

Mirror of the reference overlay's ``_hh_fused_hide_decode_paged``
(sglang_overlay/mli-sglang-v0.5.16.patch:1282-1548): same arguments, same modes
(``"full"``, ``"attn_only"``, ``"scan_only"``), same ``select`` values and return
shapes, same conventions (outputs are VIEWS of persistent scratch keyed by the
static shape, overwritten by the next call; ``-1`` pads the selection; per-row
lengths and the page table are read on the device).

Differences a caller can observe: a bf16 ``kv_pool`` is attended in place through
the slot numbers (the reference first gathers the rows with ``index_select``);
``select="approx"`` runs the exact selection; the work is a few launches in
stream order instead of one launch with an in-kernel row barrier
(kernels/cuda_fused_sparse_splitk.py:2025-2028).
"""

from __future__ import annotations

from typing import Dict, Optional, Tuple, Union

import torch

from . import ops

_FP8_ROW = ops.FP8_LATENT_ROW
_plans: Dict[Tuple, "_Plan"] = {}
_SELECT = {"kernel": "exact", "approx": "exact", "exact": "exact", "prod": "prod",
           "prod_side": "prod",  # the side-stream placement is the caller's business
           "torch": "torch"}


class _Plan:
    """Persistent scratch of one static shape (patch :1274-1279), each buffer allocated on first use and
    reused by every later call and by graph replays."""

    def __init__(self, device, B: int, H_real: int, skv_cap: int, nsplit: int, topk: int) -> None:
        self.device, self.B, self.skv_cap, self.nsplit, self.topk = device, B, skv_cap, nsplit, topk
        # Head-geometry convention of the reference (:1443-1452): pad the heads to a multiple of 16
        # with zero queries (a persistent buffer) and slice them off on return.
        self.H_real, self.H = H_real, (H_real + 15) // 16 * 16
        self.qpad = self.attn = self.attn_out = self.part = None
        self.slab = self.logits = self.hist = None
        self.next_idx = self.pos = self.topk_ws = self.paged = None

    def attention_buffers(self) -> None:
        dev, B, H = self.device, self.B, self.H
        if H != self.H_real:
            self.qpad = torch.zeros(1, B, H, ops.LATENT_DIM, dtype=torch.bfloat16, device=dev)
        out = torch.zeros(1, B, H, ops.VALUE_DIM, dtype=torch.bfloat16, device=dev)
        self.part = ops.MlaScratch(B, H, self.nsplit, dev) if self.nsplit > 1 else None  # (one split: no partials)
        self.attn_out = out if H == self.H_real else out[:, :, :self.H_real]
        self.attn = out.view(B, H, ops.VALUE_DIM)

    def scan_buffers(self) -> None:
        self.slab = torch.empty(self.B, (self.skv_cap + 3) // 4 * 4, dtype=torch.float32, device=self.device)
        self.logits = self.slab[:, :self.skv_cap]
        self.hist = torch.zeros(self.B, ops.HIST_BINS, dtype=torch.int32, device=self.device)

    def select_buffers(self) -> None:
        self.next_idx = torch.full((self.B, self.topk), -1, dtype=torch.int32, device=self.device)
        self.pos = torch.full((self.B, self.topk), -1, dtype=torch.int32, device=self.device)
        self.topk_ws = ops.topk_workspace(self.B, self.skv_cap, self.device)
        self.paged = self.topk_ws.numel() <= 16  # rows short enough for the top-k that emits slots itself


def _is_slot_map(out_index_pool: torch.Tensor, skv_cap: int) -> bool:
    """Whether the top-k can read ``out_index_pool`` as its index map."""
    return out_index_pool.dtype == torch.int32 and out_index_pool.shape[1] == skv_cap and out_index_pool.is_contiguous()


def clear_scratch() -> None:
    _plans.clear()
    _operands.clear()


def fused_hide_decode_paged(
    q_all: torch.Tensor,
    kv_pool: torch.Tensor,
    incumbent_slots: torch.Tensor,
    index_q_fp8: torch.Tensor,
    index_weights: torch.Tensor,
    index_k_paged: torch.Tensor,
    page_table: torch.Tensor,
    seq_lens: torch.Tensor,
    skv_cap: int,
    sm_scale: float,
    out_index_pool: Optional[torch.Tensor],
    nsplit: Optional[int] = None,
    index_topk: Optional[int] = None,
    nsplit_attn: Optional[int] = None,
    return_logits: bool = False,
    select: Union[bool, str] = True,
    mode: str = "full",
):
    """Attention over each row's incumbent KV slots + this layer's FP8 indexer over
    the row's full paged prefix -> next index set (patch :1352-1366 for the
    arguments). Returns, as the reference does (:1518-1548): ``attn_out
    [1,B,H,512]`` for ``mode="attn_only"``; the ``[B, skv_cap]`` logit slab for
    ``"scan_only"``; for ``"full"``: ``(attn_out, logits)`` under
    ``select=False/"prod"``, ``(attn_out, next_idx int32 [B, topk])`` under
    ``select=True/"kernel"/"exact"/"approx"`` (KV-slot space, ``-1`` padded;
    plus ``logits`` with ``return_logits``), ``(attn_out, next_idx int64)`` under
    ``select="torch"`` (torch.topk gate).

    The returned tensors are buffers of the call's static shape, overwritten by the next call of that shape.
    The attention is enqueued last and runs beside the top-k, unless ``incumbent_slots`` is the ``next_idx`` that
    the call before returned: the selection is then written over it, so the attention has to come first (3
    requests of 9152 tokens: 34.4 us instead of 24.7). A caller that chains layers of one shape gets the shorter
    order by keeping the selection in a tensor of its own."""
    if mode not in ("full", "attn_only", "scan_only"):
        raise ValueError(f"unknown mode={mode!r}")
    # (by identity: 1 and 0 equal True and False, and are no selections)
    sel_mode = "exact" if select is True else "prod" if select is False else _SELECT.get(select) if isinstance(select, str) else None
    if sel_mode is None:
        raise ValueError(f"unknown select={select!r}")
    q_shape = q_all.shape
    if len(q_shape) != 4 or q_shape[0] != 1:
        raise ValueError(f"q_all must be [1,B,H,dqk], got {tuple(q_shape)}")
    _, B, H_real, dqk = q_shape
    device = q_all.device
    if dqk != ops.LATENT_DIM:
        raise ValueError(f"dqk must be {ops.LATENT_DIM}, got {dqk}")
    iq_shape = index_q_fp8.shape
    if len(iq_shape) != 3 or iq_shape[0] != B:
        raise ValueError(f"index_q_fp8 must be [B={B},Hidx,didx], got {tuple(iq_shape)}")
    Hidx, didx = int(iq_shape[1]), int(iq_shape[2])
    if didx != ops.INDEX_DIM or Hidx % 16:
        raise ValueError(f"unsupported indexer geometry Hidx={Hidx} didx={didx}")
    if index_q_fp8.dtype not in (torch.float8_e4m3fn, torch.uint8):
        raise ValueError(f"index_q_fp8 dtype {index_q_fp8.dtype}")
    if index_weights.shape != (B, Hidx):
        raise ValueError(f"index_weights must be [B,Hidx]=({B},{Hidx}), got {tuple(index_weights.shape)}")
    if seq_lens.shape != (B,) or seq_lens.dtype != torch.int32:
        raise ValueError(f"seq_lens must be int32 [B={B}], got {tuple(seq_lens.shape)} {seq_lens.dtype}")
    pt_shape = page_table.shape
    if len(pt_shape) != 2 or pt_shape[0] != B or page_table.dtype != torch.int32:
        raise ValueError(f"page_table must be int32 [B={B}, pt_stride], got {tuple(pt_shape)} {page_table.dtype}")
    pt_stride = int(pt_shape[1])
    skv_cap = int(skv_cap)
    if pt_stride * ops.PAGE_TOKENS < skv_cap:
        raise ValueError(f"page table ({pt_stride} pages) does not cover skv_cap={skv_cap}")
    if index_k_paged.dtype != torch.uint8 or index_k_paged.dim() != 2 or index_k_paged.shape[1] != ops.INDEX_PAGE_BYTES:
        raise ValueError(f"index_k_paged must be uint8 [num_pages, {ops.INDEX_PAGE_BYTES}]")
    if out_index_pool is not None and (out_index_pool.shape[0] != B or out_index_pool.shape[1] < skv_cap):
        raise ValueError(f"out_index_pool must be [B={B}, >= {skv_cap}], got {tuple(out_index_pool.shape)}")
    inc_shape = incumbent_slots.shape
    if inc_shape[0] != B:
        raise ValueError(f"incumbent batch {inc_shape[0]} != {B}")
    topk = int(inc_shape[1])
    index_topk = topk if index_topk is None else int(index_topk)
    S_pool, row_w = kv_pool.shape
    kv_fp8 = row_w == _FP8_ROW and kv_pool.dtype in (torch.uint8, torch.float8_e4m3fn)
    if not kv_fp8 and not (row_w == dqk and kv_pool.dtype == torch.bfloat16):
        raise ValueError(f"kv_pool must be bf16 [S,{dqk}] or fp8-packed uint8 [S,{_FP8_ROW}], got "
                         f"{kv_pool.dtype} {tuple(kv_pool.shape)}")

    if nsplit_attn is None:
        nsplit_attn = nsplit if nsplit is not None else ops.default_nsplit(B, (H_real + 15) // 16 * 16, topk)
    key = (device, B, H_real, skv_cap, nsplit_attn, topk)
    plan = _plans.get(key)
    if plan is None:
        plan = _plans[key] = _Plan(device, B, H_real, skv_cap, int(nsplit_attn), topk)

    attn_out = None
    behind = False
    if mode != "scan_only":
        if plan.attn is None:
            plan.attention_buffers()
        # one shared pool of S_pool slots: every row is a query row of the same "sequence",
        # entries < 0 or >= S_pool are skipped in the kernel
        if plan.qpad is not None:
            plan.qpad[:, :, :H_real].copy_(q_all)
            q_all = plan.qpad
        slots = incumbent_slots if incumbent_slots.dtype == torch.int32 else incumbent_slots.to(torch.int32)
        slots = slots.contiguous()
        q_rows = q_all.contiguous().view(B, plan.H, dqk)
        kv = kv_pool if kv_pool.dtype != torch.float8_e4m3fn else kv_pool.view(torch.uint8)
        attn_out = plan.attn_out

        # The attention needs neither the scan nor the top-k. Where the selection is one launch it goes
        # behind the two and runs beside the top-k (3 requests of 9152 tokens, the whole step 34.4 -> 25.8 us;
        # 32 of up to 64K, where the attention fills the device by itself, 108.3 -> 106.9); not where it
        # reads the list that the top-k writes, nor where it will refuse its operands: a refused call
        # leaves the selection of the one before it alone.
        if mode == "full" and sel_mode == "exact" and index_topk == topk:
            if plan.next_idx is None:
                plan.select_buffers()
            behind = plan.paged and ops.attention_last(q_rows, kv, slots, sm_scale, plan.next_idx, out_index_pool, skv_cap)
        if not behind:
            ops.sparse_mla_decode(q_rows, kv, slots, sm_scale, None, rows_per_seq=B, nsplit=plan.nsplit, scratch=plan.part,
                                  out=plan.attn)
        if mode == "attn_only":
            return attn_out

    if plan.slab is None:
        plan.scan_buffers()
    use_hist = mode == "full" and sel_mode == "exact"
    iq = index_q_fp8 if index_q_fp8.is_contiguous() else index_q_fp8.contiguous()
    weights = index_weights if index_weights.dtype == torch.float32 else index_weights.to(torch.float32)
    table = page_table.contiguous()
    logits = plan.logits
    ops.indexer_scan_fp8_paged(iq, weights.contiguous(), index_k_paged, table, seq_lens.contiguous(), skv_cap, out=plan.slab,
                               hist=plan.hist if use_hist else None)
    if mode == "scan_only":
        return logits
    if sel_mode == "prod":
        return attn_out, logits

    if sel_mode == "exact":
        if index_topk != topk:
            raise ValueError("the in-launch select emits exactly topk indices")
        if plan.next_idx is None:
            plan.select_buffers()
        next_idx = plan.next_idx
        if out_index_pool is None and plan.paged:
            # the selection leaves the top-k as KV slots, page * 64 + offset from the page-64 table
            # (kernels/cuda_fused_sparse_splitk.py:1142-1144)
            ops.topk_select_paged(logits, topk, seq_lens, plan.hist, table, next_idx)
        elif out_index_pool is not None and plan.paged and (behind or _is_slot_map(out_index_pool, skv_cap)):
            # positions -> KV slots through out_index_pool, read by the top-k as its index map
            ops.topk_select(logits, topk, seq_lens, hist=plan.hist, index_map=out_index_pool, out_idx=next_idx,
                            workspace=plan.topk_ws)
        else:
            pos = plan.pos
            ops.topk_select(logits, topk, seq_lens, hist=plan.hist, out_idx=pos, workspace=plan.topk_ws)
            safe = pos.clamp(min=0).long()
            if out_index_pool is not None:
                mapped = torch.gather(out_index_pool[:, :skv_cap], 1, safe).to(torch.int32)
            else:
                mapped = torch.gather(page_table, 1, safe >> 6) * ops.PAGE_TOKENS + (pos & (ops.PAGE_TOKENS - 1))
            torch.where(pos >= 0, mapped, pos, out=next_idx)  # padding stays -1
        if behind:
            ops.sparse_mla_decode(q_rows, kv, slots, sm_scale, None, rows_per_seq=B, nsplit=plan.nsplit, scratch=plan.part,
                                  out=plan.attn, beside_previous=True)
        if return_logits:
            return attn_out, next_idx, logits
        return attn_out, next_idx

    # torch top-k over the full-prefix logits (gate only, :1531-1548)
    if out_index_pool is None:
        raise ValueError("select='torch' needs out_index_pool")
    k = min(index_topk, skv_cap)
    top_v, top_pos = torch.topk(logits, k, dim=-1)
    next_idx = torch.gather(out_index_pool.long()[:, :skv_cap], 1, top_pos)
    next_idx = torch.where(torch.isfinite(top_v), next_idx, torch.full_like(next_idx, -1))
    if k < index_topk:
        next_idx = torch.cat([next_idx, torch.full((B, index_topk - k), -1, dtype=next_idx.dtype, device=device)], 1)
    if return_logits:
        return attn_out, next_idx, logits.clone()
    return attn_out, next_idx


_operands: Dict[Tuple, Tuple[torch.Tensor, torch.Tensor]] = {}


def forward_hide_operands(
    q_proj: torch.Tensor,
    k_proj: torch.Tensor,
    head_gates: torch.Tensor,
    k_norm_weight: torch.Tensor,
    k_norm_bias: torch.Tensor,
    k_norm_eps: float,
    rope_cos: torch.Tensor,
    rope_sin: torch.Tensor,
    positions: torch.Tensor,
    index_k_paged: torch.Tensor,
    page_table_64: torch.Tensor,
    seq_lens: torch.Tensor,
    rope_interleave: bool = False,
    scale_fmt: Optional[str] = None,
    softmax_scale: Optional[float] = None,
):
    """This layer's indexer PREPARE + STORE without a top-k, for a batch of decode
    rows: the operands ``fused_hide_decode_paged`` scans with. Counterpart of the
    overlay's ``Indexer.forward_hide_operands`` after its projections
    (sglang_overlay/mli-sglang-v0.5.16.patch:252-363, non-fusion branch :322-342):
    ``q_proj`` = wq_b(q_lora) ``[B, Hidx, 128]`` bf16, ``k_proj`` = wk(x) ``[B, 128]``
    bf16, ``head_gates`` = weights_proj(x) ``[B, Hidx]`` fp32 (not yet scaled). One
    launch rotates, quantises, folds ``n_heads^-0.5 * q_scale * softmax_scale`` into
    the gates and stores each row's key at ``positions[b]`` in its page.

    Returns the reference's tuple ``(q_fp8 [B,Hidx,128] uint8 bytes, weights [B,Hidx]
    fp32, index_k_paged, page_table_64 int32, seq_lens int32, skv_cap)``; the first
    two are views of persistent scratch keyed by the static shape (graph-capturable:
    no host integer is read from the device). Raises where the reference refuses to
    engage (:279-312): page size other than 64, missing table or lengths."""
    if page_table_64 is None or seq_lens is None:
        raise RuntimeError("[HIDE VOID] page-64 table / int32 seqlens unavailable")
    if index_k_paged.dim() != 2 or index_k_paged.shape[1] != ops.INDEX_PAGE_BYTES:
        raise RuntimeError(f"[HIDE VOID] index-K pages must be [num_pages, {ops.INDEX_PAGE_BYTES}] "
                           "(64-token pages)")
    if page_table_64.dtype != torch.int32:
        page_table_64 = page_table_64.to(torch.int32)
    if seq_lens.dtype != torch.int32:
        seq_lens = seq_lens.to(torch.int32)
    B, n_heads = q_proj.shape[0], q_proj.shape[1]
    device = q_proj.device
    key = (device, B, n_heads)
    buffers = _operands.get(key)
    if buffers is None:
        buffers = _operands[key] = (torch.empty(B, n_heads, ops.INDEX_DIM, dtype=torch.uint8, device=device),
                                    torch.empty(B, n_heads, dtype=torch.float32, device=device))
    q_fp8, weights = buffers
    ops.indexer_stage_fp8(q_proj, k_proj, head_gates, k_norm_weight, k_norm_bias, k_norm_eps, rope_cos, rope_sin,
                          positions, q_fp8, weights, pages=index_k_paged, page_table=page_table_64,
                          rope_interleave=rope_interleave, scale_fmt=scale_fmt, softmax_scale=softmax_scale)
    skv_cap = int(page_table_64.shape[1]) * ops.PAGE_TOKENS
    return q_fp8, weights, index_k_paged, page_table_64, seq_lens, skv_cap


_hh_fused_hide_decode_paged = fused_hide_decode_paged  # the reference's name for it
