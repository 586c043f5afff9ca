"""Tensor-level entry points over the C ABI: checks shapes and dtypes, hands raw
device pointers and the current CUDA stream to libdsa_b200.so.

torch is used here for device memory and streams only. Nothing in this module
computes on the host or falls back to torch kernels; a missing library raises
at the first call (``_lib.lib()``). The entry points of a step run their checks, allocations and
the call natively (``_lib.host()``, csrc/host_ops.cpp); the rest goes through ctypes.
"""

from __future__ import annotations

from typing import Optional, Tuple

import torch

from . import _lib

LATENT_DIM = 576
VALUE_DIM = 512
INDEX_DIM = 128
HEAD_BLOCK = 16
PAGE_TOKENS = 64
INDEX_PAGE_BYTES = 8448
FP8_LATENT_ROW = 656
HIST_BINS = 4096

_FP8 = torch.float8_e4m3fn
_STAGES = {"both": 0, "partials": 1, "combine": 2}
_LATENT_FORMATS = {"bf16": 0, "bf16_quant": 1, "fp8": 2}
_host = _lib.host


def _ptr(t: Optional[torch.Tensor]) -> Optional[int]:
    return None if t is None else t.data_ptr()


def _stream() -> int:
    return torch.cuda.current_stream().cuda_stream


def _need(cond: bool, msg: str) -> None:
    if not cond:
        raise ValueError(msg)


def _cuda_contig(t: torch.Tensor, name: str, dtypes) -> None:
    _need(t.is_cuda, f"{name} must be a CUDA tensor")
    _need(t.is_contiguous(), f"{name} must be contiguous")
    _need(t.dtype in dtypes, f"{name} has dtype {t.dtype}, expected one of {dtypes}")


def _lens(seq_lens: Optional[torch.Tensor], rows: int) -> Optional[torch.Tensor]:
    if seq_lens is not None:
        _cuda_contig(seq_lens, "seq_lens", (torch.int32,))
        _need(seq_lens.numel() == rows, f"seq_lens has {seq_lens.numel()} entries, expected {rows}")
    return seq_lens


# --------------------------------------------------------------------------- a7
def quantize_e4m3_rowwise(x: torch.Tensor, clamp_min: float = 1e-6) -> Tuple[torch.Tensor, torch.Tensor]:
    """Per-row absmax e4m3 quantisation: ``(q, scale)`` with ``x ~ q * scale[..., None]``
    (reference kernels/cuda_fused_sparse_splitk.py:2969-2974)."""
    _cuda_contig(x, "x", (torch.float32,))
    cols = x.shape[-1]
    rows = x.numel() // cols
    q = torch.empty(x.shape, dtype=torch.uint8, device=x.device)
    scale = torch.empty(x.shape[:-1], dtype=torch.float32, device=x.device)
    _lib.check(_lib.lib().dsa_quantize_e4m3_rowwise(_ptr(x), _ptr(q), _ptr(scale), rows, cols,
                                                   float(clamp_min), _stream()))
    return q.view(_FP8), scale


# --------------------------------------------------------------------------- a1
def indexer_scan_fp8(
    index_q: torch.Tensor,
    index_w: torch.Tensor,
    index_k: torch.Tensor,
    k_scale: torch.Tensor,
    seq_lens: Optional[torch.Tensor] = None,
    *,
    rows_per_seq: int = 1,
    ctx: Optional[int] = None,
    out: Optional[torch.Tensor] = None,
    hist: Optional[torch.Tensor] = None,
    impl: int = 0,
) -> torch.Tensor:
    """Indexer logits ``[R, ctx]`` (fp32) from e4m3 queries/keys.

    index_q ``[R, Hidx, 128]`` e4m3 (or uint8 bytes), index_w ``[R, Hidx]`` fp32
    with the query scale folded in, index_k ``[n_seq, cap, 128]`` (or ``[cap, 128]``),
    k_scale ``[n_seq, cap]`` fp32. Row r reads sequence ``r // rows_per_seq``.
    """
    return _host().scan_fp8(index_q, index_w, index_k, k_scale, seq_lens, rows_per_seq, ctx, out, hist, impl)


def indexer_scan_fp8_paged(
    index_q: torch.Tensor,
    index_w: torch.Tensor,
    index_k_pages: torch.Tensor,
    page_table: torch.Tensor,
    seq_lens: torch.Tensor,
    ctx: int,
    *,
    out: Optional[torch.Tensor] = None,
    hist: Optional[torch.Tensor] = None,
) -> torch.Tensor:
    """Paged form: index_k_pages ``[num_pages, 8448]`` uint8, page_table ``[R, pt_stride]`` int32."""
    return _host().scan_paged(index_q, index_w, index_k_pages, page_table, seq_lens, ctx, out, hist)


def indexer_scan_f32(
    index_q: torch.Tensor,
    index_w: torch.Tensor,
    index_k: torch.Tensor,
    seq_lens: Optional[torch.Tensor] = None,
    *,
    rows_per_seq: int = 1,
    ctx: Optional[int] = None,
    out: Optional[torch.Tensor] = None,
) -> torch.Tensor:
    """fp32 logits for any head count / key width: q ``[R, H, D]``, k ``[n_seq, cap, D]`` of which
    the first ``ctx`` keys are scanned (default: all)."""
    return _host().scan_f32(index_q, index_w, index_k, seq_lens, rows_per_seq, ctx, out)


# --------------------------------------------------------------------------- a3
def topk_workspace(rows: int, n: int, device) -> torch.Tensor:
    """Zeroed scratch for ``topk_select`` on ``rows`` rows of ``n`` logits. It is
    left re-armed by every call, so one allocation serves a whole decode loop;
    calls that share it must not overlap on the device."""
    nbytes = int(_lib.lib().dsa_topk_workspace_bytes(rows, n))
    return torch.zeros(nbytes, dtype=torch.uint8, device=device)


def topk_select(
    logits: torch.Tensor,
    topk: int,
    seq_lens: Optional[torch.Tensor] = None,
    *,
    hist: Optional[torch.Tensor] = None,
    index_map: Optional[torch.Tensor] = None,
    pad_value: int = -1,
    index_offset: int = 0,
    out_idx: Optional[torch.Tensor] = None,
    out_val: Optional[torch.Tensor] = None,
    return_values: bool = False,
    workspace: Optional[torch.Tensor] = None,
):
    """Exact top-k per row of ``logits[R, n]`` (a view of a wider slab is fine):
    int32 positions in ascending order, ties to the lower position, padded with
    ``pad_value``."""
    return _host().topk(logits, topk, seq_lens, hist, index_map, pad_value, index_offset, out_idx, out_val, return_values,
                        workspace)


def topk_select_paged(logits: torch.Tensor, topk: int, seq_lens: Optional[torch.Tensor], hist: torch.Tensor,
                      page_table: torch.Tensor, out_idx: torch.Tensor, pad_value: int = -1) -> torch.Tensor:
    """:func:`topk_select` over paged caches: ``out_idx`` receives cache slots,
    ``page_table[r, p // 64] * 64 + p % 64`` for position p (rows that need no workspace)."""
    return _host().topk_paged(logits, topk, seq_lens, hist, page_table, pad_value, out_idx)


# --------------------------------------------------------------------------- a4, a5
class MlaScratch:
    """Caller-owned split-K partials (the reference's PartAcc / PartM / PartL,
    kernels/cuda_fused_sparse_splitk.py:3005-3009), sized once and reused."""

    def __init__(self, rows: int, heads: int, nsplit: int, device) -> None:
        self.rows, self.heads, self.nsplit = rows, heads, nsplit
        self.acc = torch.empty(rows, nsplit, heads, VALUE_DIM, dtype=torch.float32, device=device)
        self.m = torch.empty(rows, nsplit, heads, dtype=torch.float32, device=device)
        self.l = torch.empty(rows, nsplit, heads, dtype=torch.float32, device=device)


def default_nsplit(rows: int, heads: int, topk: int, sm_count: int = 148) -> int:
    """Splits of the index list, each a whole number of 64-key tiles, that :func:`sparse_mla_decode` takes by
    itself: enough CTAs for the SMs without more partials than the merge should read (csrc/host_ops.cpp)."""
    return _host().default_nsplit(rows, heads, topk, sm_count)


def sparse_mla_decode(
    q: torch.Tensor,
    kv: torch.Tensor,
    indices: Optional[torch.Tensor],
    sm_scale: float,
    seq_lens: Optional[torch.Tensor] = None,
    *,
    rows_per_seq: int = 1,
    nsplit: Optional[int] = None,
    scratch: Optional[MlaScratch] = None,
    out: Optional[torch.Tensor] = None,
    dense_keys: Optional[int] = None,
    stage: str = "both",
    beside_previous: bool = False,
    prompt: bool = False,
) -> torch.Tensor:
    """Sparse MLA decode: q ``[R, H, 576]`` bf16, kv ``[n_seq, cap, 576]`` bf16 or
    ``[n_seq, cap, 656]`` uint8 (fp8-packed rows), indices ``[R, topk]`` int32 or
    None for dense attention over ``dense_keys`` positions. Returns ``[R, H, 512]`` bf16.
    ``beside_previous``: none of the operands comes from the two kernels enqueued just before
    this call (the lagged schedule's attention behind this layer's scan and top-k); the attention
    then runs beside the top-k and completes after it. ``prompt``: the rows of each sequence are its
    first positions (row i sees at most its first i + 1 keys), so that neighbours attend nearly the same
    keys and may share a launch's CTAs; for speed alone, the results are the same without it."""
    if stage not in _STAGES:
        raise ValueError(f"unknown stage {stage!r}")
    if scratch is None:
        acc = m = l = None
    else:
        acc, m, l = scratch.acc, scratch.m, scratch.l
    return _host().mla(q, kv, indices, sm_scale, seq_lens, rows_per_seq, nsplit, acc, m, l, out, dense_keys, _STAGES[stage],
                       beside_previous, prompt)


def attention_last(q, kv, slots, sm_scale, next_idx, index_map, cap) -> bool:
    """Whether the serving entry may enqueue the attention behind scan and top-k (csrc/host_ops.cpp)."""
    return _host().attention_last(q, kv, slots, sm_scale, next_idx, index_map, cap)


def sparse_mla_f32(
    q: torch.Tensor,
    kv: torch.Tensor,
    indices: Optional[torch.Tensor],
    value_dim: int,
    sm_scale: float,
    seq_lens: Optional[torch.Tensor] = None,
    *,
    rows_per_seq: int = 1,
) -> torch.Tensor:
    """fp32 attention for any width: q ``[R, H, Dqk]``, kv ``[n_seq, ctx, Dqk]``;
    indices None = dense causal over ``seq_lens``."""
    return _host().mla_f32(q, kv, indices, value_dim, sm_scale, seq_lens, rows_per_seq)


# --------------------------------------------------------------------------- a6
def fused_decode(
    q: torch.Tensor,
    kv: torch.Tensor,
    attend_indices: torch.Tensor,
    sm_scale: float,
    index_q: torch.Tensor,
    index_w: torch.Tensor,
    index_k: torch.Tensor,
    k_scale: torch.Tensor,
    seq_lens: Optional[torch.Tensor] = None,
    *,
    rows_per_seq: int = 1,
    nsplit: Optional[int] = None,
    scratch: Optional[MlaScratch] = None,
    out: Optional[torch.Tensor] = None,
    logits: Optional[torch.Tensor] = None,
    hist: Optional[torch.Tensor] = None,
) -> Tuple[torch.Tensor, torch.Tensor]:
    """One launch for a layer's sparse MLA over ``attend_indices`` AND its indexer
    scan (then the LSE merge): returns ``(attention_out [R,H,512] bf16, logits [R,ctx] fp32)``.
    Same operands as :func:`sparse_mla_decode` (bf16 cache) and :func:`indexer_scan_fp8`."""
    _cuda_contig(q, "q", (torch.bfloat16,))
    _need(q.dim() == 3 and q.shape[2] == LATENT_DIM and q.shape[1] % HEAD_BLOCK == 0, "q must be [R, H % 16 == 0, 576]")
    R, H = q.shape[0], q.shape[1]
    if kv.dim() == 2:
        kv = kv.unsqueeze(0)
    _cuda_contig(kv, "kv", (torch.bfloat16,))
    _need(kv.dim() == 3 and kv.shape[2] == LATENT_DIM, "kv must be [n_seq, cap, 576] bf16")
    _cuda_contig(attend_indices, "attend_indices", (torch.int32,))
    _need(attend_indices.dim() == 2 and attend_indices.shape[0] == R, "attend_indices must be [R, topk]")
    topk = attend_indices.shape[1]
    _cuda_contig(index_q, "index_q", (_FP8, torch.uint8))
    _cuda_contig(index_w, "index_w", (torch.float32,))
    _cuda_contig(index_k, "index_k", (_FP8, torch.uint8))
    _cuda_contig(k_scale, "k_scale", (torch.float32,))
    if index_k.dim() == 2:
        index_k = index_k.unsqueeze(0)
        k_scale = k_scale.reshape(1, -1)
    n_seq, cap = index_k.shape[0], index_k.shape[1]
    _need(kv.shape[0] == n_seq and R == n_seq * rows_per_seq, "R must equal n_seq * rows_per_seq for both caches")
    _need(index_q.shape[0] == R and tuple(index_w.shape) == (R, index_q.shape[1]), "index_q / index_w rows differ from q")
    seq_lens = _lens(seq_lens, R)
    if nsplit is None:
        nsplit = scratch.nsplit if scratch is not None else default_nsplit(R, H, topk)
    if scratch is None:
        scratch = MlaScratch(R, H, nsplit, q.device)
    _need(scratch.rows >= R and scratch.heads == H and scratch.nsplit == nsplit, "scratch does not match the launch")
    if out is None:
        out = torch.empty(R, H, VALUE_DIM, dtype=torch.bfloat16, device=q.device)
    if logits is None:
        logits = torch.empty(R, (cap + 3) // 4 * 4, dtype=torch.float32, device=q.device)
    _cuda_contig(logits, "logits", (torch.float32,))
    if hist is not None:
        _cuda_contig(hist, "hist", (torch.int32, torch.uint32))
        _need(hist.numel() == R * HIST_BINS, "hist must be [R, 4096]")
    _lib.check(_lib.lib().dsa_fused_decode(
        _ptr(q), _ptr(kv), _ptr(attend_indices), _ptr(seq_lens), _ptr(scratch.acc), _ptr(scratch.m),
        _ptr(scratch.l), _ptr(out), _ptr(index_q), _ptr(index_w), _ptr(index_k), _ptr(k_scale), _ptr(seq_lens),
        _ptr(logits), _ptr(hist), R, rows_per_seq, H, topk, nsplit, float(sm_scale), kv.shape[1],
        index_q.shape[1], cap, n_seq, cap, cap, logits.shape[1], _stream()))
    return out, logits[:, :cap]


# --------------------------------------------------------------------------- decode-step preparation
def rmsnorm(x: torch.Tensor, weight: torch.Tensor, eps: float) -> torch.Tensor:
    """RMSNorm over the last dimension in one launch (fp32 math, one rounding)."""
    return _host().rmsnorm(x, weight, eps)


def add_rmsnorm(x: torch.Tensor, delta: torch.Tensor, weight: torch.Tensor, eps: float):
    """``s = x + delta`` and ``rmsnorm(s)`` in one launch (bf16 rows of at most 8192
    elements, a multiple of 8, or fp32 rows): returns ``(s, normed)``, both rounded exactly as the
    separate addition and norm would be."""
    return _host().add_rmsnorm(x, delta, weight, eps)


def silu_mul(gate: torch.Tensor, up: torch.Tensor) -> torch.Tensor:
    """``silu(gate) * up`` over bf16 or fp32 tensors in one launch, rounded as the two separate operations."""
    return _host().silu_mul(gate, up)


def copy_bytes(dst: torch.Tensor, src: torch.Tensor, beside_previous: bool = False) -> None:
    """``dst <- src`` (same byte count, a multiple of 16) by a kernel on the current stream.
    Each side is a contiguous CUDA tensor or pinned host memory. With ``beside_previous`` the
    copy runs beside the kernel enqueued just before it and completes after it; what is enqueued
    next sees both. Neither of the two kernels enqueued before it may write or read these bytes
    (the top-k releases its dependents before it waits for the scan)."""
    for t, name in ((dst, "dst"), (src, "src")):
        _need((t.is_cuda or t.is_pinned()) and t.is_contiguous(), f"{name} must be contiguous CUDA or pinned memory")
    nbytes = dst.numel() * dst.element_size()
    _need(nbytes == src.numel() * src.element_size() and nbytes % 16 == 0, "byte counts must match and be a multiple of 16")
    fn = _lib.lib().dsa_copy_bytes_beside if beside_previous else _lib.lib().dsa_copy_bytes
    _lib.check(fn(_ptr(dst), _ptr(src), nbytes, _stream()))


def post_epoch(counter: torch.Tensor, host_flag: torch.Tensor) -> None:
    """Enqueues the completion signal: ``counter`` (one int32 on the device) is bumped and
    its value posted to ``host_flag`` (one int32 of pinned host memory) after everything
    enqueued so far on the current stream."""
    _need(counter.is_cuda and counter.dtype == torch.int32 and counter.numel() == 1, "counter: one CUDA int32")
    _need(host_flag.is_pinned() and host_flag.dtype == torch.int32 and host_flag.numel() == 1,
          "host_flag: one pinned int32")
    _lib.check(_lib.lib().dsa_post_epoch(_ptr(counter), _ptr(host_flag), _stream()))


def copy_post_epoch(dst: torch.Tensor, src: torch.Tensor, counter: torch.Tensor, host_flag: torch.Tensor,
                    beside_previous: bool = False) -> None:
    """:func:`copy_bytes` of at most 1 MiB followed by :func:`post_epoch`, as one launch: the last
    node of a step when a few KB (the selection) still have to reach the host before the signal.
    ``beside_previous``: ``src`` does not come from the two kernels enqueued before this call; it is
    copied beside the last of them and only the signal waits for it."""
    for t, name in ((dst, "dst"), (src, "src")):
        _need((t.is_cuda or t.is_pinned()) and t.is_contiguous(), f"{name} must be contiguous CUDA or pinned memory")
    nbytes = dst.numel() * dst.element_size()
    _need(nbytes == src.numel() * src.element_size() and nbytes % 16 == 0 and nbytes <= 1 << 20,
          "byte counts must match, be a multiple of 16 and at most 1 MiB")
    _need(counter.is_cuda and counter.dtype == torch.int32 and counter.numel() == 1, "counter: one CUDA int32")
    _need(host_flag.is_pinned() and host_flag.dtype == torch.int32 and host_flag.numel() == 1,
          "host_flag: one pinned int32")
    _lib.check(_lib.lib().dsa_copy_post_epoch(_ptr(dst), _ptr(src), nbytes, _ptr(counter), _ptr(host_flag),
                                              1 if beside_previous else 0, _stream()))


def _gemv_operand(x: torch.Tensor, weight: torch.Tensor, most: int) -> torch.Tensor:
    _need(x.is_cuda and x.dtype == torch.bfloat16 and weight.dtype == torch.bfloat16 and x.dim() == 2,
          "x must be a CUDA bf16 [B, k] tensor and weight bf16")
    _need(weight.dim() == 2 and weight.shape[1] == x.shape[1] and weight.is_contiguous(), "weight must be contiguous [n, k]")
    _need(1 <= x.shape[0] <= most and x.shape[1] % 8 == 0, f"batch 1..{most}, k a multiple of 8")
    return x if x.stride(1) == 1 and x.stride(0) % 8 == 0 else x.contiguous()


def gemv(x: torch.Tensor, weight: torch.Tensor, ahead: bool = False) -> torch.Tensor:
    """``x @ weight.T`` for a decode batch of 1..4 rows (bf16, fp32 accumulation): the weight
    matrix ``[n, k]`` is streamed once. ``ahead`` (here and below): its first part while the kernels before
    are still running, which the caller may say where none of them writes it (see ``dsa_gemv_ahead_bf16``)."""
    x = _gemv_operand(x, weight, 4)
    (b, k), n = x.shape, weight.shape[0]
    y = torch.empty(b, n, dtype=torch.bfloat16, device=x.device)
    fn = _lib.lib().dsa_gemv_ahead_bf16 if ahead else _lib.lib().dsa_gemv_bf16
    _lib.check(fn(_ptr(weight), _ptr(x), _ptr(y), b, n, k, x.stride(0) if b > 1 else k, n, _stream()))
    return y


def gemv_swiglu(x: torch.Tensor, gate: torch.Tensor, up: torch.Tensor, ahead: bool = False) -> torch.Tensor:
    """``silu(x @ gate.T) * (x @ up.T)`` for one or two rows in one launch, rounded as the separate operations."""
    x = _gemv_operand(x, gate, 2)
    _need(up.shape == gate.shape and up.dtype == torch.bfloat16 and up.is_contiguous(), "gate and up must have one shape")
    (b, k), n = x.shape, gate.shape[0]
    if b * k > 32768:  # x beside the weights' ring in shared memory: the streaming kernel's limit is a little above
        return silu_mul(gemv(x, gate, ahead), gemv(x, up, ahead))
    y = torch.empty(b, n, dtype=torch.bfloat16, device=x.device)
    _lib.check(_lib.lib().dsa_gemv_swiglu_bf16(_ptr(gate), _ptr(up), _ptr(x), _ptr(y), b, n, k, x.stride(0) if b > 1 else k, n,
                                               1 if ahead else 0, _stream()))
    return y


def norm_gemv(x: torch.Tensor, delta: Optional[torch.Tensor], norm_weight: torch.Tensor, eps: float, weight: torch.Tensor,
              up: Optional[torch.Tensor] = None, ahead: bool = False):
    """``(s, rmsnorm(s) @ weight.T)`` with ``s = x + delta`` (``x`` without a delta) in one launch, for 1..4
    rows of at most 8192; with ``up`` the SwiGLU product of :func:`gemv_swiglu`."""
    x = _gemv_operand(x, weight, 2 if up is not None else 4)
    (b, k), n = x.shape, weight.shape[0]
    _cuda_contig(norm_weight, "norm_weight", (torch.bfloat16,))
    _need(norm_weight.numel() == k, "norm_weight must have k elements")
    s = x
    if delta is not None:
        _cuda_contig(delta, "delta", (torch.bfloat16,))
        _need(tuple(delta.shape) == (b, k), "delta must be [B, k]")
        s = torch.empty(b, k, dtype=torch.bfloat16, device=x.device)
    if up is not None:
        _need(up.shape == weight.shape and up.dtype == torch.bfloat16 and up.is_contiguous(), "gate and up must have one shape")
    y = torch.empty(b, n, dtype=torch.bfloat16, device=x.device)
    _lib.check(_lib.lib().dsa_norm_gemv_bf16(_ptr(weight), _ptr(up), _ptr(x), _ptr(delta), _ptr(norm_weight), float(eps),
                                             _ptr(s) if delta is not None else None, _ptr(y), b, n, k,
                                             x.stride(0) if b > 1 else k, n, 1 if ahead else 0, _stream()))
    return s, y


def norm_gemv_fits(b: int, k: int) -> bool:
    """Rows that dsa_norm_gemv_bf16 takes."""
    return 1 <= b <= 4 and k % 8 == 0 and k <= 8192


HEAD_TOKENS = 8  # tokens that share one reading of kv_b_proj's weight in decode_token / value_project


def value_project(kv_b: torch.Tensor, o: torch.Tensor, heads: int, v_dim: int, ahead: bool = False) -> torch.Tensor:
    """``[B, heads, v_dim]``: every head's latent output ``o`` ``[B, >= heads, 512]`` through W_UV, the last
    ``v_dim`` rows of the head's part of ``kv_b`` ``[heads * per_head, 512]``; at most HEAD_TOKENS rows."""
    _cuda_contig(kv_b, "kv_b", (torch.bfloat16,))
    _cuda_contig(o, "o", (torch.bfloat16,))
    _need(o.dim() == 3 and o.shape[2] == VALUE_DIM and o.shape[1] >= heads and kv_b.dim() == 2 and kv_b.shape[1] == VALUE_DIM
          and kv_b.shape[0] % heads == 0 and kv_b.shape[0] // heads >= v_dim,
          "kv_b must be [heads * per_head, 512], o [B, >= heads, 512]")
    ov = torch.empty(o.shape[0], heads, v_dim, dtype=torch.bfloat16, device=o.device)
    _lib.check(_lib.lib().dsa_value_project(_ptr(kv_b), _ptr(o), _ptr(ov), o.shape[0], heads, o.shape[1],
                                            kv_b.shape[0] // heads - v_dim, v_dim, 1 if ahead else 0, _stream()))
    return ov


def decode_token(iq_raw, w_raw, ik_raw, kv_a, q, kv_b, kv_norm_w, mla_cos, mla_sin, idx_cos, idx_sin, positions, index_q,
                 index_w, q_full, cache_index_k, cache_k_scale, cache_kv, interleave: bool, eps: float,
                 ahead: bool = False) -> None:
    """:func:`decode_prep` for at most HEAD_TOKENS tokens with the query's absorption in the launch: ``q``
    ``[B, H * (nope + 64)]`` and ``kv_b`` ``[H * per_head, 512]`` instead of ``q_abs`` and ``q_pe``. The five
    inputs are 2-D and may be column ranges of a stacked projection's output (see ``dsa_decode_token``)."""
    B, H = q_full.shape[0], q_full.shape[1]
    n_idx = index_w.shape[1]
    per_head = kv_b.shape[0] // H
    nope = q.shape[1] // H - 64
    for t, n, width in ((iq_raw, "iq_raw", n_idx * INDEX_DIM), (w_raw, "w_raw", n_idx), (ik_raw, "ik_raw", INDEX_DIM),
                        (kv_a, "kv_a", LATENT_DIM), (q, "q", H * (nope + 64))):
        _need(t.is_cuda and t.dtype == torch.bfloat16 and tuple(t.shape) == (B, width) and t.stride(1) == 1,
              f"{n} must be a CUDA bf16 [B, {width}] tensor with dense rows")
    for t, n in ((kv_b, "kv_b"), (q_full, "q_full"), (kv_norm_w, "kv_norm_w"), (mla_cos, "mla_cos"), (mla_sin, "mla_sin"),
                 (idx_cos, "idx_cos"), (idx_sin, "idx_sin")):
        _cuda_contig(t, n, (torch.bfloat16,))
    _cuda_contig(positions, "positions", (torch.int64,))
    _need(q_full.shape[2] == LATENT_DIM and kv_b.shape[1] == VALUE_DIM and kv_b.shape[0] == H * per_head and per_head > nope > 0,
          "kv_b must be [H * (nope + v), 512], q [B, H * (nope + 64)], q_full [B, H, 576]")
    cap = cache_kv.shape[1]
    _need(cache_kv.shape[0] == B and cache_index_k.shape[:2] == (B, cap), "caches must be [B, cap, ...]")
    _lib.check(_lib.lib().dsa_decode_token(
        _ptr(iq_raw), iq_raw.stride(0), _ptr(w_raw), w_raw.stride(0), _ptr(ik_raw), ik_raw.stride(0), _ptr(kv_a), kv_a.stride(0),
        _ptr(q), q.stride(0), _ptr(kv_b), _ptr(kv_norm_w), _ptr(mla_cos), _ptr(mla_sin), _ptr(idx_cos), _ptr(idx_sin),
        _ptr(positions), _ptr(index_q), _ptr(index_w), _ptr(q_full), _ptr(cache_index_k), _ptr(cache_k_scale), _ptr(cache_kv),
        B, H, nope, per_head - nope, n_idx, cap, 1 if interleave else 0, float(eps), 1 if ahead else 0, _stream()))


def indexer_stage_fp8(q_raw, k_raw, w_raw, k_norm_weight, k_norm_bias, k_norm_eps: float, rope_cos, rope_sin,
                      positions, index_q, index_w, cache_index_k=None, cache_k_scale=None, pages=None,
                      page_table=None, rope_interleave: bool = False, scale_fmt: Optional[str] = None,
                      softmax_scale: Optional[float] = None) -> None:
    """Serving-form indexer staging in one launch: the reference's
    ``Indexer.stage_fp8_operands`` after its three projections
    (inference/modeling/transformer.py:1015-1066) -- LayerNorm of the key, rotary
    embedding, Hadamard rotation, ``act_quant`` (``scale_fmt`` not None = power-of-two
    scales), folded head weights, and the append of the key to the dense cache
    (``cache_index_k`` [B, cap, 128] u8 + ``cache_k_scale`` [B, cap]) or to 64-token
    ``pages`` through ``page_table``. ``q_raw`` [B, heads, 128] / ``k_raw`` [B, 128] bf16,
    ``w_raw`` [B, heads] fp32, ``rope_cos`` / ``rope_sin`` [cap, 32] fp32."""
    _host().indexer_stage(q_raw, k_raw, w_raw, k_norm_weight, k_norm_bias, k_norm_eps, rope_cos, rope_sin, positions, index_q,
                          index_w, cache_index_k, cache_k_scale, pages, page_table, rope_interleave, scale_fmt is not None,
                          softmax_scale)


def latent_append(kv_a, kv_norm_weight, eps: float, rope_cos, rope_sin, positions, slots, pool,
                  rope_interleave: bool = True, fmt: str = "fp8", scale_fmt: Optional[str] = None) -> None:
    """Serving-form latent append in one launch (inference/modeling/transformer.py:3264-3276
    in the reference): RMSNorm of the 512 latent dims of ``kv_a`` [B, 576] bf16, rotary
    embedding of its 64 rope dims, row written at ``slots[b]`` of ``pool``: ``fmt="bf16"``
    [n_slots, 576] bf16 as it is, ``"bf16_quant"`` the same with the latent dims passed
    through act_quant and back, ``"fp8"`` the 656-byte packed rows [n_slots, 656] uint8."""
    if fmt not in _LATENT_FORMATS:
        raise ValueError(f"fmt must be one of {sorted(_LATENT_FORMATS)}")
    _host().latent_append(kv_a, kv_norm_weight, eps, rope_cos, rope_sin, positions, slots, pool, rope_interleave,
                          _LATENT_FORMATS[fmt], scale_fmt is not None)


def decode_prep(iq_raw, w_raw, ik_raw, kv_a, q_abs, q_pe, kv_norm_w, mla_cos, mla_sin, idx_cos, idx_sin,
                positions, index_q, index_w, q_full, cache_index_k, cache_k_scale, cache_kv,
                interleave: bool, eps: float) -> None:
    """One launch for the chain between the projection GEMVs and the hot path
    (see ``dsa_decode_prep`` in the header). All operands bf16 CUDA tensors;
    ``q_pe`` may be a strided view ``q[..., nope:]`` of the q_b_proj output."""
    for t, n in ((iq_raw, "iq_raw"), (w_raw, "w_raw"), (ik_raw, "ik_raw"), (kv_a, "kv_a"), (q_abs, "q_abs"),
                 (kv_norm_w, "kv_norm_w"), (mla_cos, "mla_cos"), (mla_sin, "mla_sin"), (idx_cos, "idx_cos"),
                 (idx_sin, "idx_sin")):
        _cuda_contig(t, n, (torch.bfloat16,))
    _need(q_pe.dtype == torch.bfloat16 and q_pe.dim() == 3 and q_pe.shape[2] == 64 and q_pe.stride(2) == 1
          and (q_pe.shape[0] == 1 or q_pe.stride(0) == q_pe.shape[1] * q_pe.stride(1)),
          "q_pe must be a [B, H, 64] bf16 view with dense rows")
    _cuda_contig(positions, "positions", (torch.int64,))
    B, n_idx = iq_raw.shape[0], iq_raw.shape[1]
    H = q_abs.shape[1]
    _need(iq_raw.shape[2] == INDEX_DIM and kv_a.shape[-1] == LATENT_DIM and q_abs.shape[2] == VALUE_DIM,
          "decode prep needs the production geometry")
    cap = cache_kv.shape[1]
    _need(cache_kv.shape[0] == B and cache_index_k.shape[:2] == (B, cap), "caches must be [B, cap, ...]")
    _lib.check(_lib.lib().dsa_decode_prep(
        _ptr(iq_raw), _ptr(w_raw), _ptr(ik_raw), _ptr(kv_a), _ptr(q_abs), _ptr(q_pe), q_pe.stride(1), _ptr(kv_norm_w),
        _ptr(mla_cos), _ptr(mla_sin), _ptr(idx_cos), _ptr(idx_sin), _ptr(positions), _ptr(index_q), _ptr(index_w),
        _ptr(q_full), _ptr(cache_index_k), _ptr(cache_k_scale), _ptr(cache_kv), B, H, n_idx, cap,
        1 if interleave else 0, float(eps), _stream()))


# --------------------------------------------------------------------------- full-sequence preparation
def prefill_latents(qa, kv_a, ik, q_norm_w, kv_norm_w, rope, c_q, kv_out, ik_out, ik_scale, seq: int,
                    interleave: bool, eps: float) -> None:
    """Behind the GEMM that reads x_norm (see ``dsa_prefill_latents`` in the header): ``qa`` / ``kv_a`` /
    ``ik`` are 2-D row views (any may be None), ``kv_out`` ``[n_seq, cap, w]`` and ``ik_out``
    ``[n_seq, cap, D]`` (e4m3 bytes with ``ik_scale``, else the operands' type) receive their rows in
    place. ``rope``: tables of the operands' type (``RopeCaches``)."""
    _host().prefill_latents(qa, kv_a, ik, q_norm_w, kv_norm_w, rope.mla_cos, rope.mla_sin, rope.idx_cos, rope.idx_sin, c_q,
                            kv_out, ik_out, ik_scale, seq, interleave, eps)


def prefill_queries(q, nope: int, iq, w, rope, q_full, index_q, index_w, seq: int, interleave: bool) -> None:
    """Behind the GEMM that reads c_q (see ``dsa_prefill_queries``): ``q`` ``[rows, H, nope + rope]`` (a
    strided view is fine) or None, ``iq`` / ``w`` 2-D row views or None; the rope columns of ``q_full``
    ``[rows, H, kv_rank + rope]`` and ``index_q`` ``[rows, Hidx, D]`` (e4m3 bytes with ``index_w``, else
    the operands' type) are written."""
    _host().prefill_queries(q, nope, iq, w, rope.mla_cos, rope.mla_sin, rope.idx_cos, rope.idx_sin, q_full, index_q, index_w,
                            seq, interleave)


# --------------------------------------------------------------------------- exchanges between GPUs
class PeerArena:
    """ONE zeroed device allocation per rank that the other ranks of a node store into, plus the
    addresses under which this process reaches every rank's copy. Those come from CUDA IPC
    (``connect``: one process per GPU, handles exchanged over the process group) or, for ranks
    emulated on one GPU, are simply the other objects' own pointers (``local_group``)."""

    def __init__(self, nbytes: int, world: int, rank: int, device) -> None:
        import ctypes as C

        _need(1 <= world <= 8 and 0 <= rank < world, "world must be 1..8 and rank inside it")
        self.world, self.rank = world, rank
        self.arena = torch.zeros((nbytes + 255) // 256 * 256, dtype=torch.uint8, device=device)
        self._bases = [None] * world       # every rank's arena as this process addresses it
        self._bases[rank] = self.arena.data_ptr()
        self._opened = []                  # (mapped pointer, offset) of the peers' allocations
        self._C = C

    def _peer_pointers(self, offset: int):
        """ctypes array of ``world`` pointers: byte ``offset`` of every rank's arena."""
        _need(all(b is not None for b in self._bases), "not every rank's buffer is mapped: call connect() first")
        return (self._C.c_void_p * self.world)(*[b + offset for b in self._bases])

    def _mapped(self) -> None:
        """Hook: called once every rank's arena is addressable."""

    def connect(self, group=None):
        """One process per GPU: exchanges CUDA IPC handles of the arenas over ``group`` and maps
        the peers' arenas. Collective: every rank of the group calls it."""
        import torch.distributed as dist

        C = self._C
        if self.world > 1:
            handle = (C.c_ubyte * 64)()
            offset = C.c_int64(0)
            _lib.check(_lib.lib().dsa_ipc_export(self.arena.data_ptr(), handle, C.byref(offset)))
            everyone = [None] * self.world
            dist.all_gather_object(everyone, (bytes(handle), int(offset.value)), group=group)
            for r, (h, off) in enumerate(everyone):
                if r == self.rank:
                    continue
                buf = (C.c_ubyte * 64).from_buffer_copy(h)
                out = C.c_void_p(0)
                _lib.check(_lib.lib().dsa_ipc_open(buf, off, C.byref(out)))
                self._bases[r] = int(out.value)
                self._opened.append((int(out.value), off))
        self._mapped()
        if self.world > 1:
            torch.cuda.synchronize()
            dist.barrier(group=group)  # nobody stores before every arena is zeroed and mapped
        return self

    @classmethod
    def local_group(cls, *args, world: int, **kwargs):
        """``world`` ranks emulated on ONE GPU (tests, single-GPU checks): every "peer" buffer is
        an ordinary local allocation. The ranks' launches must then be enqueued one after the
        other on one stream, every push before the first wait."""
        xs = [cls(*args, world=world, rank=r, **kwargs) for r in range(world)]
        for x in xs:
            x._bases = [y.arena.data_ptr() for y in xs]
            x._mapped()
        return xs

    def close(self) -> None:
        for ptr, off in self._opened:
            _lib.lib().dsa_ipc_close(ptr, off)
        self._opened = []


class CandidateExchange(PeerArena):
    """One rank's side of the candidate exchange of a KV-sequence-sharded indexer
    (``dsa_topk_select_push`` / ``dsa_topk_merge_wait``): this rank's gather buffers
    ``[2, rows, world, topk]`` (index and logit), the flag words the other ranks post to and
    the two step counters. After set-up a step is two launches and touches no host state."""

    def __init__(self, rows: int, topk: int, world: int, rank: int, device, wait_limit_s: float = 2.0) -> None:
        self.rows, self.topk = rows, topk
        self.wait_limit_ns = int(wait_limit_s * 1e9)
        n_gather = 2 * rows * world * topk
        self._off_val = n_gather * 4
        self._off_flags = 2 * n_gather * 4
        self._off_sent = self._off_flags + world * rows * 4
        self._off_seen = self._off_sent + rows * 4
        super().__init__(self._off_seen + rows * 4, world, rank, device)
        a = self.arena
        self.gather_idx = a[:self._off_val].view(torch.int32).view(2, rows, world, topk)
        self.gather_val = a[self._off_val:self._off_flags].view(torch.float32).view(2, rows, world, topk)
        self.flags = a[self._off_flags:self._off_sent].view(torch.int32).view(world, rows)
        self.sent = a[self._off_sent:self._off_seen].view(torch.int32)
        self.seen = a[self._off_seen:self._off_seen + rows * 4].view(torch.int32)
        self._ptr_arrays = None

    def _mapped(self) -> None:
        self._ptr_arrays = (self._peer_pointers(0), self._peer_pointers(self._off_val),
                            self._peer_pointers(self._off_flags))

    @classmethod
    def local_group(cls, rows: int, topk: int, world: int, device, wait_limit_s: float = 2.0):
        return super().local_group(rows, topk, world=world, device=device, wait_limit_s=wait_limit_s)

    # -- the two launches of a step ------------------------------------------------
    def push(self, logits: torch.Tensor, seq_lens: Optional[torch.Tensor] = None, *,
             hist: Optional[torch.Tensor] = None, index_offset: int = 0, pad_value: int = -1) -> None:
        """Local top-k of ``logits[rows, n]`` whose (position + index_offset, logit) pairs are
        stored into every rank's gather buffers, then the step is posted to every rank."""
        _need(self._ptr_arrays is not None, "call connect() (or build the ranks with local_group) first")
        _need(logits.is_cuda and logits.dtype == torch.float32 and logits.dim() == 2 and logits.stride(1) == 1,
              "logits must be CUDA fp32 [rows, n] with dense rows")
        R, n = logits.shape
        _need(R == self.rows, f"logits has {R} rows, the exchange was built for {self.rows}")
        seq_lens = _lens(seq_lens, R)
        if hist is not None:
            _cuda_contig(hist, "hist", (torch.int32, torch.uint32))
            _need(hist.numel() == R * HIST_BINS, "hist must be [R, 4096]")
        gi, gv, fl = self._ptr_arrays
        slab_stride = logits.stride(0) if R > 1 else max(logits.stride(0), n)
        _lib.check(_lib.lib().dsa_topk_select_push(
            _ptr(logits), _ptr(seq_lens), _ptr(hist), R, n, slab_stride, self.topk, int(pad_value),
            int(index_offset), self.world, self.rank, gi, gv, fl, _ptr(self.sent), _stream()))

    def merge(self, out_idx: torch.Tensor, pad_value: int = -1) -> torch.Tensor:
        """Waits (on the device, bounded) for this step's candidates of every rank, then writes the
        exact global top-k into ``out_idx[rows, topk]``."""
        _cuda_contig(out_idx, "out_idx", (torch.int32,))
        _need(tuple(out_idx.shape) == (self.rows, self.topk), "out_idx must be [rows, topk]")
        _lib.check(_lib.lib().dsa_topk_merge_wait(
            _ptr(self.gather_idx), _ptr(self.gather_val), _ptr(self.flags), _ptr(self.seen), _ptr(out_idx),
            self.rows, self.world, self.topk, int(pad_value), self.wait_limit_ns, _stream()))
        return out_idx


class PeerAllReduce(PeerArena):
    """Sum of a small activation (up to ``max_elems`` values: the [B, hidden] output of a
    row-parallel projection at decode) over the ranks of a tensor-parallel group, as two small
    launches in stream order (``dsa_allreduce_push`` / ``dsa_allreduce_wait_sum``): capturable
    in a CUDA graph, deterministic (rank order), with a bounded wait on the device."""

    def __init__(self, max_elems: int, world: int, rank: int, device, wait_limit_s: float = 2.0) -> None:
        _need(max_elems > 0 and max_elems % 4 == 0, "max_elems must be a positive multiple of 4")
        self.max_elems = max_elems
        self.wait_limit_ns = int(wait_limit_s * 1e9)
        self._off_flags = 2 * world * max_elems * 4
        self._off_sent = self._off_flags + 64
        self._off_seen = self._off_sent + 16
        super().__init__(self._off_seen + 16, world, rank, device)
        a = self.arena
        self.flags = a[self._off_flags:self._off_flags + world * 4].view(torch.int32)
        self.sent = a[self._off_sent:self._off_sent + 4].view(torch.int32)
        self.seen = a[self._off_seen:self._off_seen + 4].view(torch.int32)
        self._ptr_arrays = None

    def _mapped(self) -> None:
        self._ptr_arrays = (self._peer_pointers(0), self._peer_pointers(self._off_flags))

    @classmethod
    def local_group(cls, max_elems: int, world: int, device, wait_limit_s: float = 2.0):
        return super().local_group(max_elems, world=world, device=device, wait_limit_s=wait_limit_s)

    def push(self, x: torch.Tensor) -> None:
        """Stores this rank's partial ``x`` (bf16 or fp32, contiguous) into every rank's slots."""
        _need(self._ptr_arrays is not None, "call connect() (or build the ranks with local_group) first")
        _cuda_contig(x, "x", (torch.bfloat16, torch.float32))
        n = x.numel()
        _need(n % 4 == 0 and n <= self.max_elems, f"x has {n} elements: a multiple of 4, at most {self.max_elems}")
        self._n = n
        slots, flags = self._ptr_arrays
        # the slot stride is the element count of THIS call: every rank passes the same shape
        _lib.check(_lib.lib().dsa_allreduce_push(_ptr(x), 1 if x.dtype == torch.bfloat16 else 0, n, self.world,
                                                 self.rank, slots, flags, _ptr(self.sent), _stream()))

    def wait_sum(self, out: torch.Tensor, residual: Optional[torch.Tensor] = None) -> torch.Tensor:
        """``out = sum over ranks (+ residual)``, once every rank's partial of this step is there."""
        _cuda_contig(out, "out", (torch.bfloat16, torch.float32))
        n = out.numel()
        _need(n == getattr(self, "_n", n), "out must have the element count that was pushed")
        if residual is not None:
            _cuda_contig(residual, "residual", (out.dtype,))
            _need(residual.numel() == n, "residual must have out's element count")
        _lib.check(_lib.lib().dsa_allreduce_wait_sum(
            _ptr(self.arena), _ptr(self.flags), _ptr(self.seen), _ptr(residual), _ptr(out),
            1 if out.dtype == torch.bfloat16 else 0, n, self.world, self.wait_limit_ns, _stream()))
        return out

    def all_reduce(self, x: torch.Tensor, residual: Optional[torch.Tensor] = None,
                   out: Optional[torch.Tensor] = None) -> torch.Tensor:
        self.push(x)
        return self.wait_sum(torch.empty_like(x) if out is None else out, residual)
