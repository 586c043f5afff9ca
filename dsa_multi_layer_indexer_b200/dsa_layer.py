"""One DSA transformer block on the GPU, with the reference's layer API.

Same module tree, parameter names and construction order as the reference's
``DSALayer`` (src/lagged_indexer_dsa/dsa_layer.py:55-196), so a ``state_dict``
(or a seed) gives identical weights in both. Large projections are the GEMM library's; the three
hot operations -- indexer logits, top-k selection, sparse MLA -- and, without gradients and with plain
modules, the norms, rotary embeddings, quantisation, SwiGLU product, small fp32 products and the
projections of a few decode rows go to the CUDA library (otherwise torch ops, module by module):

* production geometry (576-wide latent, 128-wide index keys) in bf16: FP8
  tcgen05 scan, exact top-k, split-K bf16 attention;
* any other geometry or fp32 weights: the library's fp32 kernels, which follow
  the reference arithmetic (attention_core.py:27-160) to ~1e-5.

Beside the reference's full-sequence methods there is a decode form
(``decode_project`` / ``decode_indexer`` / ``decode_attention``) over per-layer
caches, which the reference layer lacks.
"""

from __future__ import annotations

import dataclasses
from typing import List, Optional, Tuple

import torch
from torch import nn
from torch.nn.modules import module as _module_hooks

from . import _lib, ops
from .config import DSAConfig
from .rope import apply_rotary, apply_rotary_at

# What fuse_decode_weights stacks: everything that reads x_norm, then everything that reads c_q.
_STACKS = (("_wx", ("q_a_proj", "kv_a_proj", "index_k_proj")), ("_wc", ("q_b_proj", "index_q_proj", "index_weights_proj")))


def _bare(m: nn.Module, cls: type) -> bool:
    """Whether calling ``m`` is ``cls.forward`` and nothing else: no subclass, no hooks (its own or those of every
    module), no replaced ``forward``."""
    d = m.__dict__
    return (m.__class__ is cls and not d["_forward_hooks"] and not d["_forward_pre_hooks"] and "forward" not in d
            and not _module_hooks._global_forward_hooks and not _module_hooks._global_forward_pre_hooks)


def _plain_weights(mods, names, dtype: torch.dtype) -> Optional[List[torch.Tensor]]:
    """The weights of the named modules, each a bias-free ``nn.Linear`` of ``dtype`` that only multiplies by its own -
    nothing hooked, replaced, patched or quantised - or None. (Hooks of every module: see ``_bare``.)"""
    return _lib.host().plain_weights(mods, names, nn.Linear, nn.Parameter, torch.Tensor, dtype == torch.bfloat16)


# The linear projections of a layer, in construction order.
_PROJECTIONS = ("q_a_proj", "q_b_proj", "kv_a_proj", "kv_b_proj", "o_proj", "index_q_proj", "index_k_proj",
                "index_weights_proj", "gate_proj", "up_proj", "down_proj")


@dataclasses.dataclass
class RopeCaches:
    """Rotary tables shared by all layers (reference dsa_layer.py:32-39)."""

    mla_cos: torch.Tensor
    mla_sin: torch.Tensor
    idx_cos: torch.Tensor
    idx_sin: torch.Tensor


class RMSNorm(nn.Module):
    def __init__(self, dim: int, eps: float) -> None:
        super().__init__()
        self.weight = nn.Parameter(torch.ones(dim))
        self.eps = eps

    def add_forward(self, x: torch.Tensor, delta: torch.Tensor):
        """``(x + delta, self(x + delta))``: the residual addition and this norm, one
        launch for bf16 and fp32 rows on a CUDA device, two separate steps otherwise."""
        if (x.is_cuda and not torch.is_grad_enabled() and x.dtype == delta.dtype and x.shape == delta.shape
                and (x.dtype == torch.float32
                     or (x.dtype == torch.bfloat16 and x.shape[-1] % 8 == 0 and x.shape[-1] <= 8192))):
            return ops.add_rmsnorm(x, delta, self.weight, self.eps)
        s = x + delta
        return s, self(s)

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        if x.is_cuda and x.dtype in (torch.float32, torch.bfloat16):
            return ops.rmsnorm(x, self.weight, self.eps)  # one launch
        xf = x.float()
        inv = torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + self.eps)
        return (xf * inv * self.weight.float()).to(x.dtype)


def add_norm(norm: nn.Module, x: torch.Tensor, delta: torch.Tensor):
    """``(x + delta, norm(x + delta))``, in one launch where the norm is a plain RMSNorm (``add_forward``)."""
    if _bare(norm, RMSNorm):
        return norm.add_forward(x, delta)
    s = x + delta
    return s, norm(s)


@dataclasses.dataclass
class LayerDecodeCache:
    """Decode caches of one layer for ``n_seq`` sequences of capacity ``cap``.

    fp8 mode: index_k e4m3 ``[n_seq, cap, 128]`` + k_scale fp32, kv bf16
    ``[n_seq, cap, 576]``. fp32 mode: index_k and kv are fp32 of any width."""

    index_k: torch.Tensor
    k_scale: Optional[torch.Tensor]
    kv: torch.Tensor

    @property
    def capacity(self) -> int:
        return self.kv.shape[1]


@dataclasses.dataclass
class IndexerWorkspace:
    """Persistent buffers of one layer's decode indexer: logits slab, the scan's
    histogram (zero once, re-armed by the select), top-k scratch and result."""

    logits: torch.Tensor
    hist: Optional[torch.Tensor]
    topk_ws: torch.Tensor
    indices: torch.Tensor

    @staticmethod
    def create(n_seq: int, capacity: int, topk: int, device, fp8: bool) -> "IndexerWorkspace":
        slab = (capacity + 3) // 4 * 4
        return IndexerWorkspace(
            torch.empty(n_seq, slab, dtype=torch.float32, device=device),
            torch.zeros(n_seq, ops.HIST_BINS, dtype=torch.int32, device=device) if fp8 else None,
            ops.topk_workspace(n_seq, capacity, device),
            torch.full((n_seq, topk), -1, dtype=torch.int32, device=device))


@dataclasses.dataclass
class FullOperands:
    """A full-sequence layer's operands of the scan and the attention (``DSALayer.full_operands``).

    With ``weights`` (the fused chain's): ready for the kernels -- q [B*S,H,Dqk], kv [B,cap,Dqk], iq / iw /
    ik (/ ik_scale) of the FP8 scan (ik [B,cap,128] e4m3 bytes) or of the fp32 scan. Otherwise the torch
    tensors as computed."""

    b: int
    s: int
    lens: torch.Tensor  # int32 [B*S]: causally visible keys of every row
    weights: Optional[List[torch.Tensor]]
    q: Optional[torch.Tensor]
    kv: Optional[torch.Tensor]
    iq: Optional[torch.Tensor]
    iw: Optional[torch.Tensor]
    ik: Optional[torch.Tensor]
    ik_scale: Optional[torch.Tensor]

    @property
    def fused(self) -> bool:
        return self.weights is not None


def _pad_heads(t: torch.Tensor, multiple: int) -> torch.Tensor:
    """Zero-pads dim 1 (heads) to a multiple; zero queries attend uniformly and
    are dropped by the caller (reference fused_decode.py:38-43)."""
    h = t.shape[1]
    extra = (-h) % multiple
    if extra == 0:
        return t
    pad = torch.zeros(t.shape[0], extra, *t.shape[2:], dtype=t.dtype, device=t.device)
    return torch.cat([t, pad], dim=1)


class DSALayer(nn.Module):
    def __init__(self, config: DSAConfig) -> None:
        super().__init__()
        self.config = config
        c = config
        h = c.num_attention_heads
        self.attn_norm = RMSNorm(c.hidden_size, c.rms_norm_eps)
        self.ffn_norm = RMSNorm(c.hidden_size, c.rms_norm_eps)
        # MLA query path
        self.q_a_proj = nn.Linear(c.hidden_size, c.q_lora_rank, bias=False)
        self.q_a_layernorm = RMSNorm(c.q_lora_rank, c.rms_norm_eps)
        self.q_b_proj = nn.Linear(c.q_lora_rank, h * (c.qk_nope_head_dim + c.qk_rope_head_dim), bias=False)
        # MLA key/value path
        self.kv_a_proj = nn.Linear(c.hidden_size, c.kv_lora_rank + c.qk_rope_head_dim, bias=False)
        self.kv_a_layernorm = RMSNorm(c.kv_lora_rank, c.rms_norm_eps)
        self.kv_b_proj = nn.Linear(c.kv_lora_rank, h * (c.qk_nope_head_dim + c.v_head_dim), bias=False)
        self.o_proj = nn.Linear(h * c.v_head_dim, c.hidden_size, bias=False)
        # lightning indexer
        self.index_q_proj = nn.Linear(c.q_lora_rank, c.index_n_heads * c.index_head_dim, bias=False)
        self.index_k_proj = nn.Linear(c.hidden_size, c.index_head_dim, bias=False)
        self.index_weights_proj = nn.Linear(c.q_lora_rank, c.index_n_heads, bias=False)
        # SwiGLU MLP
        self.gate_proj = nn.Linear(c.hidden_size, c.intermediate_size, bias=False)
        self.up_proj = nn.Linear(c.hidden_size, c.intermediate_size, bias=False)
        self.down_proj = nn.Linear(c.intermediate_size, c.hidden_size, bias=False)
        # Set by DSAModel.tensor_parallel: this module then holds one rank's heads and MLP columns,
        # and the outputs of o_proj / down_proj are partial sums that `tp.reduce` completes.
        self.tp = None

    def _reduced(self, partial: torch.Tensor) -> torch.Tensor:
        return partial if self.tp is None else self.tp.reduce(partial)

    # ------------------------------------------------------------------ helpers
    def _fast_path(self, t: torch.Tensor) -> bool:
        """True when the FP8/bf16 tensor-core kernels apply to tensors like ``t``."""
        return self.config.is_production_geometry and t.dtype == torch.bfloat16

    @property
    def sm_scale(self) -> float:
        # the reference layer uses sparse_mla_core's default D_qk ** -0.5 (attention_core.py:141-142)
        return self.config.qk_head_dim ** -0.5

    def _w_uk_uv(self) -> Tuple[torch.Tensor, torch.Tensor]:
        c = self.config
        w = self.kv_b_proj.weight.view(c.num_attention_heads, c.qk_nope_head_dim + c.v_head_dim, c.kv_lora_rank)
        return w[:, : c.qk_nope_head_dim, :], w[:, c.qk_nope_head_dim:, :]

    # ------------------------------------------------------------------ stacked decode projections
    def fuse_decode_weights(self) -> None:
        """Stacks the weights of the three projections that read x_norm (q_a, kv_a,
        index_k) and of the three that read c_q (q_b, index_q, index_weights), so a
        decode step needs two GEMVs instead of six small launches. The parameters
        become views of the stacked tensors: no extra memory, ``state_dict`` and
        ``load_state_dict`` keep working, and moving or casting the module afterwards
        simply drops the stacking (``decode_project`` notices and uses the six)."""
        with torch.no_grad():
            for name, parts in _STACKS:
                mods = [self._modules[p] for p in parts]
                stacked = torch.cat([m.weight for m in mods], dim=0)
                row = 0
                for m in mods:
                    n = m.weight.shape[0]
                    m.weight.data = stacked[row:row + n]
                    row += n
                setattr(self, name, stacked)

    def _stacked(self) -> bool:
        """Whether the stacked weights are still the six parameters' own memory (any of them may have been given
        other memory since, by assignment to the parameter or its data)."""
        d, mods = self.__dict__, self._modules
        for name, parts in _STACKS:
            stack = d.get(name)
            if stack is None:
                return False
            at, step = stack.data_ptr(), stack.stride(0) * stack.element_size()
            for part in parts:
                w = mods[part].weight
                if w.data_ptr() != at or w.dtype != stack.dtype:
                    return False
                at += w.shape[0] * step
        return True

    # ------------------------------------------------------------------ projections (torch)
    def q_latent(self, x_norm: torch.Tensor) -> torch.Tensor:
        """c_q = q_a_layernorm(q_a_proj(x_norm)), shared by attention and indexer."""
        return self.q_a_layernorm(self.q_a_proj(x_norm))

    def _mla_qkv(self, x_norm, c_q, rope: RopeCaches):
        c = self.config
        b, s, _ = x_norm.shape
        h = c.num_attention_heads
        q = self.q_b_proj(c_q).view(b, s, h, c.qk_nope_head_dim + c.qk_rope_head_dim)
        q_nope, q_rope = q.split([c.qk_nope_head_dim, c.qk_rope_head_dim], dim=-1)
        q_rope = apply_rotary(q_rope.transpose(1, 2), rope.mla_cos, rope.mla_sin).transpose(1, 2)
        kv_a = self.kv_a_proj(x_norm)
        c_kv, k_rope = kv_a.split([c.kv_lora_rank, c.qk_rope_head_dim], dim=-1)
        c_kv = self.kv_a_layernorm(c_kv)
        k_rope = apply_rotary(k_rope.unsqueeze(1), rope.mla_cos, rope.mla_sin).squeeze(1)
        w_uk, _ = self._w_uk_uv()
        q_abs = torch.einsum("bshd,hdl->bshl", q_nope, w_uk)  # absorb W_UK into the query
        return torch.cat([q_abs, q_rope], dim=-1), torch.cat([c_kv, k_rope], dim=-1)

    def _project_output(self, o_latent: torch.Tensor) -> torch.Tensor:
        c = self.config
        _, w_uv = self._w_uk_uv()
        o = torch.einsum("bshl,hdl->bshd", o_latent, w_uv)
        return self._reduced(self.o_proj(o.reshape(o.shape[0], o.shape[1], c.num_attention_heads * c.v_head_dim)))

    def _indexer_qkw(self, x_norm, c_q, rope: RopeCaches):
        c = self.config
        b, s, _ = x_norm.shape
        il = c.indexer_rope_interleave
        iq = self.index_q_proj(c_q).view(b, s, c.index_n_heads, c.index_head_dim)
        iq = apply_rotary(iq.transpose(1, 2), rope.idx_cos, rope.idx_sin, interleave=il).transpose(1, 2)
        ik = apply_rotary(self.index_k_proj(x_norm).unsqueeze(1), rope.idx_cos, rope.idx_sin, interleave=il).squeeze(1)
        return iq, ik, self.index_weights_proj(c_q)

    # ------------------------------------------------------------------ hot ops (CUDA library)
    @staticmethod
    def _causal_lens(b: int, s: int, device) -> torch.Tensor:
        return torch.arange(1, s + 1, dtype=torch.int32, device=device).repeat(b)

    def _select(self, iq, ik, w, seq_lens, rows_per_seq: int, pad_value: int) -> torch.Tensor:
        """Top-k key positions per query row. iq [R,H,D], ik [n_seq,N,D], w [R,H]."""
        topk = self.config.index_topk
        if self._fast_path(iq):
            iq8, sq = ops.quantize_e4m3_rowwise(iq.float().contiguous())
            ik8, sk = ops.quantize_e4m3_rowwise(ik.float().contiguous())
            logits = ops.indexer_scan_fp8(iq8, (sq * w.float()).contiguous(), ik8, sk, seq_lens,
                                          rows_per_seq=rows_per_seq)
        else:
            logits = ops.indexer_scan_f32(iq.float().contiguous(), w.float().contiguous(), ik.float().contiguous(),
                                          seq_lens, rows_per_seq=rows_per_seq)
        return ops.topk_select(logits, topk, seq_lens, pad_value=pad_value)

    def _attend(self, q, kv, indices, seq_lens, rows_per_seq: int) -> torch.Tensor:
        """Latent attention output [R,H,Dv] of sequences from their first position. q [R,H,Dqk], kv [n_seq,N,Dqk];
        indices int32 or None (dense)."""
        c = self.config
        if self._fast_path(q):
            h = q.shape[1]
            out = ops.sparse_mla_decode(_pad_heads(q, ops.HEAD_BLOCK).contiguous(), kv.contiguous(), indices,
                                        self.sm_scale, seq_lens, rows_per_seq=rows_per_seq, prompt=True)
            return out[:, :h]
        out = ops.sparse_mla_f32(q.float().contiguous(), kv.float().contiguous(), indices, c.kv_lora_rank,
                                 self.sm_scale, seq_lens, rows_per_seq=rows_per_seq)
        return out.to(q.dtype)

    # ------------------------------------------------------------------ full sequence
    def full_operands(self, x_norm, rope: RopeCaches, c_q=None, attention: bool = True, indexer: bool = True,
                      cache: Optional["LayerDecodeCache"] = None, lens: Optional[torch.Tensor] = None) -> "FullOperands":
        """Everything a full-sequence layer computes from x_norm [B,S,hidden] before its scan and its
        attention, once for both. With a ``cache`` the latent rows and index keys are written to (and
        read from) the first S rows of the cache. ``lens``: the causal lengths, if the caller has them."""
        b, s, _ = x_norm.shape
        if lens is None:
            lens = self._causal_lens(b, s, x_norm.device)
        weights = self._full_weights(x_norm)
        if weights is not None and (cache is None or self._cache_fits(cache, x_norm)):
            return self._full_operands_fused(weights, x_norm, rope, c_q, attention, indexer, cache, lens)
        if c_q is None:
            c_q = self.q_latent(x_norm)
        q = kv = iq = ik = w = None
        if attention or cache is not None:
            q, kv = self._mla_qkv(x_norm, c_q, rope)
            q = q.reshape(b * s, *q.shape[2:])
        if indexer or cache is not None:
            iq, ik, w = self._indexer_qkw(x_norm, c_q, rope)
            iq, w = iq.reshape(b * s, *iq.shape[2:]), w.reshape(b * s, -1)
        if cache is not None:
            cache.kv[:, :s] = kv.to(cache.kv.dtype)
            if cache.k_scale is not None:
                ik8, sk = ops.quantize_e4m3_rowwise(ik.float().contiguous())
                cache.index_k[:, :s] = ik8.view(torch.uint8)
                cache.k_scale[:, :s] = sk
            else:
                cache.index_k[:, :s] = ik.float()
        return FullOperands(b, s, lens, None, q, kv, iq, w, ik, None)

    def _full_weights(self, t: torch.Tensor) -> Optional[List[torch.Tensor]]:
        """The projections' weights, in construction order, where the fused full-sequence chain applies
        to ``t``, else None: it has no autograd or autocast, knows the fp32 form of any geometry and the
        bf16 / e4m3 form of the production geometry, and needs every projection to be a plain
        ``nn.Linear`` (not replaced, no bias, no hooks on it). It norms the two latents itself: their norms
        must be plain too, with one eps and weights of ``t``'s type (the module converts them)."""
        dtype = t.dtype
        if not (t.is_cuda and (dtype == torch.float32 or self._fast_path(t))) or torch.is_grad_enabled() or torch.is_autocast_enabled():
            return None
        if dtype == torch.bfloat16 and self.config.qk_nope_head_dim % 4:  # (8-byte reads behind the query heads' nope part)
            return None
        mods = self._modules
        qn, kn = mods["q_a_layernorm"], mods["kv_a_layernorm"]
        if not (_bare(qn, RMSNorm) and _bare(kn, RMSNorm) and qn.eps == kn.eps and qn.weight.dtype == dtype == kn.weight.dtype):
            return None
        return _plain_weights(mods, _PROJECTIONS, dtype)

    def _cache_fits(self, cache: "LayerDecodeCache", x: torch.Tensor) -> bool:
        """Whether the fused chain can write ``cache`` in place: a dense cache of the scan's form and the
        activations' type, one sequence each, on their device. Any other is filled by assignment, which
        converts, broadcasts and copies across devices, or refuses."""
        b, s, _ = x.shape
        fp8 = self._fast_path(x)
        kv, ik, scale = cache.kv, cache.index_k, cache.k_scale
        return ((scale is not None) == fp8 and kv.dtype == x.dtype and ik.dtype == (torch.uint8 if fp8 else x.dtype)
                and (not fp8 or scale.dtype == torch.float32)
                and all(t.device == x.device and t.is_contiguous() and t.shape[0] == b and t.shape[1] >= s
                        for t in (kv, ik, scale) if t is not None))

    def _full_operands_fused(self, weights, x_norm, rope, c_q, attention, indexer, cache, lens) -> "FullOperands":
        c = self.config
        b, s, _ = x_norm.shape
        dt = x_norm.dtype
        fp8 = self._fast_path(x_norm)
        q_a, q_b, kv_a, kv_b, _, iq_w, ik_w, w_w = weights[:8]
        if rope.mla_cos.dtype != dt:
            rope = RopeCaches(*(t.to(dt) for t in (rope.mla_cos, rope.mla_sin, rope.idx_cos, rope.idx_sin)))
        wx = wc = None
        if fp8 and self._stacked():
            wx, wc = self._wx, self._wc
        kv = ik = ik_scale = None
        if cache is not None:
            kv, ik, ik_scale = cache.kv, cache.index_k, cache.k_scale
        parts = _lib.host().full_operands(
            x_norm, s, c_q, wx, wc, q_a, kv_a, ik_w, q_b, iq_w, w_w, self.q_a_layernorm.weight, self.kv_a_layernorm.weight,
            kv_b, rope.mla_cos, rope.mla_sin, rope.idx_cos, rope.idx_sin, kv, ik, ik_scale, attention, indexer, fp8,
            c.num_attention_heads, c.qk_nope_head_dim, c.index_n_heads, c.indexer_rope_interleave, self.q_a_layernorm.eps)
        return FullOperands(b, s, lens, weights, *parts)

    def full_select(self, op: "FullOperands", pad_value: int = -1, padded: bool = True) -> torch.Tensor:
        """int32 [B*S, topk] selected key positions of every row. ``padded`` False: without the columns
        that no row of a short sequence can fill (min(topk, S) columns)."""
        if op.weights is None:
            return self._select(op.iq, op.ik, op.iw, op.lens, op.s, pad_value)
        topk = self.config.index_topk if padded else min(self.config.index_topk, op.s)
        if op.ik_scale is not None:
            logits = ops.indexer_scan_fp8(op.iq, op.iw, op.ik, op.ik_scale, op.lens, rows_per_seq=op.s, ctx=op.s)
        else:
            logits = ops.indexer_scan_f32(op.iq, op.iw, op.ik, op.lens, rows_per_seq=op.s, ctx=op.s)
        return ops.topk_select(logits, topk, op.lens, pad_value=pad_value)

    def full_attend(self, op: "FullOperands", indices: Optional[torch.Tensor]) -> torch.Tensor:
        """Attention hidden output [B,S,hidden]; indices int32 [B*S, topk] or None (dense causal)."""
        c = self.config
        if op.weights is None:
            o = self._attend(op.q, op.kv, indices, op.lens, op.s)
            return self._project_output(o.view(op.b, op.s, *o.shape[1:]))
        h = op.q.shape[1]
        if op.q.dtype == torch.bfloat16:
            o = ops.sparse_mla_decode(_pad_heads(op.q, ops.HEAD_BLOCK), op.kv, indices, self.sm_scale, op.lens,
                                      rows_per_seq=op.s, dense_keys=op.s, prompt=True)
        else:
            o = ops.sparse_mla_f32(op.q, op.kv, indices, c.kv_lora_rank, self.sm_scale, op.lens, rows_per_seq=op.s)
        return self._reduced(_lib.host().project_output(o, op.weights[3], op.weights[4], h, c.v_head_dim).view(op.b, op.s, -1))

    # ------------------------------------------------------------------ reference API (full sequence)
    def indexer_indices(self, x_norm, rope: RopeCaches, c_q=None) -> torch.Tensor:
        """int64 [B,S,topk] selected key positions, padded with S (reference :145-153)."""
        op = self.full_operands(x_norm, rope, c_q, attention=False)
        return self.full_select(op, pad_value=op.s).view(op.b, op.s, -1).long()

    def attention_output(self, x_norm, rope: RopeCaches, indices, c_q=None) -> torch.Tensor:
        """Attention hidden output; ``indices=None`` is dense causal (reference :156-171)."""
        op = self.full_operands(x_norm, rope, c_q, indexer=False)
        idx32 = None if indices is None else indices.reshape(op.b * op.s, -1).to(torch.int32).contiguous()
        return self.full_attend(op, idx32)

    def fused_attention_and_indices(self, x_norm, rope: RopeCaches, attn_indices, produce_indexer: bool = True):
        """One shared query latent for both consumers (reference :173-192)."""
        op = self.full_operands(x_norm, rope, indexer=produce_indexer)
        idx32 = None if attn_indices is None else attn_indices.reshape(op.b * op.s, -1).to(torch.int32).contiguous()
        attn_hidden = self.full_attend(op, idx32)
        nxt = self.full_select(op, pad_value=op.s).view(op.b, op.s, -1).long() if produce_indexer else None
        return attn_hidden, nxt

    def mlp(self, h_norm: torch.Tensor, weights=None, ahead: bool = False) -> torch.Tensor:
        if (h_norm.is_cuda and h_norm.dtype == torch.bfloat16 and h_norm.dim() == 2 and h_norm.shape[0] <= 2
                and not torch.is_grad_enabled()):
            return self._reduced(self._skinny("down_proj", ops.gemv_swiglu(h_norm, self.gate_proj.weight, self.up_proj.weight,
                                                                         ahead)))
        w = self._full_weights(h_norm) if h_norm.dim() == 3 and weights is None else weights
        if w is not None:
            y = _lib.host().mlp(h_norm.reshape(-1, h_norm.shape[2]), w[8], w[9], w[10])
            return self._reduced(y.view(h_norm.shape[0], h_norm.shape[1], -1))
        gate, up = self.gate_proj(h_norm), self.up_proj(h_norm)
        if gate.is_cuda and gate.dtype in (torch.bfloat16, torch.float32) and not torch.is_grad_enabled():
            return self._reduced(self.down_proj(ops.silu_mul(gate, up)))  # one launch instead of two
        return self._reduced(self.down_proj(torch.nn.functional.silu(gate) * up))

    # ------------------------------------------------------------------ decode form
    def _skinny(self, name: str, x: torch.Tensor) -> torch.Tensor:
        """A projection of one or two bf16 rows behind another launch of the same call: the library's GEMV, which
        starts on its weights while the kernel before it runs, unless the module is not a plain ``nn.Linear``."""
        m = self._modules[name]
        if x.shape[0] > 2 or x.dtype != torch.bfloat16 or not x.is_cuda or torch.is_grad_enabled() or not self._plain(name):
            return m(x)
        return ops.gemv(x, m.weight, ahead=True)

    def _plain(self, name: str) -> bool:
        """A bias-free bf16 ``nn.Linear`` that only multiplies, of a width that the GEMV takes."""
        w = _plain_weights(self._modules, (name,), torch.bfloat16)
        return (w is not None and not _module_hooks._global_forward_hooks and not _module_hooks._global_forward_pre_hooks
                and not torch.is_autocast_enabled() and w[0].shape[1] % 8 == 0 and w[0].is_contiguous())

    def _absorbed_rows(self, x: torch.Tensor) -> bool:
        """Whether a decode batch takes the kernels that read kv_b_proj's weight in place (one reading for all
        tokens; beyond HEAD_TOKENS rows the products are GEMMs)."""
        c, w = self.config, self.kv_b_proj.weight
        return (x.shape[0] <= ops.HEAD_TOKENS and x.dtype == torch.bfloat16 and w.__class__ in (nn.Parameter, torch.Tensor)
                and w.dtype == torch.bfloat16 and w.is_contiguous() and c.qk_nope_head_dim <= 512 and c.qk_nope_head_dim % 8 == 0 and c.q_lora_rank % 8 == 0 and not torch.is_grad_enabled())

    def new_cache(self, n_seq: int, capacity: int, device, fp8: bool) -> LayerDecodeCache:
        c = self.config
        if fp8:
            return LayerDecodeCache(
                torch.zeros(n_seq, capacity, c.index_head_dim, dtype=torch.uint8, device=device),
                torch.zeros(n_seq, capacity, dtype=torch.float32, device=device),
                torch.zeros(n_seq, capacity, c.qk_head_dim, dtype=torch.bfloat16, device=device))
        return LayerDecodeCache(
            torch.zeros(n_seq, capacity, c.index_head_dim, dtype=torch.float32, device=device), None,
            torch.zeros(n_seq, capacity, c.qk_head_dim, dtype=torch.float32, device=device))

    def fill_cache(self, cache: LayerDecodeCache, x_norm: torch.Tensor, rope: RopeCaches) -> None:
        """Writes the keys of a whole prefix x_norm [B,S,hidden] (prefill)."""
        self.full_operands(x_norm, rope, attention=False, indexer=False, cache=cache)

    def _norm_folds(self, norm: RMSNorm, x: torch.Tensor) -> bool:
        """Whether ``norm`` can run inside the projection that follows it (:func:`ops.norm_gemv`)."""
        return (_bare(norm, RMSNorm) and x.is_cuda and x.dtype == torch.bfloat16 and norm.weight.dtype == torch.bfloat16
                and not torch.is_grad_enabled() and ops.norm_gemv_fits(x.shape[0], x.shape[1]))

    def decode_residual_project(self, x, delta, rope: RopeCaches, positions, cache: LayerDecodeCache, batch_index,
                                ahead: bool = False):
        """``x + delta`` (``delta`` None: ``x``) and :func:`decode_project` of its attention norm. ``ahead`` (here
        and in the methods below): this call's first launch may read its weights while the kernels in front still
        run, as every later one does: nothing enqueued since the last launch that waited writes them (inside a
        decode step; not at its start, where whatever updates weights may be in front)."""
        wide = self._wx.shape[0] if self._stacked() else 0
        # One or two rows: the norm's launch goes. Four where the product has few outputs of long rows, which the
        # library's GEMM runs at 1.4 TB/s (norm, [2240, 7168] and the copy of its strided columns 27 us, here 13).
        if wide and x.dim() == 2 and (x.shape[0] <= 2 or (x.shape[0] <= 4 and wide <= 4096 <= x.shape[1])) and self._norm_folds(self.attn_norm, x):
            x, ya = ops.norm_gemv(x, delta, self.attn_norm.weight, self.attn_norm.eps, self._wx, ahead=ahead)
            return x, self.decode_project(x, rope, positions, cache, batch_index, ya)
        if delta is None:
            x_norm = self.attn_norm(x)
        else:
            x, x_norm = add_norm(self.attn_norm, x, delta)
        return x, self.decode_project(x_norm, rope, positions, cache, batch_index, ahead=ahead)

    def decode_mlp(self, x: torch.Tensor, attn: torch.Tensor, ahead: bool = False):
        """``(h, mlp(ffn_norm(h)))`` with ``h = x + attn``."""
        if (x.shape == attn.shape and x.dim() == 2 and x.shape[0] <= 2 and attn.dtype == x.dtype and attn.is_contiguous()
                and self._norm_folds(self.ffn_norm, x) and self._plain("gate_proj") and self._plain("up_proj")):
            h, act = ops.norm_gemv(x, attn, self.ffn_norm.weight, self.ffn_norm.eps, self.gate_proj.weight, self.up_proj.weight,
                                   ahead)
            return h, self._reduced(self._skinny("down_proj", act))
        h, h_norm = add_norm(self.ffn_norm, x, attn)
        return h, self.mlp(h_norm, ahead=ahead)

    def decode_project(self, x_norm, rope: RopeCaches, positions, cache: LayerDecodeCache, batch_index, ya=None,
                       ahead: bool = False):
        """Projections of one new token per sequence, and its keys appended to
        the caches at ``positions`` [B]. Returns (q [B,H,Dqk], index_q, index_w).

        With FP8 caches and bf16 weights everything after the GEMVs (RoPE, e4m3
        quantisation with the scale folded into the head weights, both cache
        appends, assembly of the absorbed query) is ONE launch; index_q then
        comes back already quantised (uint8) with index_w fp32. ``ya``: the stacked
        projection of ``x_norm``, where the caller has it (then only x_norm's shape is read)."""
        c = self.config
        b = x_norm.shape[0]
        h = c.num_attention_heads
        il = c.indexer_rope_interleave
        if self._stacked():  # two GEMVs: everything that reads x_norm, then everything that reads c_q
            if ya is None:
                # few output rows, long rows: the GEMM library's GEMV is latency-bound there (19-32 us against
                # 7.5 for [2240, 7168] at one token); the other shapes stay with it
                skinny = b <= 2 and x_norm.dtype == torch.bfloat16 and self._wx.shape[0] <= 4096 <= self._wx.shape[1]
                ya = ops.gemv(x_norm, self._wx, ahead) if skinny else torch.nn.functional.linear(x_norm, self._wx)
            qa, kv_a, ik_raw = ya.split(
                [c.q_lora_rank, c.kv_lora_rank + c.qk_rope_head_dim, c.index_head_dim], dim=-1)
            n = self.q_a_layernorm
            # one or two tokens: the norm runs inside the c_q-side projection, as attn_norm and ffn_norm do
            if b <= 2 and self._norm_folds(n, qa):
                yc = ops.norm_gemv(qa, None, n.weight, n.eps, self._wc, ahead=True)[1]
            else:
                c_q = n(qa)
                yc = ops.gemv(c_q, self._wc, ahead=True) if b <= 2 and c_q.dtype == torch.bfloat16 else torch.nn.functional.linear(c_q, self._wc)
            q, iq_raw, w = yc.split(
                [h * (c.qk_nope_head_dim + c.qk_rope_head_dim), c.index_n_heads * c.index_head_dim, c.index_n_heads],
                dim=-1)
        else:
            c_q = self.q_latent(x_norm)
            q = self.q_b_proj(c_q)
            kv_a = self.kv_a_proj(x_norm)
            iq_raw = self.index_q_proj(c_q)
            ik_raw = self.index_k_proj(x_norm)
            w = self.index_weights_proj(c_q)
        fused = cache.k_scale is not None and x_norm.dtype == torch.bfloat16
        if fused:
            index_q = torch.empty(b, c.index_n_heads, c.index_head_dim, dtype=torch.uint8, device=x_norm.device)
            index_w = torch.empty(b, c.index_n_heads, dtype=torch.float32, device=x_norm.device)
            q_full = torch.empty(b, h, c.qk_head_dim, dtype=torch.bfloat16, device=x_norm.device)
            norm_w = self.kv_a_layernorm.weight
            if norm_w.dtype != torch.bfloat16:  # (norms kept in fp32: the launch reads bf16, as ops.rmsnorm converts it)
                norm_w = norm_w.to(torch.bfloat16)
            if self._absorbed_rows(x_norm):
                ops.decode_token(iq_raw, w, ik_raw, kv_a, q, self.kv_b_proj.weight, norm_w, rope.mla_cos,
                                 rope.mla_sin, rope.idx_cos, rope.idx_sin, positions, index_q, index_w, q_full, cache.index_k,
                                 cache.k_scale, cache.kv, il, c.rms_norm_eps, ahead=True)
                return q_full, index_q, index_w
        q = q.contiguous().view(b, h, c.qk_nope_head_dim + c.qk_rope_head_dim)  # (a column range of a stacked product)
        iq_raw = iq_raw.reshape(b, c.index_n_heads, c.index_head_dim)
        q_nope, q_rope = q.split([c.qk_nope_head_dim, c.qk_rope_head_dim], dim=-1)
        w_uk, _ = self._w_uk_uv()
        q_abs = torch.einsum("bhd,hdl->bhl", q_nope, w_uk)
        if fused:
            ops.decode_prep(iq_raw.contiguous(), w.contiguous(), ik_raw.contiguous(), kv_a.contiguous(),
                            q_abs.contiguous(), q_rope, norm_w, rope.mla_cos, rope.mla_sin,
                            rope.idx_cos, rope.idx_sin, positions, index_q, index_w, q_full, cache.index_k,
                            cache.k_scale, cache.kv, il, c.rms_norm_eps)
            return q_full, index_q, index_w
        q_rope = apply_rotary_at(q_rope, rope.mla_cos, rope.mla_sin, positions)
        c_kv, k_rope = kv_a.split([c.kv_lora_rank, c.qk_rope_head_dim], dim=-1)
        k_rope = apply_rotary_at(k_rope, rope.mla_cos, rope.mla_sin, positions)
        q_full = torch.cat([q_abs, q_rope], dim=-1)
        kv_row = torch.cat([self.kv_a_layernorm(c_kv), k_rope], dim=-1)
        cache.kv[batch_index, positions] = kv_row.to(cache.kv.dtype)
        iq = apply_rotary_at(iq_raw, rope.idx_cos, rope.idx_sin, positions, interleave=il)
        ik = apply_rotary_at(ik_raw, rope.idx_cos, rope.idx_sin, positions, interleave=il)
        if cache.k_scale is not None:
            ik8, sk = ops.quantize_e4m3_rowwise(ik.float().contiguous())
            cache.index_k[batch_index, positions] = ik8.view(torch.uint8)
            cache.k_scale[batch_index, positions] = sk
        else:
            cache.index_k[batch_index, positions] = ik.float()
        return q_full, iq, w

    def decode_indexer(self, iq, w, cache: LayerDecodeCache, seq_lens, pad_value: int = -1,
                       ws: Optional["IndexerWorkspace"] = None) -> torch.Tensor:
        """int32 [B, topk] selection over each sequence's first seq_lens keys. With
        a workspace the logits slab, the histogram, the top-k scratch and the
        result live in persistent buffers (nothing is allocated per step)."""
        topk = self.config.index_topk
        if cache.k_scale is not None:
            if iq.dtype == torch.uint8:  # already quantised by decode_project's fused launch
                iq8, wf = iq, w
            else:
                iq8, sq = ops.quantize_e4m3_rowwise(iq.float().contiguous())
                wf = (sq * w.float()).contiguous()
            if ws is None:
                logits = ops.indexer_scan_fp8(iq8, wf, cache.index_k, cache.k_scale, seq_lens)
                return ops.topk_select(logits, topk, seq_lens, pad_value=pad_value)
            logits = ops.indexer_scan_fp8(iq8, wf, cache.index_k, cache.k_scale, seq_lens, out=ws.logits, hist=ws.hist)
            return ops.topk_select(logits, topk, seq_lens, hist=ws.hist, pad_value=pad_value, out_idx=ws.indices,
                                   workspace=ws.topk_ws)
        logits = ops.indexer_scan_f32(iq.float().contiguous(), w.float().contiguous(), cache.index_k, seq_lens,
                                      out=None if ws is None else ws.logits)
        if ws is None:
            return ops.topk_select(logits, topk, seq_lens, pad_value=pad_value)
        return ops.topk_select(logits, topk, seq_lens, pad_value=pad_value, out_idx=ws.indices, workspace=ws.topk_ws)

    def decode_attention(self, q, cache: LayerDecodeCache, indices, seq_lens, beside_previous: bool = False) -> torch.Tensor:
        """Attention hidden output [B, hidden] of the new tokens; indices None = dense.
        ``beside_previous``: see :func:`ops.sparse_mla_decode` (used only when the queries need no
        conversion or padding launch in front of the attention)."""
        c = self.config
        if cache.k_scale is not None:
            h = q.shape[1]
            direct = q.dtype == torch.bfloat16 and h % ops.HEAD_BLOCK == 0 and q.is_contiguous()
            o = ops.sparse_mla_decode(_pad_heads(q.to(torch.bfloat16), ops.HEAD_BLOCK).contiguous(), cache.kv,
                                      indices, self.sm_scale, seq_lens, beside_previous=beside_previous and direct)
            if self._absorbed_rows(q):
                ov = ops.value_project(self.kv_b_proj.weight, o, h, c.v_head_dim, ahead=True)
                return self._reduced(self._skinny("o_proj", ov.view(ov.shape[0], h * c.v_head_dim)))
            o = o[:, :h].to(q.dtype)
        else:
            o = ops.sparse_mla_f32(q.float().contiguous(), cache.kv, indices, c.kv_lora_rank, self.sm_scale,
                                   seq_lens).to(q.dtype)
        _, w_uv = self._w_uk_uv()
        ov = torch.einsum("bhl,hdl->bhd", o, w_uv)
        return self._reduced(self.o_proj(ov.reshape(ov.shape[0], c.num_attention_heads * c.v_head_dim)))
