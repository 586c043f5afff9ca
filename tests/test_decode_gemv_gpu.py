"""GPU tests of the decode projections that read their weights ahead of the dependency wait, against
fp64 products of the same bf16 operands: one bf16 rounding (2^-8 relative) plus fp32 accumulation
(2^-23 per term of the row's magnitudes)."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from dsa_multi_layer_indexer_b200 import _lib, ops as _ops

    yield _ops
    _lib.check_device_status()


def close(got, ref, mag):
    assert float(((got.double() - ref).abs() - ref.abs() * 2.0 ** -8 - mag * 2.0 ** -20).max()) <= 0.0


# k below, at and above one piece of a row, uneven last pieces, odd row counts, fewer rows than SMs, more sums
# than one CTA per SM holds, x too long for the streaming kernel, three and four rows
@pytest.mark.parametrize("b,n,k", [(1, 1, 8), (1, 515, 16384), (2, 2240, 7168), (1, 7168, 520), (2, 18432, 264), (4, 300, 2048),
                                   (3, 4097, 512), (1, 1001, 1024), (2, 77, 2056), (2, 320001, 64), (1, 600001, 8), (1, 9, 49152),
                                   (2, 31, 24576)])
def test_gemv_and_swiglu(ops, b, n, k):
    torch.manual_seed(n + k)
    x = torch.randn(b, k, device="cuda").to(torch.bfloat16)
    w, u = (torch.randn(n, k, device="cuda").div_(k ** 0.5).to(torch.bfloat16) for _ in range(2))
    g = x.double() @ w.double().T
    close(ops.gemv(x, w), g, x.double().abs() @ w.double().abs().T)
    if b <= 2:
        # the factors within the bound above (the sums' order differs from the single product's), |silu'| < 1.1,
        # and a rounding each of silu and of the product
        up, mag = x.double() @ u.double().T, [x.double().abs() @ m.double().abs().T * 2.0 ** -20 for m in (w, u)]
        dg, du = g.abs() * 2.0 ** -8 + mag[0], up.abs() * 2.0 ** -8 + mag[1]
        silu = torch.nn.functional.silu(g)
        ds = 1.1 * dg + (silu.abs() + 1.1 * dg) * 2.0 ** -8
        err = ds * (up.abs() + du) + silu.abs() * du
        err = err + ((silu * up).abs() + err) * 2.0 ** -8
        assert float(((ops.gemv_swiglu(x, w, u).double() - silu * up).abs() - err).max()) <= 0.0
    view = torch.randn(b, k + 24, device="cuda").to(torch.bfloat16)[:, :k]
    assert torch.equal(ops.gemv(view, w), ops.gemv(view.contiguous(), w))


@pytest.mark.parametrize("B,H,nope,v,pad", [(1, 128, 128, 128, 0), (2, 64, 192, 256, 0), (1, 5, 33, 7, 11), (2, 16, 512, 32, 0)])
def test_absorbed_projections(ops, B, H, nope, v, pad):
    torch.manual_seed(H + nope)
    kv_b = torch.randn(H * (nope + v), 512, device="cuda").div_(16).to(torch.bfloat16)
    q = torch.randn(B, H, nope + 64, device="cuda").to(torch.bfloat16)
    q_full = torch.full((B, H, 576), 3.0, dtype=torch.bfloat16, device="cuda")
    ops.absorb_query(kv_b, q, nope, q_full)
    w = kv_b.view(H, nope + v, 512).double()
    ref = torch.einsum("bhd,hdl->bhl", q[..., :nope].double(), w[:, :nope])
    close(q_full[..., :512], ref, torch.einsum("bhd,hdl->bhl", q[..., :nope].double().abs(), w[:, :nope].abs()))
    assert float((q_full[..., 512:].float() - 3.0).abs().max()) == 0.0
    o = torch.randn(B, H + pad, 512, device="cuda").to(torch.bfloat16)
    ov = ops.value_project(kv_b, o, H, v)
    ref = torch.einsum("bhl,hdl->bhd", o[:, :H].double(), w[:, nope:])
    close(ov, ref, torch.einsum("bhl,hdl->bhd", o[:, :H].double().abs(), w[:, nope:].abs()))
