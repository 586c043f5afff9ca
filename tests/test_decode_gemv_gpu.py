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
# than one CTA per SM holds, x so long that the streaming kernel's pieces are half as long, three and four rows
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


# one row per template, padded rows, a strided x, the widest row, with and without a residual and the second matrix
@pytest.mark.parametrize("b,n,k,residual", [(1, 300, 7168, True), (2, 515, 1536, False), (3, 301, 6144, True), (4, 77, 8192, True),
                                            (3, 148, 264, False), (1, 9, 8, True)])
def test_norm_gemv(ops, b, n, k, residual):
    torch.manual_seed(n + k)
    bf = lambda *s: torch.randn(*s, device="cuda").to(torch.bfloat16)
    assert ops.norm_gemv_fits(b, k)
    wide, delta, nw = bf(b, k + 64), bf(b, k) if residual else None, bf(k)
    x = wide[:, :k]
    w, u = (torch.randn(n, k, device="cuda").div_(k ** 0.5).to(torch.bfloat16) for _ in range(2))
    s, y = ops.norm_gemv(x, delta, nw, 1e-6, w)
    if residual:
        want_s, normed = ops.add_rmsnorm(x.contiguous(), delta, nw, 1e-6)
        assert torch.equal(s, want_s)
    else:
        normed = ops.rmsnorm(x.contiguous(), nw, 1e-6)
    # the sum of squares is taken in another order: 2^-20 relative in the factor, which may move a normed element
    # to its neighbour (2^-8) - few of them, counted here as if all fell on the largest products
    prod = normed.double().unsqueeze(1) * w.double().unsqueeze(0)
    moved = prod.abs().topk(min(k, 4), dim=-1).values.sum(-1) * 2.0 ** -8
    ref, mag = prod.sum(-1), prod.abs().sum(-1)
    close(y, ref, mag + moved * 2.0 ** 20)
    if b <= 2:
        s2, act = ops.norm_gemv(x, delta, nw, 1e-6, w, u)
        assert torch.equal(s2, s)
        up = ops.norm_gemv(x, delta, nw, 1e-6, u)[1]
        # as test_gemv_and_swiglu: the factors may lie one rounding from the single products
        g, v = y.double(), up.double()
        silu = torch.nn.functional.silu(g)
        dg, dv = g.abs() * 2.0 ** -7 + mag * 2.0 ** -19, v.abs() * 2.0 ** -7 + mag * 2.0 ** -19
        ds = 1.1 * dg + (silu.abs() + 1.1 * dg) * 2.0 ** -8
        err = ds * (v.abs() + dv) + silu.abs() * dv
        assert float(((act.double() - silu * v).abs() - err - ((silu * v).abs() + err) * 2.0 ** -8).max()) <= 0.0


# one to eight tokens, remainders of the row groups (nope) and of the rows per warp step (v), padded heads
@pytest.mark.parametrize("B,H,nope,v,pad", [(1, 128, 128, 128, 0), (2, 64, 192, 256, 0), (3, 5, 36, 7, 11), (8, 16, 512, 66, 0), (5, 8, 64, 128, 0)])
def test_absorbed_projections(ops, B, H, nope, v, pad):
    torch.manual_seed(H + nope)
    bf = lambda *s: torch.randn(*s, device="cuda").to(torch.bfloat16)
    kv_b = bf(H * (nope + v), 512).div_(16)
    n_idx, cap, d = 64, 40, H * (nope + 64)
    yc, ya = bf(B, d + n_idx * 129), bf(B, 16 + 576 + 128)  # stacked projections; their ranges are strided
    q, iq, w = yc.split([d, n_idx * 128, n_idx], dim=-1)
    _, kv_a, ik = ya.split([16, 576, 128], dim=-1)
    tab = [torch.rand(cap, n, device="cuda").to(torch.bfloat16) for n in (64, 64, 128, 128)]
    pos = torch.randint(0, cap, (B,), device="cuda")
    norm_w = bf(512)

    def outputs():
        return (torch.zeros(B, n_idx, 128, dtype=torch.uint8, device="cuda"), torch.zeros(B, n_idx, device="cuda"),
                torch.zeros(B, H, 576, dtype=torch.bfloat16, device="cuda"), torch.zeros(B, cap, 128, dtype=torch.uint8, device="cuda"),
                torch.zeros(B, cap, device="cuda"), torch.zeros(B, cap, 576, dtype=torch.bfloat16, device="cuda"))

    got, want = outputs(), outputs()
    ops.decode_token(iq, w, ik, kv_a, q, kv_b, norm_w, *tab, pos, *got, False, 1e-6)
    q3 = q.reshape(B, H, nope + 64).contiguous()
    weight = kv_b.view(H, nope + v, 512).double()
    ref = torch.einsum("bhd,hdl->bhl", q3[..., :nope].double(), weight[:, :nope])
    close(got[2][..., :512], ref, torch.einsum("bhd,hdl->bhl", q3[..., :nope].double().abs(), weight[:, :nope].abs()))
    # everything else: the launch that takes the absorbed query, bit for bit
    ops.decode_prep(iq.reshape(B, n_idx, 128).contiguous(), w.contiguous(), ik.contiguous(), kv_a.contiguous(),
                    got[2][..., :512].contiguous(), q3[..., nope:], norm_w, *tab, pos, *want, False, 1e-6)
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    o = bf(B, H + pad, 512)
    ov = ops.value_project(kv_b, o, H, v)
    ref = torch.einsum("bhl,hdl->bhd", o[:, :H].double(), weight[:, nope:])
    close(ov, ref, torch.einsum("bhl,hdl->bhd", o[:, :H].double().abs(), weight[:, nope:].abs()))


def test_weights_may_come_from_the_launch_in_front(ops):
    """Without ``ahead`` a weight is read when the kernels in front are done, also one that releases its
    dependents before it has stored anything, as this library's norms do."""
    torch.manual_seed(3)
    n, k = 8192, 2048
    bf = lambda *s: torch.randn(*s, device="cuda").to(torch.bfloat16)
    x, ones, raw = bf(2, k), torch.ones(k, dtype=torch.bfloat16, device="cuda"), [bf(n, k) for _ in range(4)]
    ref = [ops.rmsnorm(r, ones, 1e-6) for r in raw]
    torch.cuda.synchronize()
    fresh = lambda i: ops.rmsnorm(raw[i], ones, 1e-6)  # (into whatever memory the last one has left)
    for i in range(4):
        torch.cuda.synchronize()
        assert torch.equal(ops.gemv(x, fresh(i)), ops.gemv(x, ref[i]))
        assert torch.equal(ops.gemv_swiglu(x, fresh(i), ref[i]), ops.gemv_swiglu(x, ref[i], ref[i]))
        assert torch.equal(ops.norm_gemv(x, None, ones, 1e-6, fresh(i))[1], ops.norm_gemv(x, None, ones, 1e-6, ref[i])[1])
    heads = raw[0].view(-1, 512)[:16 * 256]
    unit = torch.ones(512, dtype=torch.bfloat16, device="cuda")
    o = bf(2, 16, 512)
    want = ops.value_project(ops.rmsnorm(heads, unit, 1e-6).clone(), o, 16, 128)
    torch.cuda.synchronize()
    assert torch.equal(ops.value_project(ops.rmsnorm(heads, unit, 1e-6), o, 16, 128), want)


@pytest.mark.parametrize("b", [1, 2, 4])
def test_reading_ahead_changes_nothing_but_the_time(ops, b):
    torch.manual_seed(b)
    bf = lambda *s: torch.randn(*s, device="cuda").to(torch.bfloat16)
    x, w, u, nw = bf(b, 1024), bf(700, 1024), bf(700, 1024), bf(1024)
    torch.cuda.synchronize()
    assert torch.equal(ops.gemv(x, w), ops.gemv(x, w, ahead=True))
    assert torch.equal(ops.norm_gemv(x, None, nw, 1e-6, w)[1], ops.norm_gemv(x, None, nw, 1e-6, w, ahead=True)[1])
    if b <= 2:
        assert torch.equal(ops.gemv_swiglu(x, w, u), ops.gemv_swiglu(x, w, u, ahead=True))
    kv_b, o = bf(16 * 256, 512), bf(b, 16, 512)
    torch.cuda.synchronize()
    assert torch.equal(ops.value_project(kv_b, o, 16, 128), ops.value_project(kv_b, o, 16, 128, ahead=True))


# both sides of the lines between the row kernel and the streaming kernel: few short rows of W, and rows of x too
# long to lie beside the streaming kernel's ring
@pytest.mark.parametrize("b,n,k", [(1, 256, 512), (2, 256, 520), (3, 257, 2048), (4, 1280, 2048), (3, 1281, 2048), (1, 1024, 2048), (1, 1025, 2048), (2, 1480, 1416), (2, 1481, 64), (3, 5, 8),
                                   (1, 9, 90112), (2, 9, 47104), (4, 9, 24576), (3, 9, 24576)])
def test_gemv_by_either_kernel(ops, b, n, k):
    torch.manual_seed(n + k)
    x = torch.randn(b, k + 16, device="cuda").to(torch.bfloat16)[:, 8:k + 8]
    w = torch.randn(n, k, device="cuda").div_(k ** 0.5).to(torch.bfloat16)
    close(ops.gemv(x, w), x.double() @ w.double().T, x.double().abs() @ w.double().abs().T)
    torch.cuda.synchronize()
    assert torch.equal(ops.gemv(x, w), ops.gemv(x, w, ahead=True))
