"""The fully connected product on csrc/fctp_tri.cu and csrc/fctp_gw.cu: output, input gradients and weight gradient against
float64 sums, over every multiplicity the kernels are built for (96: the weight gradient only), partial sample tiles, sums divided among thread blocks or
not, and an irrep of the result without any path."""
import pytest
import torch

import cuequivariance_b200 as cb

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _sums(d, w, x1, x2, g):
    """(out, gw, gx1, gx2) of the product in the dtype of the operands, rows in ir_mul layout; coefficients by magnitude when
    the operands are."""
    off = [op.offsets() for op in d.operands]
    out, gw, g1, g2 = torch.zeros_like(g), torch.zeros_like(w), torch.zeros_like(x1), torch.zeros_like(x2)
    mag = bool((w >= 0).all())
    for p in d.paths:
        sw, s1, s2, so = p.indices
        c = torch.as_tensor(p.coefficients, dtype=w.dtype)
        c = c.abs() if mag else c
        U, V, W = d.operands[0].segments[sw]
        d1, d2, d3 = c.shape
        cut = lambda t, b, s, n, m: t[:, off[b][s] : off[b][s] + n * m].view(-1, n, m)  # noqa: E731
        wp = w[0, off[0][sw] : off[0][sw] + U * V * W].view(U, V, W)
        a, b, h = cut(x1, 1, s1, d1, U), cut(x2, 2, s2, d2, V), cut(g, 3, so, d3, W)
        z = torch.einsum("ijk,ziu,zjv->zkuv", c, a, b)
        y = torch.einsum("zkw,uvw->zkuv", h, wp)
        cut(out, 3, so, d3, W).add_(torch.einsum("zkuv,uvw->zkw", z, wp))
        gw[0, off[0][sw] : off[0][sw] + U * V * W] += torch.einsum("zkuv,zkw->uvw", z, h).reshape(-1)
        cut(g1, 1, s1, d1, U).add_(torch.einsum("ijk,zjv,zkuv->ziu", c, b, y))
        cut(g2, 2, s2, d2, V).add_(torch.einsum("ijk,ziu,zkuv->zjv", c, a, y))
    return out, gw, g1, g2


@pytest.mark.parametrize("mul,lmax,batch,dtype", [
    (32, 2, 1, "float32"), (32, 2, 129, "float32"), (64, 2, 200, "float32"), (64, 1, 1000, "float32"), (96, 2, 130, "float32"),
    (128, 1, 70, "bfloat16"), (128, 2, 40, "bfloat16"), (128, 1, 300, "bfloat16"),
])
def test_against_float64_sums(mul, lmax, batch, dtype):
    s = "+".join(f"{mul}x{l}{'eo'[l % 2]}" for l in range(lmax + 1))  # noqa: E741
    dt = getattr(torch, dtype)
    m = cb.FullyConnectedTensorProduct(s, s, s, layout=cb.ir_mul, internal_weights=False, shared_weights=True)
    prog = m.f._program(torch.float32)
    assert prog._tri_channels(dt) == (0 if mul == 96 else mul) and (dt == torch.bfloat16 or prog._gw_channels() == mul)
    gen = torch.Generator().manual_seed(mul + batch)
    x1, x2, g = (torch.randn(batch, m.irreps_in1.dim, generator=gen).to(dt) for _ in range(3))
    w = (torch.randn(1, m.weight_numel, generator=gen) / mul).to(dt)
    dev = [t.to(DEV).requires_grad_(True) for t in (x1, x2, w)]
    out = m(*dev)
    got = [out.detach(), *torch.autograd.grad(out, [dev[2], dev[0], dev[1]], g.to(DEV))]
    dbl = [t.double() for t in (w, x1, x2, g)]
    ref, mag = _sums(prog.d, *dbl), _sums(prog.d, *(t.abs() for t in dbl))
    # TF32 halves: 2^-21 per product.  Sums that need not round to nearest: 36 additions of 2^-23 per accumulator; float32
    # multiply-adds: one rounding of 2^-24 per (q, a), at most 128 * 5 * 6 paths.  The weight gradient is summed over the
    # samples on other kernels: its bf16 form rounds the products of the inputs to bf16.
    terms = 2.0 ** -21 + 36 * 2.0 ** -23 + mul * 5 * 6 * 2.0 ** -24
    for name, a, b, t in zip(("out", "gw", "gx1", "gx2"), got, ref, mag):
        bound = (terms + (batch * 2.0 ** -23 if name == "gw" else 0)) * t + 1e-30
        if dt == torch.bfloat16:
            bound = bound + 2.0 ** -8 * b.abs() + (3 * 2.0 ** -8 * t if name == "gw" else 0)
        err = (a.cpu().double() - b).abs()
        assert bool((err <= bound).all()), (name, (err / bound).max().item())
        # ... and the typical error is that of float32 sums, not the worst case
        rel = (err.norm() / b.norm()).item()
        typical = 2.0 ** -8 if dt == torch.bfloat16 else 2.0 ** -19
        if mul == 96 and name == "out":
            # the memory route: up to six paths' (u, v) in one sum, eight per instruction on four accumulators that cut up to
            # 2^-23 of the sum, 2^-24 on average, with each addition
            typical = 6 * mul * mul / (8 * 4) * 2.0 ** -24
        assert rel <= typical, (name, rel)


def test_missing_paths_passes_and_second_order():
    """An irrep of the result without a path stays zero; a batch cut in two; derivatives of the gradients."""
    m = cb.FullyConnectedTensorProduct("64x0e+64x1o", "64x0e+64x1o", "64x0e+64x2o+64x1o", layout=cb.ir_mul, internal_weights=False, shared_weights=True)
    prog = m.f._program(torch.float32)
    assert prog._tri_channels(torch.float32) == 64
    gen = torch.Generator().manual_seed(3)
    B = 300
    x1, x2, g = (torch.randn(B, r.dim, generator=gen).to(DEV) for r in (m.irreps_in1, m.irreps_in2, m.irreps_out))
    w = (torch.randn(1, m.weight_numel, generator=gen) / 64).to(DEV)
    whole = [prog.tri_map(2, w, (x1, x2), "t"), prog.tri_map(0, w, (x2, g), "t"), prog.tri_map(1, w, (x1, g), "t")]
    ref = _sums(prog.d, *(t.cpu().double() for t in (w, x1, x2, g)))
    for a, b in zip(whole, (ref[0], ref[2], ref[3])):
        assert (a.cpu().double() - b).abs().max() <= 1e-5 * b.abs().max()
    parts = [torch.cat([prog.tri_map(2, w, (x1[a:b], x2[a:b]), "t") for a, b in ((0, 128), (128, B))])]
    assert torch.allclose(parts[0], whole[0], rtol=1e-5, atol=1e-6)
    xs = [t.clone().requires_grad_(True) for t in (w, x1, x2)]
    (o,) = m.f([xs[0], xs[1], xs[2]])
    grads = torch.autograd.grad((o * g).sum(), xs, create_graph=True)
    second = torch.autograd.grad(sum(t.pow(2).sum() for t in grads), xs)
    for a, x in zip(second, xs):
        assert a.shape == x.shape and bool(torch.isfinite(a).all()) and float(a.abs().max()) > 0
