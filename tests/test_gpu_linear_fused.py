"""The equivariant linear layer in one launch per result (csrc/linear_fused.cu) against float64 sums: partial tiles (128 / d
nodes) and K blocks (32 / d nodes), multiplicities below 128, both layouts on either side, weight classes with and without
rows, rows of no class, blocks of rows that no path touches."""
import pytest
import torch

import cuequivariance_b200 as cb
from cuequivariance_b200.operations import linear as linear_mod

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _offsets(irreps):
    o, out = 0, []
    for mul, ir in irreps:
        out.append(o)
        o += mul * ir.dim
    return out


def _blocks(x, irreps, layout):
    """[rows, mul, dim] per irrep of a row-major tensor."""
    out = []
    for o, (mul, ir) in zip(_offsets(irreps), irreps):
        t = x[:, o : o + mul * ir.dim]
        out.append(t.reshape(-1, mul, ir.dim) if layout is cb.mul_ir else t.reshape(-1, ir.dim, mul).transpose(1, 2))
    return out


def _join(blocks, layout):
    return torch.cat([(b if layout is cb.mul_ir else b.transpose(1, 2)).reshape(b.shape[0], -1) for b in blocks], dim=1)


def _reference(plan, m, bounds, w, x, cot, lin, lout):
    """(out, gw, gx) by plain sums in the dtype of the operands."""
    offs_in = {o: k for k, o in enumerate(_offsets(m.irreps_in))}
    offs_out = {o: k for k, o in enumerate(_offsets(m.irreps_out))}
    xb, gb = _blocks(x, m.irreps_in, lin), _blocks(cot, m.irreps_out, lout)
    ob, gxb, gw = [torch.zeros_like(t) for t in gb], [torch.zeros_like(t) for t in xb], torch.zeros_like(w)
    for wo, u, v, xo, oo, d, c in plan["paths"]:
        i, o = offs_in[xo], offs_out[oo]
        for k in range(len(bounds) - 1):
            s = slice(bounds[k], bounds[k + 1])
            W = w[k, wo : wo + u * v].reshape(u, v) * abs(c)
            ob[o][s] = torch.einsum("zui,uv->zvi", xb[i][s], W)
            gxb[i][s] = torch.einsum("zvi,uv->zui", gb[o][s], W)
            gw[k, wo : wo + u * v] = (torch.einsum("zui,zvi->uv", xb[i][s], gb[o][s]) * abs(c)).reshape(-1)
        assert c > 0
    return _join(ob, lout), gw, _join(gxb, lin)


@pytest.mark.parametrize("s_in,s_out,rows,classes,lin,lout", [
    ("128x0e+128x1o+128x2e+128x3o", "128x0e+128x1o+128x2e+128x3o", 257, 1, "mul_ir", "mul_ir"),
    ("128x0e+128x1o+128x2e+128x3o", "128x0e+128x1o+128x2e+128x3o", 20011, 1, "mul_ir", "mul_ir"),
    ("32x0e+96x1o+64x2e+32x3o", "96x0e+32x1o+64x2e+128x3o", 421, 1, "ir_mul", "mul_ir"),
    ("96x0e+64x1o", "32x0e+96x1o", 1000, 1, "mul_ir", "ir_mul"),
    ("64x0e+64x1o+64x2e+64x3o", "64x0e+64x1o+64x2e+64x3o", 911, 10, "ir_mul", "ir_mul"),
    ("128x1o+64x3o", "64x0e+32x1o+32x3o", 3001, 3, "mul_ir", "mul_ir"),
    ("32x0e", "32x0e", 256, 64, "mul_ir", "mul_ir"),
])
def test_against_float64_sums(s_in, s_out, rows, classes, lin, lout):
    lin, lout = getattr(cb, lin), getattr(cb, lout)
    m = cb.Linear(s_in, s_out, layout_in=lin, layout_out=lout, internal_weights=False, shared_weights=True, weight_classes=classes)
    assert m._fused_plan is not None
    gen = torch.Generator().manual_seed(rows)
    x, w = torch.randn(rows, m.irreps_in.dim, generator=gen), torch.randn(classes, m.weight_numel, generator=gen)
    cot = torch.randn(rows, m.irreps_out.dim, generator=gen)
    idx, bounds = None, (0, rows)
    if classes > 1:   # class 1 owns no row
        idx = torch.sort(torch.randint(0, classes, (rows,), generator=gen)).values
        idx[idx == 1] = 0
        bounds = torch.searchsorted(idx, torch.arange(classes + 1)).tolist()
    xd, wd = x.to(DEV).requires_grad_(True), w.to(DEV).requires_grad_(True)
    out = m(xd, wd, None if idx is None else idx.to(DEV))
    assert "FusedLinear" in type(out.grad_fn).__name__
    gw, gx = torch.autograd.grad(out, (wd, xd), cot.to(DEV))
    ref = _reference(m._fused_plan, m, bounds, w.double(), x.double(), cot.double(), lin, lout)
    mag = _reference(m._fused_plan, m, bounds, w.double().abs(), x.double().abs(), cot.double().abs(), lin, lout)
    # products: 2^-21 (dropped lo*lo, rounding of lo); float32 sums that need not round to nearest: 2^-23 of the magnitude
    # per addition of a chain - 8 large and 16 small ones per accumulator and the sum of two, and for the weight gradient
    # 4 * 128 / 3 per accumulator, four accumulators and one addition per thread block
    for name, a, b, s, chain in (("out", out, ref[0], mag[0], 16), ("gw", gw, ref[1], mag[1], 200 + rows // 64), ("gx", gx, ref[2], mag[2], 16)):
        err = (a.detach().cpu().double() - b).abs()
        assert bool((err <= (2.0 ** -21 + chain * 2.0 ** -23) * s + 1e-30).all()), (name, err.max().item())


def test_route_boundaries():
    """What the fused kernels do not take keeps its route: two paths on one block of rows, multiplicities above 128 or not a
    multiple of 32, l = 4, few rows, float64; rows that do not start on a 16-byte boundary are copied."""
    fused = lambda a, b, **kw: cb.Linear(a, b, layout=cb.mul_ir, internal_weights=False, shared_weights=True, **kw)._fused_plan  # noqa: E731
    assert fused("32x0e+32x0e", "32x0e") is None and fused("160x0e", "32x0e") is None and fused("48x0e", "32x0e") is None
    assert fused("32x4e", "32x4e") is None
    m = cb.Linear("32x0e+32x1o", "32x0e+32x1o", layout=cb.mul_ir, internal_weights=False, shared_weights=True)
    x, w = torch.randn(300, 128, device=DEV), torch.randn(1, m.weight_numel, device=DEV)
    a = m(x, w)
    old, linear_mod.DENSE_ROUTE = linear_mod.DENSE_ROUTE, False
    try:
        b = m(x, w)
    finally:
        linear_mod.DENSE_ROUTE = old
    assert torch.allclose(a, b, rtol=1e-5, atol=1e-5)
    assert torch.allclose(m(x[:40], w), b[:40], rtol=1e-5, atol=1e-5)
    assert torch.allclose(m(x.double(), w.double()).float(), b, rtol=1e-5, atol=1e-5)
    y = torch.randn(300 * 128 + 1, device=DEV)[1:].view(300, 128)
    assert torch.equal(m(y, w), m(y.clone(), w))
