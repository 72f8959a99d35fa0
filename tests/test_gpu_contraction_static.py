"""Symmetric contractions on kernels written out at build time: every registered shape, both layouts (whole warps and
partial ones, which decides whether mul_ir outputs are stored in place), one atom to several blocks of threads."""
import numpy as np
import pytest
import torch

import cuequivariance_b200 as cb
from cuequivariance_b200 import profiling
from oracle import naive

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _abs(d):
    d = d.copy()
    d.paths = [type(p)(p.indices, np.abs(p.coefficients)) for p in d.paths]
    return d


@pytest.mark.parametrize("degree", [2, 3])
@pytest.mark.parametrize("l_in,l_out", [(1, 0), (1, 1), (2, 0), (2, 1), (3, 0), (3, 1)])
@pytest.mark.parametrize("mul,atoms,lin,lout", [(32, 1, "mul_ir", "mul_ir"), (64, 37, "mul_ir", "mul_ir"), (6, 11, "mul_ir", "mul_ir"),
                                                (32, 5, "ir_mul", "mul_ir"), (96, 3, "mul_ir", "ir_mul")])
def test_against_oracle(l_in, l_out, degree, mul, atoms, lin, lout):
    irreps = lambda n: "+".join(f"{mul}x{l}{'eo'[l % 2]}" for l in range(n + 1))  # noqa: E731,E741
    m = cb.SymmetricContraction(irreps(l_in), irreps(l_out), degree, 3, layout_in=getattr(cb, lin), layout_out=getattr(cb, lout),
                                dtype=torch.float32, device=DEV)
    gen = torch.Generator().manual_seed(100 * l_in + 10 * l_out + degree)
    x = torch.randn(atoms, m.irreps_in.dim, generator=gen)
    w = torch.randn(3, *m.weight_shape, generator=gen)
    sp = torch.randint(0, 3, (atoms,), generator=gen)
    cot = torch.randn(atoms, m.irreps_out.dim, generator=gen)
    with torch.no_grad():
        m.weight.copy_(w)
    blocks = [[(mu, ir.dim) for mu, ir in r] for r in (m.irreps_in, m.irreps_out)]

    def grads(magnitudes=False):
        x_, w_, c_ = (t.double().abs() if magnitudes else t.double() for t in (x, w, cot))
        poly = m.etp.polynomial
        if magnitudes:
            poly = cb.Polynomial(poly.inputs, poly.outputs, [(ope, _abs(d)) for ope, d in poly.operations])
        x_, w_ = x_.requires_grad_(True), w_.requires_grad_(True)
        xi = naive.transpose_layout(x_, blocks[0], True) if lin == "mul_ir" else x_
        rows = max(atoms, 2)     # the evaluator takes a single row for a shared operand
        xi = torch.cat([xi, xi])[:rows]
        (o,) = naive.segmented_polynomial(poly, [w_.flatten(1), xi], {0: torch.cat([sp, sp])[:rows]})
        o = o[:atoms]
        o = naive.transpose_layout(o, blocks[1], False) if lout == "mul_ir" else o
        return [o.detach(), *torch.autograd.grad(o, (x_, w_), c_)]

    ref, mag = grads(), grads(True)
    xd = x.to(DEV).requires_grad_(True)
    profiling.reset()
    profiling.enable()
    try:
        out = m(xd, sp.to(DEV))
        got = [out.detach(), *torch.autograd.grad(out, (xd, m.weight), cot.to(DEV))]
        names = set(profiling.summary())
    finally:
        profiling.enable(False)
    assert names and all(n.startswith("u1d_static") for n in names), names
    # a term is a product of at most 5 factors (4 roundings and the coefficient's), a sum has at most 300 terms and,
    # for the weights, one addition per atom; roundings of 2^-24 each against the sum of magnitudes
    for name, a, b, s in zip(("out", "gx", "gw"), got, ref, mag):
        err = (a.cpu().double() - b).abs()
        assert bool((err <= (5 + 300 + (atoms if name == "gw" else 0)) * 2.0 ** -24 * s + 1e-30).all()), (name, err.max().item())
