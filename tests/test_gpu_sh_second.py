"""Second and third derivatives of the spherical harmonics: the fused second derivative against the polynomial executor, with
and without normalisation, for single degrees and all of them, one vector to several thread blocks."""
import pytest
import torch

import cuequivariance_b200 as cb
from cuequivariance_b200 import profiling

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ls", [[0], [1], [3], [0, 1, 2, 3], [2, 4], [0, 1, 2, 3, 4]])
@pytest.mark.parametrize("normalize", [True, False])
@pytest.mark.parametrize("rows,dtype", [(1, torch.float64), (257, torch.float64), (1000, torch.float32)])
def test_against_polynomials(ls, normalize, rows, dtype):
    m = cb.SphericalHarmonics(ls, normalize=normalize)
    gen = torch.Generator().manual_seed(rows)
    vec, g = torch.randn(rows, 3, generator=gen), torch.randn(rows, m.width, generator=gen)
    h, k = torch.randn(rows, 3, generator=gen), torch.randn(rows, 3, generator=gen)

    def derivatives(route, dt):
        v, c, t = (x.to("cuda", dt).requires_grad_(True) for x in (vec, g, h))
        (gv,) = torch.autograd.grad(route(v), v, c, create_graph=True)
        if not gv.requires_grad:                  # degree 0 alone: no derivative
            return [gv]
        second = torch.autograd.grad(gv, (v, c), t, retain_graph=True, allow_unused=True)
        again = torch.autograd.grad(gv, (v, c), t, create_graph=True, allow_unused=True)
        res = [gv.detach(), *second]
        if again[0] is not None and again[0].requires_grad:
            res += list(torch.autograd.grad(again[0], (v, c, t), k.to("cuda", dt), allow_unused=True))
        return res

    profiling.reset()
    profiling.enable()
    try:
        got = derivatives(m, dtype)
        names = set(profiling.summary())
    finally:
        profiling.enable(False)
    assert "sh_fused_backward" in names and ("sh_fused_second" in names or ls == [0])
    ref = derivatives(m._polynomial_route, torch.float64)
    tol = 1e-12 if dtype == torch.float64 else 2e-5     # about 30 terms of degree 4, division by |v|^3 with |v| down to 0.1
    for n, a in enumerate(got):
        b = ref[n] if n < len(ref) else None
        if a is None or b is None:
            assert (a is None or not bool(a.any())) and (b is None or not bool(b.any())), n
            continue
        scale = b.abs().amax(dim=1, keepdim=True).clamp(min=1.0)
        assert bool(((a.double() - b).abs() <= tol * scale * (1 if normalize is False else 10)).all()), (n, (a.double() - b).abs().max().item())
