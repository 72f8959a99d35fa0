"""Second derivatives in which only some of the first gradients carry a cotangent: the same as with explicit zeros for the
others, on the channelwise kernels, the build-time kernels and the generic executor; and a derivative that vanishes."""
import pytest
import torch

import cuequivariance_b200 as cb

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _channelwise(dtype):
    m = cb.ChannelWiseTensorProduct("32x0e+32x1o", "0e+1o+2e", ["0e", "1o"], layout=cb.mul_ir, shared_weights=False, internal_weights=False)
    snd, rcv = torch.randint(0, 7, (50,), device=DEV), torch.randint(0, 7, (50,), device=DEV)
    xs = [torch.randn(50, m.weight_numel), torch.randn(7, m.irreps_in1.dim), torch.randn(50, m.irreps_in2.dim)]
    return lambda w, a, b: m(a, b, w, indices_1=snd, indices_out=rcv, size_out=7), xs


def _generic(dtype):
    m = cb.ChannelWiseTensorProduct("5x0e+5x1o", "0e+1o", ["0e", "1o"], layout=cb.ir_mul, shared_weights=False, internal_weights=False)
    xs = [torch.randn(9, m.weight_numel), torch.randn(9, m.irreps_in1.dim), torch.randn(9, m.irreps_in2.dim)]
    return lambda w, a, b: m(a, b, w), xs


@pytest.mark.parametrize("make", [_channelwise, _generic])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_missing_cotangents_are_zeros(make, dtype):
    torch.manual_seed(5)
    f, xs = make(dtype)
    xs = [x.to(DEV, dtype).requires_grad_(True) for x in xs]
    out = f(*xs)
    cot = torch.randn_like(out).requires_grad_(True)
    first = torch.autograd.grad(out, xs, cot, create_graph=True)
    wrt = [*xs, cot]
    tol = 1e-12 if dtype == torch.float64 else 1e-5
    for mask in range(1, 8):
        tan = [torch.randn_like(g) for g in first]
        some = [k for k in range(3) if mask >> k & 1]
        a = torch.autograd.grad([first[k] for k in some], wrt, [tan[k] for k in some], retain_graph=True, allow_unused=True)
        b = torch.autograd.grad(first, wrt, [t if k in some else torch.zeros_like(t) for k, t in enumerate(tan)], retain_graph=True)
        for x, y in zip(a, b):
            x = torch.zeros_like(y) if x is None else x
            assert torch.allclose(x, y, rtol=tol, atol=tol * float(y.abs().max().clamp(min=1))), mask
    # linear in the weights: no second derivative with respect to them alone
    (z,) = torch.autograd.grad(first[0], xs[0], torch.ones_like(first[0]), allow_unused=True)
    assert z is None or not bool(z.any())
