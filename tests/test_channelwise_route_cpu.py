"""Where the generic kernel is the faster one for a channelwise product (CPU: the rule on shapes, on both sides of its lines)."""
from types import SimpleNamespace

import pytest
import torch

from cuequivariance_b200 import channelwise as cw, descriptors as D

LS = ["0e", "1o", "2e", "3o"]


@pytest.mark.parametrize("dtype,mul,l_in,l_sh,l_out,edges,degree,forward,backward", [
    ("float64", 4, 3, 1, 1, 200000, 8, True, True),        # a sparse subset, few channels
    ("float64", 4, 3, 1, 1, 2000, 8, False, False),        # ... in a call that the host bounds
    ("float64", 16, 3, 1, 1, 200000, 1, True, True),       # receivers of one edge
    ("float64", 16, 3, 1, 1, 200000, 40, False, False),
    ("float64", 64, 3, 1, 1, 200000, 1, False, False),     # enough channels
    ("float64", 4, 3, 3, 3, 200000, 8, False, False),      # whole groups have work enough
    ("float64", 2, 3, 3, 3, 200000, 1, False, True),
    ("float32", 4, 3, 1, 1, 200000, 8, True, True),
    ("float32", 8, 3, 1, 1, 200000, 8, False, False),
    ("float32", 4, 2, 2, 2, 200000, 8, False, False),      # most of the groups' paths
    ("float32", 4, 3, 3, 3, 200000, 1, False, False),      # whole groups
    ("float32", 4, 3, 1, 1, 2000, 8, False, False),
])
def test_rule(dtype, mul, l_in, l_sh, l_out, edges, degree, forward, backward):
    e = D.channelwise_tensor_product("+".join(f"{mul}x{ir}" for ir in LS[: l_in + 1]), "+".join(LS[: l_sh + 1]), LS[: l_out + 1])
    plan = cw.match_channelwise(e.polynomial)
    prog = SimpleNamespace(math_dtype=getattr(torch, dtype))
    base = cw.ChannelwiseForward(plan)
    assert base._generic_is_faster(prog, edges, edges // degree, False) == forward
    assert base._generic_is_faster(prog, edges, edges // degree, True) == backward
    assert not base._generic_is_faster(prog, 0, 0, True) and not base._generic_is_faster(prog, 0, 5, False)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,mul", [(torch.float64, 2), (torch.float64, 6), (torch.float32, 4)])
@pytest.mark.parametrize("layout", ["mul_ir", "ir_mul"])
def test_both_routes_agree(monkeypatch, dtype, mul, layout):
    """The call that changes its route gives the same output and gradients on either, to the rounding of its sums."""
    import cuequivariance_b200 as cb

    m = cb.ChannelWiseTensorProduct("+".join(f"{mul}x{ir}" for ir in LS), "0e+1o", LS[:2], layout=getattr(cb, layout), shared_weights=False,
                                    internal_weights=False)
    torch.manual_seed(0)
    E, N = 3000, 400
    w, x1, x2 = (torch.randn(n, k, device="cuda", dtype=dtype, requires_grad=True) for n, k in ((E, m.weight_numel), (N, m.irreps_in1.dim), (E, m.irreps_in2.dim)))
    snd, rcv = torch.randint(0, N, (E,), device="cuda"), torch.randint(0, N, (E,), device="cuda")
    cot = torch.randn(N, m.irreps_out.dim, device="cuda", dtype=dtype)
    res = []
    for generic in (False, True):
        monkeypatch.setattr(cw._ChannelwiseBase, "_generic_is_faster", lambda self, *a, g=generic: g)
        out = m(x1, x2, w, indices_1=snd, indices_out=rcv, size_out=N)
        first = torch.autograd.grad(out, [w, x1, x2], cot, create_graph=True)
        second = torch.autograd.grad(sum(t.pow(2).sum() for t in first), [w, x1, x2])
        res.append([out, *first, *second])
    eps = torch.finfo(dtype).eps
    for a, b in zip(*res):
        # some hundred partly cancelling products per value, three times as many in a second derivative
        assert torch.allclose(a, b, rtol=200 * eps, atol=200 * eps * float(b.detach().abs().max()))
