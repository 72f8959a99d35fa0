"""Backward kernels for channel counts that are no multiple of 128: a thread block per receiver with two channels per thread
(with bulk reductions where 64 divides the channels), or a warp per receiver where receivers have few edges."""
import pytest
import torch

import cuequivariance_b200 as cb
from cuequivariance_b200 import descriptors as D
from oracle import naive

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("layout", ["mul_ir", "ir_mul"])
@pytest.mark.parametrize("mul", [4, 32, 64, 96, 192])
@pytest.mark.parametrize("edges,nodes,l_sh", [(150, 7, 3), (60, 40, 3), (90, 11, 2), (1, 3, 3)])
def test_gradients_against_oracle(mul, edges, nodes, l_sh, layout):
    irreps = "+".join(f"{mul}x{ir}" for ir in ("0e", "1o", "2e", "3o"))
    sh = "+".join(("0e", "1o", "2e", "3o")[: l_sh + 1])
    filt = ["0e", "1o", "2e"]
    m = cb.ChannelWiseTensorProduct(irreps, sh, filt, layout=getattr(cb, layout), shared_weights=False, internal_weights=False)
    e = D.channelwise_tensor_product(m.irreps_in1, m.irreps_in2, filt)
    gen = torch.Generator().manual_seed(mul + edges)
    xs = [torch.randn(edges, m.weight_numel, generator=gen), torch.randn(nodes, m.irreps_in1.dim, generator=gen), torch.randn(edges, m.irreps_in2.dim, generator=gen)]
    snd = torch.randint(0, nodes, (edges,), generator=gen)
    rcv = torch.randint(0, max(nodes - 1, 1), (edges,), generator=gen)
    cot = torch.randn(nodes, m.irreps_out.dim, generator=gen)
    b1, bo = ([(mu, ir.dim) for mu, ir in r] for r in (m.irreps_in1, m.irreps_out))

    def reference(w, a, b):
        a = naive.transpose_layout(a, b1, True) if layout == "mul_ir" else a
        two = lambda t: torch.cat([t, t]) if edges == 1 else t  # noqa: E731  (the evaluator takes one row for a shared operand)
        (o,) = naive.segmented_polynomial(e.polynomial, [two(w), a, two(b)], {1: two(snd)}, {0: nodes}, {0: two(rcv)})
        o = o / 2 if edges == 1 else o
        return naive.transpose_layout(o, bo, False) if layout == "mul_ir" else o

    def grads(fn, dev, dtype):
        ys = [x.to(dev, dtype).requires_grad_(True) for x in xs]
        out = fn(*ys)
        return [out.detach(), *torch.autograd.grad(out, ys, cot.to(dev, dtype))]

    ref = grads(reference, "cpu", torch.float64)
    got = grads(lambda w, a, b: m(a, b, w, indices_1=snd.to(DEV), indices_out=rcv.to(DEV), size_out=nodes), DEV, torch.float32)
    for name, a, b in zip(("out", "gw", "gx1", "gx2"), got, ref):
        f = 1 if name == "out" else 10       # the scaling of the other float32 comparisons: outputs, first derivatives
        err = (a.cpu().double() - b).abs()
        assert bool((err <= f * 1e-5 * b.abs() + f * 2e-6 * max(1.0, float(b.abs().max()))).all()), (name, err.max().item())
