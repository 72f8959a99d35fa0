"""Host side of the fully connected product (CPU): the bf16 weights belong to the values they are made from, a gradient that
nobody asks for is not computed, and a library without the tri-linear kernels falls back to the memory route."""
import pytest
import torch

import cuequivariance_b200 as cb
from cuequivariance_b200 import _lib, fused_tp


def _product(mul):
    s = f"{mul}x0e+{mul}x1o"
    return cb.FullyConnectedTensorProduct(s, s, s, layout=cb.ir_mul, internal_weights=False, shared_weights=True).f._program(torch.float32)


def test_bf16_weights_follow_the_values():
    """Changed through .data, or another tensor at the same address: neither moves the version counter."""
    prog = _product(64)
    n = prog.d.operands[0].size
    w = torch.randn(1, n)
    for _ in range(3):
        for transposed in (False, True):
            t = w.view(-1, 64, 64, 64)
            want = (t.transpose(1, 2) if transposed else t).reshape(-1, 64).to(torch.bfloat16)
            assert torch.equal(prog._weights_bf16(w, transposed).reshape(-1, 64), want)
        version = w._version
        w.data.mul_(-0.5)
        assert w._version == version
    b = w.to(torch.bfloat16)
    assert prog._weights_bf16(b, False) is b
    assert torch.equal(prog._weights_bf16(b, True).reshape(-1, 64), b.view(-1, 64, 64, 64).transpose(1, 2).reshape(-1, 64))


class _Owner:
    """out[z] = w x1[z] x2[z], elementwise, with the interface of the float32 route."""

    def __init__(self):
        self.asked = []

    def map_out(self, w, x1, x2):
        return w * x1 * x2

    def map_w(self, x1, x2, g):
        return (x1 * x2 * g).sum(0, keepdim=True)

    def map_x(self, w, x1, x2, g, need=(True, True)):
        self.asked.append(need)
        return (w * x2 * g if need[0] else None), (w * x1 * g if need[1] else None)


@pytest.mark.parametrize("need", [(True, False), (False, True), (True, True)])
def test_only_the_gradients_asked_for(need):
    torch.manual_seed(0)
    owner = _Owner()
    w, x1, x2, g = (torch.randn(n, 4, dtype=torch.float64) for n in (1, 5, 5, 5))
    xs = [t.requires_grad_(n) for t, n in zip((x1, x2), need)]
    out = fused_tp._DenseOut.apply(owner, w, *xs)
    wanted = [t for t in xs if t.requires_grad]
    grads = torch.autograd.grad(out, wanted, g)
    assert owner.asked == [need]
    ref = torch.autograd.grad(w * xs[0] * xs[1], wanted, g)
    assert all(torch.allclose(a, b, rtol=1e-14) for a, b in zip(grads, ref))


def test_derivatives_to_third_order():
    torch.manual_seed(0)
    owner = _Owner()
    xs = [torch.randn(n, 3, dtype=torch.float64, requires_grad=True) for n in (1, 4, 4)]
    f = lambda *a: fused_tp._DenseOut.apply(owner, *a)  # noqa: E731
    assert torch.autograd.gradcheck(f, xs) and torch.autograd.gradgradcheck(f, xs)

    def third(fn):
        a = torch.autograd.grad(fn(*xs).pow(2).sum(), xs, create_graph=True)
        b = torch.autograd.grad(sum(t.pow(2).sum() for t in a), xs, create_graph=True)
        return torch.autograd.grad(sum(t.pow(2).sum() for t in b), xs)

    for a, b in zip(third(f), third(lambda w, a, b: w * a * b)):
        assert torch.allclose(a, b, rtol=1e-10)


def test_a_build_without_usable_kernels_keeps_the_memory_route(monkeypatch):
    """The tri-linear kernels divide a fixed number of registers; a library whose compiler gave them another number says so."""
    prog, bf16 = _product(64), _product(128)
    assert prog._tri_channels(torch.float32) == 64 and bf16._tri_channels(torch.bfloat16) == 128
    asked = []

    class _Lib:
        def cueq_b200_fctp_tri_ready(self, dtype, channels):
            asked.append((dtype, channels))
            return 0

    monkeypatch.setattr(_lib, "lib", _Lib)
    for p, dt in ((_product_again(prog), torch.float32), (_product_again(bf16), torch.bfloat16)):
        assert p._tri_channels(dt) == 0 and p._tri_channels(dt) == 0
    assert asked == [(_lib.F32, 64), (_lib.BF16, 128)]
    assert _product_again(prog)._gw_channels() == 64


def _product_again(prog):
    """The same product with nothing decided yet."""
    new = object.__new__(type(prog))
    new.__dict__.update(prog.__dict__, _tri_mul=None, _tri_ready={})
    return new
