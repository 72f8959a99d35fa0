"""A polynomial whose outputs get no cotangent at all, because the function behind it returned None: its inputs take part in
the graph, so their gradients are zeros (CPU, with a program that only allocates)."""
import torch

from cuequivariance_b200.executor import PolynomialFunction


class _Program:
    def run(self, cfg, xs):
        return [xs[0] * 2, xs[1] * 3]


class _Cut(torch.autograd.Function):
    @staticmethod
    def forward(ctx, a, b):
        return a.sum() + b.sum()

    @staticmethod
    def backward(ctx, g):
        return None, None


def test_no_cotangent_at_all_gives_zeros():
    a, b, c = torch.ones(2, 3, requires_grad=True), torch.ones(4, requires_grad=True), torch.ones(5)
    out = _Cut.apply(*PolynomialFunction.apply(_Program(), None, a, b, c))
    ga, gb = torch.autograd.grad(out, (a, b), retain_graph=True)
    assert torch.equal(ga, torch.zeros(2, 3)) and torch.equal(gb, torch.zeros(4))
    out.backward()
    assert torch.equal(a.grad, torch.zeros(2, 3)) and c.grad is None
