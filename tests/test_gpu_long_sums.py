"""Long inputs of the tensor-core kernels: batches that the fully connected product cuts into chunks (the limits lowered for
the test), a weight gradient of the linear layer with more K blocks than its usual grid covers, and second derivatives of
the fully connected product by value."""
import pytest
import torch

import cuequivariance_b200 as cb
from cuequivariance_b200 import fused_tp
from tests.test_gpu_fctp_tri import _sums
from tests.test_gpu_linear_fused import _reference

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("mul,lmax,batch", [(32, 2, 700), (64, 1, 513)])
def test_chunks_of_a_batch(monkeypatch, mul, lmax, batch):
    s = "+".join(f"{mul}x{l}{'eo'[l % 2]}" for l in range(lmax + 1))  # noqa: E741
    m = cb.FullyConnectedTensorProduct(s, s, s, layout=cb.ir_mul, internal_weights=False, shared_weights=True)
    prog = m.f._program(torch.float32)
    gen = torch.Generator().manual_seed(batch)
    cpu = [torch.randn(1, m.weight_numel, generator=gen) / mul, *(torch.randn(batch, m.irreps_in1.dim, generator=gen) for _ in range(3))]
    w, x1, x2, g = (t.to(DEV) for t in cpu)
    monkeypatch.setattr(fused_tp, "TRI_CHUNK", 256 * x1.shape[1])           # 256 samples at a time
    monkeypatch.setattr(fused_tp, "GW_CHUNK", 256 * 3 * x1.shape[1])
    got = prog.map_out(w, x1, x2), prog.map_w(x1, x2, g), *prog.map_x(w, x1, x2, g)
    ref, mag = (_sums(prog.d, *(f(t.double()) for t in cpu)) for f in (lambda t: t, torch.abs))
    # the bound of test_gpu_fctp_tri.py
    terms = 2.0 ** -21 + 36 * 2.0 ** -23 + mul * 5 * 6 * 2.0 ** -24
    for name, a, b, t in zip(("out", "gw", "gx1", "gx2"), got, ref, mag):
        bound = (terms + (batch * 2.0 ** -23 if name == "gw" else 0)) * t + 1e-30
        assert bool(((a.cpu().double() - b).abs() <= bound).all()), name
        assert float((a.cpu().double() - b).norm() / b.norm()) <= 2.0 ** -19, name


@pytest.mark.parametrize("rows,classes", [(60011, 1), (60011, 3)])
def test_linear_weight_gradient_beyond_the_usual_grid(rows, classes):
    """4 and 6 nodes per K block: 25,005 of them, 148 x 128 are what one wave of thread blocks takes."""
    s = "32x3o+64x2e"
    m = cb.Linear(s, s, layout=cb.mul_ir, internal_weights=False, shared_weights=True, weight_classes=classes)
    gen = torch.Generator().manual_seed(rows)
    x, cot, w = torch.randn(rows, m.irreps_in.dim, generator=gen), torch.randn(rows, m.irreps_out.dim, generator=gen), torch.randn(classes, m.weight_numel, generator=gen)
    idx, bounds = None, (0, rows)
    if classes > 1:
        idx = torch.sort(torch.randint(0, classes, (rows,), generator=gen)).values
        bounds = torch.searchsorted(idx, torch.arange(classes + 1)).tolist()
    wd = w.to(DEV).requires_grad_(True)
    out = m(x.to(DEV), wd, None if idx is None else idx.to(DEV))
    (gw,) = torch.autograd.grad(out, [wd], cot.to(DEV))
    ref, mag = (_reference(m._fused_plan, m, bounds, f(w.double()), f(x.double()), f(cot.double()), cb.mul_ir, cb.mul_ir)[1] for f in (lambda t: t, torch.abs))
    # the bound of test_gpu_linear_fused.py: 4 * 128 / 3 additions per accumulator, four accumulators, one per thread block;
    # the tensor core cuts up to 2^-23 of the sum with each addition, 2^-24 on average
    err = (gw.cpu().double() - ref).abs()
    assert bool((err <= (2.0 ** -21 + (200 + rows // 64) * 2.0 ** -23) * mag).all())
    assert float(err.norm() / ref.norm()) <= 4 * 128 / 3 * 2.0 ** -24


@pytest.mark.parametrize("mul,lmax,batch", [(32, 2, 100), (64, 1, 130)])
def test_second_derivatives_by_value(mul, lmax, batch):
    """Gradients of a sum of squares of all first gradients, against the same in float64 by plain sums: three contractions one
    after the other, each within 2^-19 of its result, and the factor of the square."""
    s = "+".join(f"{mul}x{l}{'eo'[l % 2]}" for l in range(lmax + 1))  # noqa: E741
    m = cb.FullyConnectedTensorProduct(s, s, s, layout=cb.ir_mul, internal_weights=False, shared_weights=True)
    prog = m.f._program(torch.float32)
    assert prog._tri_channels(torch.float32) == mul
    d, off = prog.d, [op.offsets() for op in prog.d.operands]
    gen = torch.Generator().manual_seed(batch)
    xs = [torch.randn(1, m.weight_numel, generator=gen) / mul, *(torch.randn(batch, m.irreps_in1.dim, generator=gen) for _ in range(2))]
    g = torch.randn(batch, m.irreps_out.dim, generator=gen)

    def plain(w, x1, x2):
        parts = [0.0] * d.operands[3].num_segments
        for p in d.paths:
            sw, s1, s2, so = p.indices
            c = torch.as_tensor(p.coefficients, dtype=w.dtype)
            U, V, W = d.operands[0].segments[sw]
            a = x1[:, off[1][s1] : off[1][s1] + c.shape[0] * U].view(-1, c.shape[0], U)
            b = x2[:, off[2][s2] : off[2][s2] + c.shape[1] * V].view(-1, c.shape[1], V)
            wp = w[0, off[0][sw] : off[0][sw] + U * V * W].view(U, V, W)
            parts[so] = parts[so] + torch.einsum("zkuv,uvw->zkw", torch.einsum("ijk,ziu,zjv->zkuv", c, a, b), wp).reshape(a.shape[0], -1)
        return torch.cat(parts, 1)

    def second(fn, xs, g):
        xs = [t.clone().requires_grad_(True) for t in xs]
        first = torch.autograd.grad((fn(*xs) * g).sum(), xs, create_graph=True)
        return torch.autograd.grad(sum(t.pow(2).sum() for t in first), xs)

    got = second(lambda w, a, b: m.f([w, a, b])[0], [t.to(DEV) for t in xs], g.to(DEV))
    ref = second(plain, [t.double() for t in xs], g.double())
    for name, a, b in zip(("w", "x1", "x2"), got, ref):
        assert float((a.cpu().double() - b).norm() / b.norm()) <= 6 * 2.0 ** -19, name
