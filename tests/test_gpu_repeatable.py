"""Results whose sums are in a fixed order: the same call on the same inputs gives the same bits, every time."""
import pytest
import torch

import cuequivariance_b200 as cb

pytestmark = pytest.mark.gpu
DEV = "cuda"
LS = ["0e", "1o", "2e", "3o"]


def _same(call, names, times=20):
    first = [t.clone() for t in call()]
    for _ in range(times):
        for name, a, b in zip(names, call(), first):
            assert torch.equal(a, b), name


@pytest.mark.parametrize("mul,l_in,l_sh", [(128, 3, 3), (64, 3, 3), (32, 2, 2), (128, 3, 2)])
@pytest.mark.parametrize("layout", ["mul_ir", "ir_mul"])
def test_channelwise_output_and_edge_gradients(mul, l_in, l_sh, layout):
    """Output, weight gradient and x2 gradient (one block of channels); the x1 gradient is reduced over edges by atomics."""
    m = cb.ChannelWiseTensorProduct("+".join(f"{mul}x{ir}" for ir in LS[: l_in + 1]), "+".join(LS[: l_sh + 1]), LS, layout=getattr(cb, layout),
                                    shared_weights=False, internal_weights=False)
    torch.manual_seed(0)
    E, N = 4001, 130
    w, x1, x2 = (torch.randn(n, k, device=DEV, requires_grad=True) for n, k in ((E, m.weight_numel), (N, m.irreps_in1.dim), (E, m.irreps_in2.dim)))
    snd, rcv = torch.randint(0, N, (E,), device=DEV), torch.randint(0, N, (E,), device=DEV)
    cot = torch.randn(N, m.irreps_out.dim, device=DEV)

    def step():
        out = m(x1, x2, w, indices_1=snd, indices_out=rcv, size_out=N)
        return [out.detach(), *torch.autograd.grad(out, [w, x2], cot)]

    _same(step, ("out", "gw", "gx2"))


@pytest.mark.parametrize("mul,lmax,batch,dtype", [(32, 2, 200, "float32"), (64, 2, 300, "float32"), (64, 2, 5000, "float32"), (96, 1, 300, "float32"),
                                                  (128, 2, 300, "bfloat16")])
def test_fully_connected_output_and_input_gradients(mul, lmax, batch, dtype):
    s = "+".join(f"{mul}x{ir}" for ir in LS[: lmax + 1])
    m = cb.FullyConnectedTensorProduct(s, s, s, layout=cb.ir_mul, internal_weights=False, shared_weights=True)
    torch.manual_seed(0)
    dt = getattr(torch, dtype)
    x1, x2, cot = (torch.randn(batch, m.irreps_in1.dim, device=DEV).to(dt) for _ in range(3))
    w = torch.randn(1, m.weight_numel, device=DEV).to(dt)
    x1.requires_grad_(True), x2.requires_grad_(True)

    def step():
        out = m(x1, x2, w)
        return [out.detach(), *(torch.autograd.grad(out, [x1, x2], cot) if mul != 96 else ())]   # 96: gradients folded by atomics

    _same(step, ("out", "gx1", "gx2"))


@pytest.mark.parametrize("mul,lmax,rows,classes", [(128, 3, 2000, 1), (128, 3, 20011, 1), (32, 1, 300, 1), (64, 2, 1500, 10), (32, 0, 256, 64)])
def test_linear_with_gradients(mul, lmax, rows, classes):
    s = "+".join(f"{mul}x{ir}" for ir in LS[: lmax + 1])
    m = cb.Linear(s, s, layout=cb.mul_ir, internal_weights=False, shared_weights=True, weight_classes=classes)
    torch.manual_seed(0)
    x, cot = (torch.randn(rows, m.irreps_in.dim, device=DEV) for _ in range(2))
    w = torch.randn(classes, m.weight_numel, device=DEV, requires_grad=True)
    x.requires_grad_(True)
    idx = torch.sort(torch.randint(0, classes, (rows,), device=DEV)).values if classes > 1 else None

    def step():
        out = m(x, w, idx)
        return [out.detach(), *torch.autograd.grad(out, [w, x], cot)]

    _same(step, ("out", "gw", "gx"))


@pytest.mark.parametrize("mul,lmax,batch", [(32, 2, 200), (32, 2, 2048), (64, 2, 300), (64, 1, 2047), (96, 1, 500)])
def test_fully_connected_weight_gradient_of_small_batches(mul, lmax, batch):
    s = "+".join(f"{mul}x{ir}" for ir in LS[: lmax + 1])
    m = cb.FullyConnectedTensorProduct(s, s, s, layout=cb.ir_mul, internal_weights=False, shared_weights=True)
    torch.manual_seed(0)
    x1, x2, cot = (torch.randn(batch, m.irreps_in1.dim, device=DEV) for _ in range(3))
    w = torch.randn(1, m.weight_numel, device=DEV, requires_grad=True)
    out = m(x1, x2, w)
    _same(lambda: torch.autograd.grad(out, [w], cot, retain_graph=True), ("gw",))
