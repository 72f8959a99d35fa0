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
