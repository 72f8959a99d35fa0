"""The channelwise product inside a CUDA graph: all groups of the call, which overlap on the device, forward and backward, on
an edge list that is first seen during the capture; a call outside the graph in between; and replays on changed inputs."""
import pytest
import torch

import cuequivariance_b200 as cb
from cuequivariance_b200 import channelwise as cw

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("mul,l_sh", [(128, 3), (96, 2)])
@pytest.mark.parametrize("itype", [torch.int32, torch.int64])
def test_capture_with_a_new_edge_list(mul, l_sh, itype):
    ls = ["0e", "1o", "2e", "3o"]
    m = cb.ChannelWiseTensorProduct("+".join(f"{mul}x{ir}" for ir in ls), "+".join(ls[: l_sh + 1]), ls, layout=cb.mul_ir, shared_weights=False,
                                    internal_weights=False)
    E, N = 500, 40
    torch.manual_seed(mul)
    w, x1, x2 = (torch.randn(n, k, device=DEV, requires_grad=True) for n, k in ((E, m.weight_numel), (N, m.irreps_in1.dim), (E, m.irreps_in2.dim)))
    cot = torch.randn(N, m.irreps_out.dim, device=DEV)
    lists = [[torch.randint(0, N, (E,), device=DEV).to(itype) for _ in range(2)] for _ in range(2)]

    def step(snd, rcv):
        out = m(x1, x2, w, indices_1=snd, indices_out=rcv, size_out=N)
        return [out, *torch.autograd.grad(out, [w, x2, x1], cot)]

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step(*lists[0])                                   # warm-up on another list
    torch.cuda.current_stream().wait_stream(side)
    before = [e[0] for e in cw._CSR.entries]
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        captured = step(*lists[1])
    assert [e[0] for e in cw._CSR.entries] == before
    eager = step(*lists[1])                               # before the first replay
    for _ in range(3):
        g.replay()
    again = step(*lists[1])
    for name, a, b, c in zip(("out", "gw", "gx2", "gx1"), captured, eager, again):
        scale = float(b.abs().max())
        assert bool(torch.isfinite(b).all()) and scale > 0
        if name in ("out", "gw"):                         # sums in a fixed order
            assert torch.equal(a, b) and torch.equal(b, c), name
        else:
            assert float((a - b).abs().max()) <= 1e-5 * scale, name
    with torch.no_grad():
        x1.mul_(2)
        lists[1][1].copy_(torch.randint(0, N, (E,), device=DEV).to(itype))
    g.replay()
    fresh = step(*lists[1])
    assert torch.equal(captured[0], fresh[0]) and torch.equal(captured[1], fresh[1])
