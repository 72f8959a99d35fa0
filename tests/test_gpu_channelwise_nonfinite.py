"""An infinite or undefined component of x2 reaches the paths that use it and no others, on the kernels for path subsets and
float64 (the table-driven kernel confines it as well)."""
import pytest
import torch

import cuequivariance_b200 as cb

pytestmark = pytest.mark.gpu
DEV = "cuda"
LS = ["0e", "1o", "2e", "3o"]


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("component", [0, 2])
@pytest.mark.parametrize("mul,l_in,l_sh,l_out,dtype", [(32, 2, 2, 2, torch.float32), (128, 3, 3, 2, torch.float32), (32, 3, 3, 3, torch.float64)])
def test_confined_to_its_paths(mul, l_in, l_sh, l_out, dtype, component, bad):
    m = cb.ChannelWiseTensorProduct("+".join(f"{mul}x{ir}" for ir in LS[: l_in + 1]), "+".join(LS[: l_sh + 1]), LS[: l_out + 1], layout=cb.ir_mul,
                                    shared_weights=False, internal_weights=False)
    prog = m.f._program(dtype)
    assert prog._special is not None
    torch.manual_seed(1)
    E, N = 12, 5
    x1, x2, w = (torch.randn(n, k, device=DEV, dtype=dtype) for n, k in ((N, m.irreps_in1.dim), (E, m.irreps_in2.dim), (E, m.weight_numel)))
    snd, rcv = torch.randint(0, N, (E,), device=DEV), torch.arange(E, device=DEV) % N
    cot = torch.randn(N, m.irreps_out.dim, device=DEV, dtype=dtype)

    def step(b):
        xs = [w.clone().requires_grad_(True), b.clone().requires_grad_(True)]
        out = m(x1, xs[1], xs[0], indices_1=snd, indices_out=rcv, size_out=N)
        return [out.detach(), *torch.autograd.grad(out, xs, cot)]

    spoiled = x2.clone()
    spoiled[3, component] = bad                               # edge 3 goes to receiver 3
    (out, gw, gx2), (ref_out, ref_gw, ref_gx2) = step(spoiled), step(x2)
    _, d = prog.original.operations[0]
    l2 = 0 if component == 0 else 1
    off_w, off_o = d.operands[0].offsets(), d.operands[3].offsets()
    for p in d.paths:
        sw, _, s2, so = p.indices
        n = d.operands[3].segments[so][0] * mul
        o, ro = out[:, off_o[so] : off_o[so] + n], ref_out[:, off_o[so] : off_o[so] + n]
        g, rg = gw[:, off_w[sw] : off_w[sw] + mul], ref_gw[:, off_w[sw] : off_w[sw] + mul]
        if s2 == l2:
            assert not bool(torch.isfinite(o[3]).all()) and not bool(torch.isfinite(g[3]).all())
            keep = torch.arange(N, device=DEV) != 3
            assert torch.equal(o[keep], ro[keep])
        else:
            assert torch.equal(o, ro) and torch.equal(g, rg)
    assert bool(torch.isfinite(gx2).all()) and torch.allclose(gx2, ref_gx2, rtol=1e-5, atol=1e-5 * float(ref_gx2.abs().max()))
