"""x2 rows longer than the 16 components that the group kernels read: harmonics up to l = 4 and 5 whose high paths are filtered
out, rows of 25 (no 16-byte pitch) and 36 components, full groups and subsets, against the CPU oracle."""
import pytest
import torch

import cuequivariance_b200 as cb
from cuequivariance_b200 import descriptors as D, profiling
from tests.test_gpu_channelwise import _close, _grads, _oracle

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
LS = ["0e", "1o", "2e", "3o", "4e", "5o"]


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("mul", [32, 128])
@pytest.mark.parametrize("l_in,l_sh,l_out", [(0, 4, 0), (0, 4, 3), (0, 5, 3), (1, 4, 2), (2, 5, 1), (3, 4, 0)])
def test_only_the_first_components_are_read(l_in, l_sh, l_out, mul, dtype):
    s1, s2, keep = "+".join(f"{mul}x{ir}" for ir in LS[: l_in + 1]), "+".join(LS[: l_sh + 1]), LS[: l_out + 1]
    e = D.channelwise_tensor_product(s1, s2, keep)
    m = cb.ChannelWiseTensorProduct(s1, s2, keep, layout=cb.mul_ir, shared_weights=False, internal_weights=False)
    gen = torch.Generator().manual_seed(mul + l_sh)
    E, N = 61, 7
    x1, x2, w = (torch.randn(n, k, generator=gen, dtype=torch.float64) for n, k in ((N, m.irreps_in1.dim), (E, m.irreps_in2.dim), (E, m.weight_numel)))
    snd, rcv = torch.randint(0, N, (E,), generator=gen), torch.randint(0, N - 1, (E,), generator=gen)
    cot = torch.randn(N, m.irreps_out.dim, generator=gen, dtype=torch.float64)
    ref_out, ref_g = _grads(_oracle(e, cb.mul_ir, snd, rcv, N), [w, x1, x2], cot)
    d = lambda t: t.to(DEV, dtype) if t.is_floating_point() else t.to(DEV)  # noqa: E731
    profiling.reset()
    out, g = _grads(lambda w_, a, b: m(a, b, w_, indices_1=d(snd), indices_out=d(rcv), size_out=N), [d(w), d(x1), d(x2)], d(cot))
    assert profiling.launch_count == 2 * len(m.f._program(dtype)._special.plan.groups), "the specialised kernels did not run"
    rtol, atol = (1e-5, 2e-6) if dtype == torch.float32 else (1e-12, 1e-12)   # as in test_gpu_channelwise_subsets.py
    _close(out, ref_out, rtol, atol, "out")
    for name, a, b in zip(["gw", "gx1", "gx2"], g, ref_g):
        _close(a, b, 10 * rtol, 10 * atol, name)
