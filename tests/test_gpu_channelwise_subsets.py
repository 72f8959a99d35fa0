"""GPU parity of the channelwise kernels on polynomials that use only some paths of a kernel group (harmonics or outputs
cut at a lower degree, x2 rows of 4 or 9 components) and in float64, against the CPU oracle.

Tolerances: float32 as in test_gpu_channelwise.py (sums of partly cancelling products, measured in units of the
tensor's magnitude); float64 1e-12 of that magnitude (at most a few thousand terms at 2^-53 each)."""
import pytest
import torch

import cuequivariance_b200 as cb
from cuequivariance_b200 import descriptors as D, profiling
from tests.test_gpu_channelwise import _close, _grads, _oracle, _sh

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
LS = ["0e", "1o", "2e", "3o"]


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("layout", [cb.mul_ir, cb.ir_mul])
@pytest.mark.parametrize("l_in,l_sh,l_out", [(0, 1, 1), (1, 2, 1), (2, 2, 2), (3, 1, 1), (3, 3, 0), (2, 3, 3)])
@pytest.mark.parametrize("mul", [4, 96, 128])   # a fraction of a warp's channels, a partly used block, the block-per-receiver kernels
def test_channelwise_path_subsets_match_oracle(mul, l_in, l_sh, l_out, layout, dtype):
    s1, s2, keep = "+".join(f"{mul}x{ir}" for ir in LS[: l_in + 1]), "+".join(LS[: l_sh + 1]), LS[: l_out + 1]
    e = D.channelwise_tensor_product(s1, s2, keep)
    m = cb.ChannelWiseTensorProduct(s1, s2, keep, layout=layout, shared_weights=False, internal_weights=False)
    gen = torch.Generator().manual_seed(mul + 10 * l_in + 100 * l_sh)
    E, N = 61, 7
    x1 = torch.randn(N, m.irreps_in1.dim, generator=gen, dtype=torch.float64)
    x2 = _sh(torch.randn(E, 3, generator=gen, dtype=torch.float64))[:, : m.irreps_in2.dim].contiguous()
    w = torch.randn(E, m.weight_numel, generator=gen, dtype=torch.float64)
    snd, rcv = torch.randint(0, N, (E,), generator=gen), torch.randint(0, N - 1, (E,), generator=gen)
    cot = torch.randn(N, m.irreps_out.dim, generator=gen, dtype=torch.float64)
    ref_out, ref_g = _grads(_oracle(e, layout, snd, rcv, N), [w, x1, x2], cot)
    d = lambda t: t.to(DEV, dtype) if t.is_floating_point() else t.to(DEV)  # noqa: E731
    profiling.reset()
    out, g = _grads(lambda w_, a, b: m(a, b, w_, indices_1=d(snd), indices_out=d(rcv), size_out=N), [d(w), d(x1), d(x2)], d(cot))
    groups = m.f._program(dtype)._special.plan.groups
    assert profiling.launch_count == 2 * len(groups), "the specialised kernels did not run"
    rtol, atol = (1e-5, 2e-6) if dtype == torch.float32 else (1e-12, 1e-12)
    _close(out, ref_out, rtol, atol, "out")
    for name, a, b in zip(["gw", "gx1", "gx2"], g, ref_g):
        _close(a, b, 10 * rtol, 10 * atol, name)
