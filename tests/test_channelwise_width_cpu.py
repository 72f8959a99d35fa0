"""Which channelwise polynomials the matcher hands to the group kernels (CPU): what it accepts, the library accepts too."""
import ctypes as C

import pytest
import torch

from cuequivariance_b200 import _lib, channelwise as cw, descriptors as D

LS = ["0e", "1o", "2e", "3o", "4e", "5o"]


@pytest.mark.parametrize("l_sh", [0, 1, 2, 3, 4, 5])
@pytest.mark.parametrize("l_in", [0, 1, 2, 3])
@pytest.mark.parametrize("l_out", [0, 1, 2, 3])
def test_matched_plans_pass_the_library_checks(l_in, l_sh, l_out):
    """The kernels read l <= 3; an x2 row may be longer (its l = 4 paths filtered out), 25 or 36 components at a time."""
    e = D.channelwise_tensor_product("+".join(f"8x{ir}" for ir in LS[: l_in + 1]), "+".join(LS[: l_sh + 1]), LS[: l_out + 1])
    plan = cw.match_channelwise(e.polynomial)
    (_, d), = e.polynomial.operations
    assert (plan is not None) == all(p.coefficients.shape[1] <= 7 for p in d.paths)
    if plan is None:
        return
    L = _lib.lib()
    for g in plan.groups:
        for which, fn in (("fwd_tab", L.cueq_b200_cw_forward_opt), ("bwd_tab", L.cueq_b200_cw_backward_opt)):
            w = torch.zeros(4, plan.row_sizes[0])
            tabs = plan.tables_on(torch.device("cpu"))[plan.groups.index(g)]
            x = torch.zeros(4, max(plan.row_sizes[1:]))
            rp = torch.zeros(1, dtype=torch.int32)
            # no receiver: the checks run, nothing is launched
            a, o, keep = cw.ChannelwiseForward(plan)._args(g, tabs, which, dict(senders=None, x1_mul_ir=False), None, rp, 0, False,
                                                        dict(w=w, x1=x, x2=x, **({"out": x} if which == "fwd_tab" else {"gout": x})))
            assert fn(g["id"], C.byref(a), C.byref(o), None) == 0, L.cueq_b200_last_error()
