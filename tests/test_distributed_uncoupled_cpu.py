"""Backward pass of the sharded product (CPU, launches and collectives replaced by stand-ins): the gradient of an irrep of x1
that couples to nothing is zero, not whatever memory the gradient was allocated in."""
import pytest
import torch
import torch.distributed as dist

from cuequivariance_b200 import channelwise as cw, descriptors as D, distributed


class _Done:
    def wait(self):
        pass


class _Handler:
    """Launches that add one to every column of their block."""

    def __init__(self, plan):
        self.plan = plan

    def launch_forward_group(self, *args):
        args[-1].zero_()

    def launch_backward_group(self, gi, common, csr, mul_ir, w, block, x2, gout, gw, gblock, gx2):
        gblock += 1


@pytest.mark.parametrize("l_in,l_sh,l_out", [(3, 1, 1), (2, 1, 0), (3, 2, 0), (3, 3, 3)])
def test_columns_of_uncoupled_irreps_are_zero(monkeypatch, l_in, l_sh, l_out):
    ls = ["0e", "1o", "2e", "3o"]
    e = D.channelwise_tensor_product("+".join(f"32x{ir}" for ir in ls[: l_in + 1]), "+".join(ls[: l_sh + 1]), ls[: l_out + 1])
    plan = cw.match_channelwise(e.polynomial)
    monkeypatch.setattr(torch, "empty", lambda shape, dtype=None, device=None: torch.full(shape, float("nan"), dtype=dtype))
    monkeypatch.setattr(dist, "get_world_size", lambda group=None: 1)
    monkeypatch.setattr(dist, "all_gather_into_tensor", lambda out, x, **kw: (out.copy_(x), _Done())[1])
    monkeypatch.setattr(dist, "reduce_scatter_tensor", lambda out, x, **kw: (out.copy_(x), _Done())[1])
    n, edges = 4, 6
    x1 = torch.ones(n, plan.row_sizes[1], requires_grad=True)
    x2, w = torch.ones(edges, plan.row_sizes[2]), torch.ones(edges, plan.row_sizes[0])
    snd = rcv = torch.tensor([0, 0, 1, 2, 3, 3], dtype=torch.int32)
    out = distributed._PipelinedShardedChannelwise.apply(_Handler(plan), None, x1, x2, w, snd, rcv)
    (g,) = torch.autograd.grad(out.sum(), x1)
    want = torch.zeros(plan.row_sizes[1])
    for grp in plan.groups:
        want[grp["x1_off"] : grp["x1_off"] + grp["x1_width"]] = 1
    assert torch.equal(g, want.expand(n, -1))
