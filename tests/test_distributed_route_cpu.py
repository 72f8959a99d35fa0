"""Which sharded products take the pipelined path (CPU, tensors replaced by stand-ins): products of whole kernel groups with a
multiple of four channels.  Path subsets keep the all-gather, whose result can be differentiated twice; channel counts that
the float32 kernels refuse are not handed to them."""
from types import SimpleNamespace

import pytest
import torch

import cuequivariance_b200 as cb
from cuequivariance_b200.distributed import ReceiverShardedChannelWise

LS = ["0e", "1o", "2e", "3o"]


@pytest.mark.parametrize("mul,l_in,l_sh,l_out,pipelined", [
    (32, 3, 3, 3, True), (4, 1, 3, 3, True), (30, 3, 3, 3, False), (10, 1, 3, 3, False),
    (32, 2, 2, 2, False), (32, 1, 1, 1, False), (32, 3, 3, 1, False),
])
def test_route(mul, l_in, l_sh, l_out, pipelined):
    tp = cb.ChannelWiseTensorProduct("+".join(f"{mul}x{ir}" for ir in LS[: l_in + 1]), "+".join(LS[: l_sh + 1]), LS[: l_out + 1],
                                     layout=cb.mul_ir, shared_weights=False, internal_weights=False)
    t = SimpleNamespace(is_cuda=True, dtype=torch.float32, shape=(8, 1))
    assert (ReceiverShardedChannelWise(tp)._handler(t, t, t) is not None) == pipelined
