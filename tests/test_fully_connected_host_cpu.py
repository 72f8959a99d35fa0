"""Host side of the fully connected product (CPU): the bf16 weights belong to the values they are made from, a gradient that
nobody asks for is not computed, and a library without the tri-linear kernels falls back to the memory route."""
import pytest
import torch

import cuequivariance_b200 as cb
from cuequivariance_b200 import _lib, fused_tp


def _product(mul):
    s = f"{mul}x0e+{mul}x1o"
    return cb.FullyConnectedTensorProduct(s, s, s, layout=cb.ir_mul, internal_weights=False, shared_weights=True).f._program(torch.float32)


def test_bf16_weights_follow_the_values():
    """Changed through .data, or another tensor at the same address: neither moves the version counter."""
    prog = _product(64)
    n = prog.d.operands[0].size
    w = torch.randn(1, n)
    for _ in range(3):
        for transposed in (False, True):
            t = w.view(-1, 64, 64, 64)
            want = (t.transpose(1, 2) if transposed else t).reshape(-1, 64).to(torch.bfloat16)
            assert torch.equal(prog._weights_bf16(w, transposed), want)
        version = w._version
        w.data.mul_(-0.5)
        assert w._version == version
