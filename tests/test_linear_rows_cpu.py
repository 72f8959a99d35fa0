"""Which linear layers take the one-launch kernels (CPU): the library accepts the argument block of every plan; rows that an
irrep without a path leaves at an odd pitch or offset keep the route they had."""
import ctypes as C

import pytest
import torch

import cuequivariance_b200 as cb
from cuequivariance_b200 import _lib


@pytest.mark.parametrize("s_in,s_out,fused", [
    ("32x0e+64x1o", "96x0e+32x1o", True), ("4x0o+32x0e", "32x0e", True), ("32x0e", "32x0e+4x0o", True),
    ("3x0o+32x0e", "32x0e", False), ("32x0e+3x1o", "32x0e", False), ("32x0e", "32x0e+1x0o", False), ("2x0o+32x0e+2x1e", "32x0e", False),
])
@pytest.mark.parametrize("classes", [1, 3])
def test_plans_pass_the_library_checks(s_in, s_out, fused, classes):
    m = cb.Linear(s_in, s_out, layout=cb.mul_ir, internal_weights=False, shared_weights=True, weight_classes=classes)
    assert (m._fused_plan is not None) == fused and m._dense_plan is not None
    if not fused:
        return
    L, t = _lib.lib(), torch.zeros(8, 512)
    for fn, ld in ((L.cueq_b200_linear_map, m.irreps_out.dim), (L.cueq_b200_linear_gw, m.irreps_out.dim)):
        a = _lib.LinearArgs()
        a.x, a.w, a.out = t.data_ptr(), t.data_ptr(), t.data_ptr()
        a.bounds = _lib.int32_array([0] * (classes + 1))                      # no rows: checked, not launched
        a.num_paths, a.num_classes, a.struct_bytes = len(m._fused_plan["paths"]), classes, C.sizeof(a)
        a.ldx, a.ldo, a.w_class_stride = m.irreps_in.dim, ld, m.weight_numel
        for q, (wo, u, v, xo, oo, d, c) in zip(a.paths, m._fused_plan["paths"]):
            q.u, q.v, q.d, q.x_off, q.out_off, q.w_off, q.c = u, v, d, xo, oo, wo, c
        assert fn(C.byref(a), None) == 0, L.cueq_b200_last_error()


@pytest.mark.gpu
@pytest.mark.parametrize("s_in,s_out,classes", [("3x0o+32x0e", "32x0e", 1), ("32x0e+3x1o", "32x0e", 3), ("32x0e+32x1o", "32x0e+1x0o+32x1o", 3)])
def test_odd_rows_against_float64_sums(s_in, s_out, classes):
    m = cb.Linear(s_in, s_out, layout=cb.ir_mul, internal_weights=False, shared_weights=True, weight_classes=classes)
    gen = torch.Generator().manual_seed(3)
    x, w = torch.randn(300, m.irreps_in.dim, generator=gen), torch.randn(classes, m.weight_numel, generator=gen)
    cot = torch.randn(300, m.irreps_out.dim, generator=gen)
    idx = torch.sort(torch.randint(0, classes, (300,), generator=gen)).values
    wd = w.cuda().requires_grad_(True)
    out = m(x.cuda(), wd, idx.cuda() if classes > 1 else None)
    (gw,) = torch.autograd.grad(out, wd, cot.cuda())
    ref, rgw = torch.zeros_like(cot).double(), torch.zeros_like(w).double()
    xd, cd = x.double(), cot.double()
    for wo, u, v, xo, oo, d, c in m._dense_plan["paths"]:
        W = w.double()[idx, wo : wo + u * v].view(-1, u, v) * c
        xb, gb = xd[:, xo : xo + d * u].view(-1, d, u), cd[:, oo : oo + d * v].view(-1, d, v)
        ref[:, oo : oo + d * v] = torch.einsum("zdu,zuv->zdv", xb, W).reshape(-1, d * v)
        rgw[:, wo : wo + u * v].index_add_(0, idx, torch.einsum("zdu,zdv->zuv", xb, gb).reshape(-1, u * v) * c)
    # 32 products of 2^-21 each and a chain of at most 300 * 3 additions of 2^-23, against sums of magnitude sqrt(terms)
    assert torch.allclose(out.detach().cpu().double(), ref, rtol=1e-5, atol=1e-5)
    assert torch.allclose(gw.cpu().double(), rgw, rtol=1e-5, atol=300 * 3 * 2.0 ** -23 * 30)
