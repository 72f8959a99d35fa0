"""Argument blocks of version 1 of the C interface, as a program built against an older header passes them (CPU): nothing
behind their end and no reserved word is read."""
import ctypes as C

import pytest

from cuequivariance_b200 import _lib, channelwise as cw, descriptors as D


class OldCwArgs(C.Structure):
    _fields_ = [
        ("w", C.c_void_p), ("x1", C.c_void_p), ("x2", C.c_void_p), ("out", C.c_void_p),
        ("gout", C.c_void_p), ("gw", C.c_void_p), ("gx1", C.c_void_p), ("gx2", C.c_void_p),
        ("senders", C.c_void_p), ("order", C.c_void_p), ("rowptr", C.c_void_p),
        ("tab_start", C.c_void_p), ("tab_j", C.c_void_p), ("tab_c", C.c_void_p), ("bwd_coef", C.c_void_p),
        ("w_stride", C.c_int64), ("x1_stride", C.c_int64), ("x2_stride", C.c_int64), ("out_stride", C.c_int64),
        ("num_receivers", C.c_int64),
        ("extent", C.c_int32), ("x1_offset", C.c_int32), ("num_paths", C.c_int32), ("num_terms", C.c_int32),
        ("w_offset", C.c_int32 * 8), ("out_offset", C.c_int32 * 8),
        ("x1_mul_ir", C.c_int32), ("out_mul_ir", C.c_int32), ("channels_per_lane", C.c_int32), ("staging", C.c_int32),
        ("status", C.c_void_p), ("recv_mod", C.c_int32), ("variant", C.c_int32),
    ]


class Padded(C.Structure):
    _fields_ = [("a", OldCwArgs), ("behind", C.c_uint8 * 256)]


@pytest.mark.parametrize("which", ["fwd_tab", "bwd_tab"])
def test_nothing_behind_the_channelwise_block_is_read(which):
    assert C.sizeof(_lib.CwArgs) == C.sizeof(OldCwArgs)
    L = _lib.lib()
    plan = cw.match_channelwise(D.channelwise_tensor_product("8x0e+8x1o+8x2e+8x3o", "0e+1o+2e+3o", ["0e", "1o", "2e", "3o"]).polynomial)
    page = (C.c_float * 64)()
    at = (C.addressof(page) + 15) // 16 * 16
    for g in plan.groups:
        b = Padded()
        C.memset(C.byref(b), 0xA5, C.sizeof(b))
        C.memset(C.byref(b.a), 0, C.sizeof(b.a))
        a = b.a
        a.w = a.x1 = a.x2 = a.out = a.gout = a.rowptr = a.tab_start = a.tab_j = a.tab_c = a.bwd_coef = at
        a.w_stride, a.x1_stride, a.x2_stride, a.out_stride = plan.row_sizes
        a.extent, a.x1_offset, a.num_paths, a.num_terms = plan.extent, g["x1_off"], g["npath"], g["nterm"] if which == "bwd_tab" else g["nterm_fwd"]
        for q in range(g["npath"]):
            a.w_offset[q], a.out_offset[q] = g["w_off"][q], g["out_off"][q]
        coef = (C.c_float * g["nterm"])()
        a.bwd_coef = C.addressof(coef)
        fn = C.CDLL(str(_lib.LIB_PATH))["cueq_b200_cw_forward" if which == "fwd_tab" else "cueq_b200_cw_backward"]
        assert fn(C.c_int(g["id"]), C.byref(b), None) == 0, L.cueq_b200_last_error()      # no receivers: checked, not launched


def test_reserved_word_of_a_buffer_is_not_read():
    L = C.CDLL(str(_lib.LIB_PATH))
    L.cueq_b200_u1d_static_name.restype = C.c_char_p
    kid = next(i for i in range(64) if L.cueq_b200_u1d_static_name(i) == b"sc_l3_l1_d3_fwd")
    bufs = (_lib.Buffer * 3)()
    C.memset(bufs, 0xA5, C.sizeof(bufs))
    page = (C.c_int32 * 64)()
    for b, (mode, rows) in zip(bufs, ((_lib.INDEXED, 4), (_lib.BATCHED, 0), (_lib.BATCHED, 0))):
        b.ptr, b.rows, b.mode, b.dtype, b.index, b.index_is_64 = C.addressof(page), rows, mode, _lib.F32, C.addressof(page), 0
    _lib.lib()
    assert L.cueq_b200_u1d_static_launch(C.c_int(kid), C.c_int64(0), C.c_int32(32), bufs, _lib.int32_array([1, 1, 1]),
                                         _lib.int32_array([8, 16, 4]), C.c_int32(3), None) == 0, _lib.lib().cueq_b200_last_error()
