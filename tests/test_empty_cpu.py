"""Operators on empty tensors: what they refuse, they refuse before any device work (none is needed to run this), with an
error code, and the process lives on.  Pointers only have to be non-null; nothing reads them."""
import ctypes as C

import pytest

import bolt_b200 as B

DUMMY = C.c_void_p(4096)


def convolution_code(n, ic, oc, out_dt=B.DT_F32, hw=8, binary=False):
    lib = B.lib()
    p = B.conv_param(oc, 3, 3, 1, 1)
    act = B.ActivationParamSpec()
    sd = B.tensor1d(B.DT_F32, 3)
    scale = (C.c_float * 3)(1.0, -1.0, 1.0)
    if binary:
        in_desc, out_desc = B.tensor4df(B.DT_F16, B.DF_NCHWC8, n, ic, hw, hw), B.tensor4df(B.DT_F16, B.DF_NCHWC8, n, oc, hw, hw)
        f_desc = B.tensor4df(B.DT_BIN11, B.DF_NCHWN16C8, oc, ic, 3, 3)
    else:
        in_desc, out_desc = B.tensor4df(B.DT_U8_Q, B.DF_NCHWC16, n, ic, hw, hw), B.tensor4df(out_dt, B.DF_NCHWC16, n, oc, hw, hw)
        f_desc = B.tensor4df(B.DT_I8, B.DF_NCHWC2NxC4, oc, ic, 3, 3)
    return lib.convolution_cuda_b200(C.byref(in_desc), DUMMY, None, C.byref(f_desc), DUMMY, C.byref(p), 0, C.byref(sd),
                                     DUMMY if binary else C.cast(scale, C.c_void_p), C.byref(sd), DUMMY if binary else None, 1 << 20, DUMMY,
                                     C.byref(out_desc), DUMMY, C.byref(act))


@pytest.mark.parametrize("n,ic,oc", [(0, 16, 64), (1, 16, 0), (1, 0, 64), (0, 0, 0)])
@pytest.mark.parametrize("out_dt", [B.DT_F32, B.DT_U8_Q])
def test_convolution_without_images_or_channels(n, ic, oc, out_dt):
    assert convolution_code(n, ic, oc, out_dt) == B.NOT_SUPPORTED


@pytest.mark.parametrize("n,ic,oc", [(0, 32, 64), (1, 32, 0), (1, 0, 64), (0, 0, 0)])
def test_one_bit_convolution_without_images_or_channels(n, ic, oc):
    """(without input channels the kernel's walk over the words of a tap would not end)"""
    assert convolution_code(n, ic, oc, binary=True) == B.NOT_SUPPORTED
