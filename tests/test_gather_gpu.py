"""GPU parity of the products whose operands TMA cannot fetch (ragged K, transposed A, unaligned operands) at the
edges of the kernel's tiles: bit for bit against the oracle."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(__file__))
import oracle as O  # noqa: E402
import bolt_b200 as B  # noqa: E402
from bolt_b200 import synth  # noqa: E402
from util import dev_zeros, dptr, to_dev, to_host  # noqa: E402

pytestmark = pytest.mark.gpu


def product(m, k, n, a_t, out, shift=0, seed=3):
    A, W = synth.u8(seed, (m, k)), synth.s8(seed + 1, (k, n))
    Cin = synth.integers(seed + 2, (m, n), -1000, 1000).astype(np.int32)
    bdesc = B.tensor2df(B.DT_I8, B.DF_NORMAL, k, n)
    nbytes, rhs = B.matrix_matrix_multiply_transform_rhs_bytes(bdesc)
    d_a, d_pack = dev_zeros(m * k + shift), dev_zeros(nbytes)
    raw = to_dev(np.ascontiguousarray(A.T) if a_t else A)
    d_a[shift: shift + m * k] = raw
    pdesc = B.matrix_matrix_multiply_transform_rhs(bdesc, dptr(to_dev(W)), dptr(d_pack))
    adesc = B.tensor2df(B.DT_U8_Q, B.DF_TRANSPOSE, k, m) if a_t else B.tensor2df(B.DT_U8_Q, B.DF_NORMAL, m, k)
    tb = B.matrix_matrix_multiply_tmp_bytes(adesc, pdesc)
    d_tmp = dev_zeros(tb)
    d_tmp[: 4 * n] = d_pack[rhs: rhs + 4 * n]
    dt, npdt, scale = {"s32": (B.DT_I32, np.int32, None), "f32": (B.DT_F32, np.float32, [0.37]), "u8": (B.DT_U8_Q, np.uint8, [-1, 0.004])}[out]
    d_c = to_dev(Cin)
    B.matrix_matrix_multiply(adesc, dptr(d_a, shift), pdesc, dptr(d_pack), tb, dptr(d_tmp), B.tensor2df(dt, B.DF_NORMAL, m, n), dptr(d_c), scale)
    B.CHECK_STATUS(B.lib().bolt_b200_synchronize(), "synchronize")
    assert B.lib().bolt_b200_last_gemm_used_tensor_cores() == 1
    got = to_host(d_c, npdt, m * n).reshape(m, n)
    ref = O.port_gemm(A, W, O.port_offsetc(W), scale, None if out == "u8" else (Cin if out == "s32" else Cin.view(np.float32)))
    return got, ref


@pytest.mark.parametrize("m,k,n", [(1, 1, 1), (2, 127, 31), (128, 129, 33), (129, 255, 64), (127, 257, 97), (130, 515, 128), (257, 640, 130), (333, 1031, 200)])
@pytest.mark.parametrize("a_t", [0, 1])
@pytest.mark.parametrize("out", ["s32", "f32", "u8"])
def test_ragged(m, k, n, a_t, out):
    got, ref = product(m, k, n, a_t, out)
    assert got.tobytes() == np.ascontiguousarray(ref).tobytes()


@pytest.mark.parametrize("shift", [1, 4, 8, 15])
@pytest.mark.parametrize("a_t", [0, 1])
def test_unaligned_operand(shift, a_t):
    got, ref = product(130, 256, 96, a_t, "f32", shift)
    assert got.tobytes() == np.ascontiguousarray(ref).tobytes()


def test_many_tiles_per_cta():
    got, ref = product(3000, 77, 3000, 0, "s32")
    assert got.tobytes() == np.ascontiguousarray(ref).tobytes()
