"""GPU parity of the matmul operator's one-launch form at the edges of its tiles: every operand type and storage
order, broadcast batches, results of one row; bit for bit against the oracle."""
import itertools
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(__file__))
import oracle as O  # noqa: E402
import bolt_b200 as B  # noqa: E402
from bolt_b200 import synth  # noqa: E402
from test_matmul_gpu import matmul_gpu  # noqa: E402
from util import dev_zeros, dptr, to_dev, to_host  # noqa: E402

pytestmark = pytest.mark.gpu
F, U, I = B.DT_F32, B.DT_U8_Q, B.DT_I8


def check(args):
    C, s = matmul_gpu(*args)
    Cp, sp = O.port_matmul(*args)
    assert C.tobytes() == Cp.tobytes() and np.float32(s) == np.float32(sp)


def operand(seed, shape, dt):
    return synth.normal(seed, shape) if dt == F else (synth.u8(seed, shape) if dt == U else synth.s8(seed, shape))


@pytest.mark.parametrize("m,k,n", [(2, 3, 5), (7, 31, 8), (32, 64, 129), (129, 65, 31), (130, 257, 100), (128, 128, 64)])
@pytest.mark.parametrize("a_dt", [F, U])
@pytest.mark.parametrize("b_dt", [F, I])
def test_products(m, k, n, a_dt, b_dt):
    for ta, tb in itertools.product((0, 1), (0, 1)):
        a = operand(1, (3, k, m) if ta else (3, m, k), a_dt)
        b = operand(2, (3, n, k) if tb else (3, k, n), b_dt)
        sa, sb = (-1.0 if a_dt == F else 11.0), (-1.0 if b_dt == F else 7.0)
        check((a, a_dt, sa, ta, b, b_dt, sb, tb, None, F, -1.0))
        check((a, a_dt, sa, ta, b, b_dt, sb, tb, None, U, 3.0))


@pytest.mark.parametrize("k,n", [(3, 5), (64, 384), (384, 64), (130, 33)])
@pytest.mark.parametrize("a_dt", [F, I])
@pytest.mark.parametrize("b_dt", [F, U])
def test_one_row(k, n, a_dt, b_dt):
    for tb, c_scale in itertools.product((0, 1), (-1.0, 3.0)):
        a, b = operand(3, (2, 5, 1, k), a_dt), operand(4, (2, 5, n, k) if tb else (2, 5, k, n), b_dt)
        sa, sb = (-1.0 if a_dt == F else 9.0), (-1.0 if b_dt == F else 13.0)
        check((a, a_dt, sa, 0, b, b_dt, sb, tb, None, F if c_scale < 0 else U, c_scale))


def test_broadcast_bias_and_scale_edges():
    a, b = synth.normal(5, (4, 3, 20, 24)), synth.normal(6, (1, 3, 24, 40))
    check((a, F, -1.0, 0, b, F, -1.0, 0, None, F, -1.0))
    check((a[:, :1], F, -1.0, 0, synth.normal(7, (4, 3, 24, 40)), F, -1.0, 0, None, F, -1.0))
    check((a, F, -1.0, 0, b, F, -1.0, 0, synth.normal(8, (40,)), F, -1.0))
    check((a, F, 500.0, 0, b, F, -1.0, 0, None, F, -1.0))              # a given scale above the dynamic one wins
    check((np.zeros_like(a), F, -1.0, 0, b, F, -1.0, 0, None, F, -1.0))


@pytest.mark.parametrize("m,k,n", [(1, 640, 640), (128, 128, 128), (300, 96, 96)])
@pytest.mark.parametrize("over", [0, 1])
def test_result_over_its_operands(m, k, n, over):
    a, b = synth.normal(21, (3, m, k)), synth.normal(22, (3, k, n))
    d_a, d_b = to_dev(a), to_dev(b)
    ad, bd, cd = B.tensor_nd(F, a.shape), B.tensor_nd(F, b.shape), B.tensor_nd(F, (3, m, n))
    tmp_bytes = B.matmul_infer_forward_tmp_bytes(ad, 0, bd, 0, cd, -1.0)
    d_c = (d_a, d_b)[over]
    if d_c.numel() < 3 * m * n * 4:
        pytest.skip("C is larger than the operand")
    B.matmul(ad, 0, dptr(d_a), -1.0, bd, 0, dptr(d_b), -1.0, None, None, tmp_bytes, dptr(dev_zeros(tmp_bytes)), cd, dptr(d_c), -1.0)
    ref, _ = O.port_matmul(a, F, -1.0, 0, b, F, -1.0, 0, None, F, -1.0)
    assert to_host(d_c, np.float32, 3 * m * n).tobytes() == np.ascontiguousarray(ref).tobytes()


SPECIAL = [np.inf, -np.inf, 3e38, -3e38, np.float32(2147483648.0), np.float32(2147483520.0), -2147483648.0, 254.5, 255.5, -0.5]


@pytest.mark.parametrize("m", [1, 5])
@pytest.mark.parametrize("given", [-1.0, 1.0, 5.0, 1e30])
def test_quantization_of_extreme_values(m, given):
    """infinities, products beyond the int32 range and ties through the quantization inside the batched kernels; a given scale
    above the dynamic one is what takes finite values out of range"""
    for i, v in enumerate(SPECIAL):
        a, b = synth.normal(31, (2, m, 40)), synth.normal(32, (2, 40, 24))
        for x in ((a, b)[i % 2], (a, b)[1 - i % 2]):
            y = x.copy()
            y[0, 0, 3] = y[1, -1, 7] = v
            A, Bm = (y, b) if x is a else (a, y)
            with np.errstate(all="ignore"):
                C, _ = matmul_gpu(A, F, given, 0, Bm, F, given, 0, None, F, -1.0)
                Cp, _ = O.port_matmul(A, F, given, 0, Bm, F, given, 0, None, F, -1.0)
            assert np.array_equal(C, Cp, equal_nan=True), (v, x is a)


@pytest.mark.parametrize("m", [1, 24])
@pytest.mark.parametrize("given", [-1.0, 5.0])
def test_nan_goes_the_way_of_the_separate_kernels(m, given):
    """a NaN is the largest magnitude for every kernel that looks for one, and makes the scale NaN; the result over its own
    operand takes the quantize and GEMM (GEMV) kernels"""
    a, b = synth.normal(33, (2, m, 32)), synth.normal(34, (2, 32, 32))
    a[1, 0, 5] = np.nan
    ad, bd = B.tensor_nd(F, a.shape), B.tensor_nd(F, b.shape)
    tmp_bytes = B.matmul_infer_forward_tmp_bytes(ad, 0, bd, 0, ad, -1.0)
    got = []
    for apart in (True, False):
        d_a, d_b = to_dev(a), to_dev(b)
        d_c = dev_zeros(a.nbytes) if apart else d_a
        B.matmul(ad, 0, dptr(d_a), given, bd, 0, dptr(d_b), -1.0, None, None, tmp_bytes, dptr(dev_zeros(tmp_bytes)), ad, dptr(d_c), -1.0)
        got.append(to_host(d_c, np.float32, a.size))
    assert np.array_equal(got[0], got[1], equal_nan=True)


@pytest.mark.parametrize("m,k,n,batch", [(40, 6001, 33, 1), (128, 9000, 128, 1), (33, 9000, 40, 2), (16, 3000, 24, 7)])
@pytest.mark.parametrize("a_dt", [F, U])
@pytest.mark.parametrize("b_dt", [F, I])
def test_long_k(m, k, n, batch, a_dt, b_dt):
    """on both sides of the rule that sends a few tiles with a long K through the separate kernels"""
    sa, sb = (-1.0 if a_dt == F else 11.0), (-1.0 if b_dt == F else 7.0)
    for ta, tb in itertools.product((0, 1), (0, 1)):
        a, b = operand(35, (batch, k, m) if ta else (batch, m, k), a_dt), operand(36, (batch, n, k) if tb else (batch, k, n), b_dt)
        check((a, a_dt, sa, ta, b, b_dt, sb, tb, None, F, -1.0))
        check((a, a_dt, sa, ta, b, b_dt, sb, tb, synth.normal(37, (n,)), F, -1.0))
        check((a, a_dt, sa, ta, b, b_dt, sb, tb, None, U, (-1.0, 0.5)[ta]))


@pytest.mark.parametrize("k,n,batch", [(4099, 65, 1), (4096, 128, 1), (9001, 96, 2), (2048, 40, 5), (768, 2, 1)])
@pytest.mark.parametrize("a_dt", [F, I])
@pytest.mark.parametrize("b_dt", [F, U])
def test_one_long_row(k, n, batch, a_dt, b_dt):
    """the same for a result of one row, whose matrix is stored either way"""
    sa, sb = (-1.0 if a_dt == F else 9.0), (-1.0 if b_dt == F else 13.0)
    for tb, c_scale in itertools.product((0, 1), (-1.0, 0.5)):
        a, b = operand(38, (batch, 1, k), a_dt), operand(39, (batch, n, k) if tb else (batch, k, n), b_dt)
        check((a, a_dt, sa, 0, b, b_dt, sb, tb, None, F if c_scale < 0 else U, c_scale))
        check((a, a_dt, sa, 0, b, b_dt, sb, tb, None, U, -1.0))


def test_single_large_product_goes_one_by_one():
    a, b = synth.normal(9, (1, 1040, 1024)), synth.normal(10, (1, 1024, 1040))
    check((a, F, -1.0, 0, b, F, -1.0, 0, None, F, -1.0))
