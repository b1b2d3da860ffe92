"""GPU parity of the few-rows GEMM at the edges of its blocks (rows in sixteens, columns in eights, K in 64-byte units,
the batches of a warp), and of a chain of layers in one call: bit for bit against the oracle."""
import ctypes as C
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(__file__))
import oracle as O  # noqa: E402
import bolt_b200 as B  # noqa: E402
from bolt_b200 import synth  # noqa: E402
from test_gather_gpu import product  # noqa: E402
from util import dev_zeros, dptr, to_dev, to_host  # noqa: E402

pytestmark = pytest.mark.gpu
F32 = B.DT_F32


@pytest.mark.parametrize("m", [1, 2, 15, 16, 17, 32, 33, 64, 65])
@pytest.mark.parametrize("k,n", [(16, 1), (48, 7), (64, 8), (80, 33), (768, 24), (4112, 40), (32, 1185), (272, 1192), (64, 6148)])
@pytest.mark.parametrize("out", ["s32", "f32", "u8"])
def test_products(m, k, n, out):
    got, ref = product(m, k, n, 0, out)
    assert got.tobytes() == np.ascontiguousarray(ref).tobytes()


def chain_layers(m, dims, seed):
    layers = []
    for i, (k, n) in enumerate(zip(dims[:-1], dims[1:])):
        W = synth.s8(seed + i, (k, n))
        desc = B.tensor2df(B.DT_I8, B.DF_NORMAL, k, n)
        nbytes, rhs = B.matrix_matrix_multiply_transform_rhs_bytes(desc)
        packed = dev_zeros(nbytes)
        B.matrix_matrix_multiply_transform_rhs(desc, dptr(to_dev(W)), dptr(packed))
        col = (np.abs(synth.normal(seed + 50 + i, (n,))) + np.float32(100)).astype(np.float32)
        layers.append((k, n, packed, rhs, to_dev(col)))
    return layers


@pytest.mark.parametrize("m", [1, 16, 32, 40, 100])
def test_chain_equals_single_calls(m):
    """more layers than fit the GPU at once, few-rows and tensor-tile layers mixed (2048 and 7168 columns)"""
    lib = B.lib()
    dims = [256, 2048, 256, 7168, 128, 128, 1024, 64]
    layers = chain_layers(m, dims, 700)
    x = to_dev(synth.u8(7, (m, dims[0])))
    results = []
    for chained in (False, True):
        bufs = [dev_zeros(m * n * 4) for _, n, _, _, _ in layers]
        calls = (B.GemmCall * len(layers))()
        a = x
        for c, (k, n, packed, rhs, col), out in zip(calls, layers, bufs):
            last = out is bufs[-1]
            c.N, c.M, c.K, c.A, c.packedB, c.offsetC, c.C = n, m, k, a.data_ptr(), packed.data_ptr(), packed.data_ptr() + rhs, out.data_ptr()
            c.epilogue.out_dt, c.epilogue.out_scale, c.epilogue.sA, c.epilogue.sB = (B.DT_F32 if last else B.DT_U8_Q), 0.6, 1.5, 1.0
            c.epilogue.col_scale = col.data_ptr()
            a = out
        for _ in range(3):      # back to back, so that a call's first layer meets the previous call's last
            if chained:
                B.CHECK_STATUS(lib.bolt_b200_gemm_u8s8_chain(calls, len(calls)))
            else:
                for c in calls:
                    B.CHECK_STATUS(lib.bolt_b200_gemm_u8s8_ex(c.N, c.M, c.K, c.A, c.packedB, c.offsetC, c.C, C.byref(c.epilogue)))
        B.CHECK_STATUS(lib.bolt_b200_synchronize(), "synchronize")
        results.append([to_host(b, np.uint8, m * n).tobytes() for b, (_, n, _, _, _) in zip(bufs[:-1], layers)] + [to_host(bufs[-1], np.float32, m * dims[-1]).tobytes()])
    assert results[0] == results[1]
    # the first layer's single call against the oracle's accumulators
    k, n, packed, rhs, col = layers[0]
    acc = O.port_gemm(to_host(x, np.uint8, m * k).reshape(m, k), synth.s8(700, (k, n)), O.port_offsetc(synth.s8(700, (k, n))))
    fac = (np.float32(0.6) / (np.float32(1.5) * to_host(col, np.float32, n))).astype(np.float32)
    r = np.rint((acc.astype(np.float32) * fac[None, :]).astype(np.float32)).astype(np.int64) + 128
    assert results[0][0] == np.where(r < 0, 255, np.minimum(r, 255)).astype(np.uint8).tobytes()


@pytest.mark.parametrize("m", [1, 16])
def test_input_scale_from_an_earlier_call(m):
    """d_sA may be what an earlier call of the chain writes.  That call has a long K, so that a later one that
    did not wait for it would read what the buffer held before."""
    lib, k0, k, n = B.lib(), 16384, 256, 512
    (_, _, w0, r0, _), (_, _, w1, r1, _), (_, _, w2, r2, col) = chain_layers(m, [k0, 8], 900) + chain_layers(m, [k, n], 910) + chain_layers(m, [k, n], 920)
    x0, x = synth.u8(31, (m, k0)), synth.u8(32, (m, k))
    d_x0, d_x, d_s, d_mid, d_out = to_dev(x0), to_dev(x), dev_zeros(m * 8 * 4), dev_zeros(m * n * 4), dev_zeros(m * n * 4)
    calls = (B.GemmCall * 3)()
    for c, (M, K, N, a, w, r, out) in zip(calls, ((m, k, n, d_x, w1, r1, d_mid), (m, k0, 8, d_x0, w0, r0, d_s), (m, k, n, d_x, w2, r2, d_out))):
        c.N, c.M, c.K, c.A, c.packedB, c.offsetC, c.C = N, M, K, a.data_ptr(), w.data_ptr(), w.data_ptr() + r, out.data_ptr()
        c.epilogue.out_dt, c.epilogue.out_scale, c.epilogue.sA, c.epilogue.sB = B.DT_F32, 1.0, 1.0, 1.0
    calls[2].epilogue.d_sA, calls[2].epilogue.col_scale = d_s.data_ptr(), col.data_ptr()
    acc0 = O.port_gemm(x0, synth.s8(900, (k0, 8)), O.port_offsetc(synth.s8(900, (k0, 8))))
    acc = O.port_gemm(x, synth.s8(920, (k, n)), O.port_offsetc(synth.s8(920, (k, n))))
    fac = (np.float32(1) / (np.float32(acc0[0, 0]) * to_host(col, np.float32, n))).astype(np.float32)
    ref = (acc.astype(np.float32) * fac[None, :]).astype(np.float32).tobytes()
    for _ in range(20):
        d_s.fill_(0x3F)
        B.CHECK_STATUS(lib.bolt_b200_gemm_u8s8_chain(calls, 3))
        B.CHECK_STATUS(lib.bolt_b200_synchronize(), "synchronize")
        assert to_host(d_out, np.float32, m * n).tobytes() == ref


@pytest.mark.parametrize("m", [1, 16, 17, 33, 64])
@pytest.mark.parametrize("n", [24, 33])
@pytest.mark.parametrize("out", [B.DT_F32, B.DT_U8_Q])
@pytest.mark.parametrize("scales", ["row", "row_col", "col", "factor", "d_sA"])
def test_scales(m, n, out, scales):
    """per-row and per-column scales, ready-made factors, an input scale in device memory: one binary32 product, one division"""
    k = 272
    A, W = synth.u8(41, (m, k)), synth.s8(42, (k, n))
    (_, _, packed, rhs, _), = chain_layers(m, [k, n], 42)
    row = (np.abs(synth.normal(43, (m,))) + 5).astype(np.float32)
    col = (np.abs(synth.normal(44, (n,))) + 100).astype(np.float32)
    num = np.float32(40.0 if out == B.DT_U8_Q else 1.0)
    ep = B.GemmEpilogue()
    ep.out_dt, ep.out_scale, ep.sA, ep.sB = out, float(num), 7.5, 90.0
    sA, sB = np.float32(7.5), np.float32(90.0)
    d_row, d_col, d_fac, d_sa = to_dev(row), to_dev(col), to_dev((num / col).astype(np.float32)), to_dev(np.array([3.25], np.float32))
    if "row" in scales:
        ep.row_scale, sA = d_row.data_ptr(), row[:, None]
    if "col" in scales:
        ep.col_scale, sB = d_col.data_ptr(), col[None, :]
    if scales == "d_sA":
        ep.d_sA, sA = d_sa.data_ptr(), np.float32(3.25)
    fac = (num / (sA * sB).astype(np.float32)).astype(np.float32) * np.ones((m, n), np.float32)
    if scales == "factor":
        ep.col_factor, fac = d_fac.data_ptr(), (num / col).astype(np.float32)[None, :]
    d_a, d_c = to_dev(A), dev_zeros(m * n * 4)
    B.CHECK_STATUS(B.lib().bolt_b200_gemm_u8s8_ex(n, m, k, dptr(d_a), dptr(packed), dptr(packed, rhs), dptr(d_c), C.byref(ep)))
    v = (O.port_gemm(A, W, O.port_offsetc(W)).astype(np.float32) * fac).astype(np.float32)
    if out == B.DT_F32:
        assert to_host(d_c, np.float32, m * n).tobytes() == np.ascontiguousarray(v).tobytes()
    else:
        r = np.rint(v).astype(np.int64) + 128
        assert to_host(d_c, np.uint8, m * n).tobytes() == np.where(r < 0, 255, np.minimum(r, 255)).astype(np.uint8).tobytes()


@pytest.mark.parametrize("m", [1, 32])
def test_chain_with_host_pointers(m):
    """the first input and the last result in host memory, the layers between them on the device"""
    lib, dims = B.lib(), [256, 128, 512, 64]
    layers = chain_layers(m, dims, 800)
    x = synth.u8(9, (m, dims[0]))
    bufs = [dev_zeros(m * n * 4) for _, n, _, _, _ in layers]
    host_out = np.zeros(m * dims[-1], np.float32)
    got = []
    for host in (False, True):
        calls = (B.GemmCall * len(layers))()
        d_x = to_dev(x)
        a = x.ctypes.data if host else d_x.data_ptr()
        for c, (k, n, packed, rhs, col), out in zip(calls, layers, bufs):
            last = out is bufs[-1]
            c.N, c.M, c.K, c.A, c.packedB, c.offsetC = n, m, k, a, packed.data_ptr(), packed.data_ptr() + rhs
            a = c.C = host_out.ctypes.data if host and last else out.data_ptr()
            c.epilogue.out_dt, c.epilogue.out_scale, c.epilogue.sA, c.epilogue.sB = (F32 if last else B.DT_U8_Q), 0.6, 1.5, 1.0
            c.epilogue.col_scale = col.data_ptr()
        B.CHECK_STATUS(lib.bolt_b200_gemm_u8s8_chain(calls, len(calls)))
        B.CHECK_STATUS(lib.bolt_b200_synchronize(), "synchronize")
        got.append(host_out.tobytes() if host else to_host(bufs[-1], np.float32, m * dims[-1]).tobytes())
    assert got[0] == got[1] and np.any(np.frombuffer(got[0], np.float32))


def test_chain_errors():
    lib = B.lib()
    assert lib.bolt_b200_gemm_u8s8_chain(None, 0) == B.SUCCESS
    assert lib.bolt_b200_gemm_u8s8_chain(None, 1) == B.NULL_POINTER
    calls = (B.GemmCall * 1)()
    calls[0].N, calls[0].M, calls[0].K = 8, 2, 16
    calls[0].epilogue.out_dt = B.DT_F32
    assert lib.bolt_b200_gemm_u8s8_chain(calls, 1) == B.NULL_POINTER
