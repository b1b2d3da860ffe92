"""Host paths of the library against a CUDA runtime without a device (fake_gpu.py)."""
import ctypes as C
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(__file__))
import bolt_b200 as B  # noqa: E402
import fake_gpu  # noqa: E402

F, U, I = B.DT_F32, B.DT_U8_Q, B.DT_I8


def matmul_code(lib, a_shape, b_shape, c_shape, a_dt=F, b_dt=F, c_dt=F, c_scale=-1.0, bias=0, ta=0, tb=0, over=None, shift=0):
    """over: C lies over A (0) or B (1), `shift` bytes behind its start"""
    a, b, c = B.tensor_nd(a_dt, a_shape), B.tensor_nd(b_dt, b_shape), B.tensor_nd(c_dt, c_shape)
    buf = [np.zeros(max(int(np.prod(s)), 1) * 4 + 4096, np.uint8) for s in (a_shape, b_shape, c_shape)]
    pa, pb, pc = (C.c_void_p(x.ctypes.data) for x in buf)
    if over is not None:
        pc = C.c_void_p(buf[over].ctypes.data + shift)
    tmp, bvec = np.zeros(1 << 22, np.uint8), np.zeros(max(bias, 1), np.float32)
    s = C.c_float(c_scale)
    bd = B.tensor1d(F, bias)
    r = lib.matmul_cuda_b200(C.byref(a), ta, pa, 5.0, C.byref(b), tb, pb, 5.0, C.byref(bd) if bias else None,
                             C.c_void_p(bvec.ctypes.data) if bias else None, tmp.size, C.c_void_p(tmp.ctypes.data), C.byref(c), pc, C.byref(s))
    return r, s.value


@pytest.mark.parametrize("m", [1, 4])
@pytest.mark.parametrize("a_dt,b_dt", [(F, F), (None, None)])
@pytest.mark.parametrize("c_dt,c_scale,bias", [(F, -1.0, 0), (F, -1.0, 8), (U, -1.0, 0), (U, 3.0, 0)])
def test_matmul_without_products(m, a_dt, b_dt, c_dt, c_scale, bias):
    """an empty batch is a success that launches nothing and leaves no error behind for the thread's next call"""
    lib = fake_gpu.load()
    a_dt, b_dt = a_dt or (I if m == 1 else U), b_dt or (U if m == 1 else I)
    assert matmul_code(lib, (0, m, 16), (0, 16, 8), (0, m, 8), a_dt, b_dt, c_dt, c_scale, bias) == (B.SUCCESS, c_scale)
    assert lib.fake_last_error() == 0 and fake_gpu.launches(lib) == []


@pytest.mark.parametrize("m", [1, 4])
@pytest.mark.parametrize("a,b", [((0,), (1,)), ((1,), (0,)), ((0,), (0,)), ((3, 0), (3, 1))])
def test_matmul_products_without_operands(m, a, b):
    """C has products but an operand has none: there is nothing to read"""
    lib = fake_gpu.load()
    c = tuple(max(x, y) for x, y in zip(a, b)) if a != b else (2,)
    assert matmul_code(lib, a + (m, 16), b + (16, 8), c + (m, 8))[0] == B.NOT_MATCH
    assert lib.fake_last_error() == 0 and fake_gpu.launches(lib) == []


def test_device_scale_counts_in_the_callers_memory():
    """calls on several streams run at the same time: what one counts in, no other may"""
    lib = fake_gpu.load()
    x, scales = np.zeros(64, np.float32), np.zeros(2, np.float32)
    words = []
    for i in range(2):
        assert lib.bolt_b200_absmax_scale_f32(C.c_void_p(x.ctypes.data), x.size, C.c_void_p(scales.ctypes.data + 4 * i)) == B.SUCCESS
        words.append(lib.fake_max_words())
    assert words[0] != words[1]


def test_the_words_of_reported_maxima_are_cleared_before_the_first_call_uses_them():
    """cudaMemset returns before the memory is set and streams that do not block on the legacy one run past it"""
    lib = fake_gpu.fresh()
    x, q, s = np.zeros(64, np.float32), np.zeros(64, np.uint8), (C.c_float * 1)(-1.0)
    d, o = B.tensor1d(F, 64), B.tensor1d(U, 64)
    assert lib.quantize_cuda_b200(C.byref(d), C.c_void_p(x.ctypes.data), C.byref(o), C.c_void_p(q.ctypes.data), s, 0) == B.SUCCESS
    assert lib.fake_unordered_fills() == 0
    assert (C.c_uint * 2).from_address(lib.fake_max_words())[:] == [0, 0]


def test_a_device_whose_words_cannot_be_cleared_is_refused():
    lib = fake_gpu.fresh()
    lib.fake_refuse_fills(1)
    x, q, s = np.zeros(64, np.float32), np.zeros(64, np.uint8), (C.c_float * 1)(-1.0)
    d, o = B.tensor1d(F, 64), B.tensor1d(U, 64)
    call = lambda: lib.quantize_cuda_b200(C.byref(d), C.c_void_p(x.ctypes.data), C.byref(o), C.c_void_p(q.ctypes.data), s, 0)
    assert call() == B.UNKNOWN and fake_gpu.launches(lib) == []
    lib.fake_refuse_fills(0)
    assert call() == B.SUCCESS


@pytest.mark.parametrize("m,n,k", [(1, 24, 24), (24, 24, 24), (40, 16, 32)])
@pytest.mark.parametrize("over", [0, 1])
def test_matmul_over_its_operands_copies_them_first(m, n, k, over):
    lib = fake_gpu.load()
    size = (m * k, k * n)[over] * 4
    args = (lib, (1, m, k), (1, k, n), (1, m, n))
    batched = lambda: any("absmax_pair_kernel" in x for x in fake_gpu.launches(lib))
    for shift in (0, size - 4):
        lib.fake_forget_launches()
        assert matmul_code(*args, over=over, shift=shift)[0] == B.SUCCESS
        assert not batched()
    lib.fake_forget_launches()
    assert matmul_code(*args, over=over, shift=size)[0] == B.SUCCESS      # right behind: no overlap
    assert batched()
    lib.fake_forget_launches()
    assert matmul_code(*args, c_dt=U, over=over)[0] == B.SUCCESS          # goes through the scratch anyway
    assert batched()


def gemm_codes(lib, m, n, k, chained):
    a, w, out = np.zeros(m * k, np.uint8), np.zeros((n + 16) * (k + 16), np.int8), np.zeros(m * n, np.float32)
    w16 = (w.ctypes.data + 15) & ~15
    calls = (B.GemmCall * 2)()
    for c in calls:
        c.N, c.M, c.K, c.A, c.packedB, c.offsetC, c.C = n, m, k, (a.ctypes.data + 15) & ~15, w16, w16, out.ctypes.data
        c.epilogue.out_dt, c.epilogue.out_scale, c.epilogue.sA, c.epilogue.sB = F, 1.0, 1.0, 1.0
    if chained:
        return [lib.bolt_b200_gemm_u8s8_chain(calls, 2)]
    return [lib.bolt_b200_gemm_u8s8_ex(c.N, c.M, c.K, c.A, c.packedB, c.offsetC, c.C, C.byref(c.epilogue)) for c in calls]


@pytest.mark.parametrize("call", [
    lambda lib: gemm_codes(lib, 8, 64, 64, False), lambda lib: gemm_codes(lib, 8, 64, 64, True), lambda lib: gemm_codes(lib, 256, 64, 64, False),
    lambda lib: [matmul_code(lib, (2, m, 16), (2, 16, 8), (2, m, 8))[0] for m in (1, 4)]])
def test_programmatic_serialization_refused(call):
    """a runtime that does not take the launch attribute gets the plain launch, from then on at once"""
    lib = fake_gpu.fresh()
    lib.fake_refuse_programmatic(1)
    assert set(call(lib)) == {B.SUCCESS} and lib.fake_last_error() == 0
    n = lib.fake_refused()
    assert n >= 1
    assert set(call(lib)) == {B.SUCCESS} and lib.fake_refused() == n


@pytest.mark.parametrize("src,dst", [(F, U), (F, I), (U, I), (B.DT_I32, U), (B.DT_I32, I)])
@pytest.mark.parametrize("scale", [-1.0, 3.0])
def test_every_launch_is_counted_once(src, dst, scale):
    lib = fake_gpu.load()
    x, q, s = np.zeros(64, np.float32), np.zeros(64, np.uint8), (C.c_float * 2)(scale, 2.0)
    d, o = B.tensor1d(src, 64), B.tensor1d(dst, 64)
    before = lib.bolt_b200_launch_count()
    assert lib.quantize_cuda_b200(C.byref(d), C.c_void_p(x.ctypes.data), C.byref(o), C.c_void_p(q.ctypes.data), s, 1) == B.SUCCESS
    assert lib.bolt_b200_launch_count() - before == lib.fake_launches() != 0
    before, _ = lib.bolt_b200_launch_count(), lib.fake_forget_launches()
    for m, n in ((1, 8), (4, 8), (4, 1)):
        for c_dt, c_scale, bias in ((F, -1.0, n), (U, -1.0, 0), (U, 3.0, 0)):
            assert matmul_code(lib, (2, m, 16), (2, 16, n), (2, m, n), c_dt=c_dt, c_scale=c_scale, bias=bias)[0] == B.SUCCESS
    assert set(gemm_codes(lib, 8, 64, 64, True) + gemm_codes(lib, 256, 64, 64, False) + gemm_codes(lib, 8, 64, 63, False)) == {B.SUCCESS}
    assert lib.bolt_b200_absmax_scale_f32(C.c_void_p(x.ctypes.data), x.size, s) == B.SUCCESS
    assert lib.bolt_b200_launch_count() - before == lib.fake_launches()


KERNELS = {"gemm_skinny_kernel": "rows", "gemm_u8s8_tcgen05_kernel": "tma", "gemm_gather_kernel": "gathered", "mvm_batch_kernel": "row"}


def kernel_of(lib):
    """the kernels of a call, those around the products left out"""
    return [v for x in fake_gpu.launches(lib) for k, v in KERNELS.items() if k in x]


@pytest.mark.parametrize("m,k,n,expect", [
    (16, 768, 6144, "rows"), (16, 768, 6145, "tma"), (1, 5456, 6144, "rows"), (1, 5472, 6144, "tma"),                 # 32 MiB and 6144 columns
    (17, 2048, 6144, "rows"), (17, 2064, 6144, "tma"), (32, 16384, 2048, "rows"), (32, 16400, 2048, "tma"), (32, 6144, 2049, "tma"),
    (33, 768, 1184, "rows"), (33, 768, 1185, "tma"), (64, 768, 1184, "rows"), (65, 768, 1184, "tma"), (64, 28336, 1184, "rows"), (64, 28352, 1184, "tma"),
    (4096, 768, 3072, "tma"), (16, 760, 768, "gathered"), (300, 515, 1001, "gathered")])
def test_gemm_dispatch(m, k, n, expect):
    """both sides of every line of the rules; nothing reads the operands here"""
    lib = fake_gpu.load()
    ep = B.GemmEpilogue()
    ep.out_dt, ep.out_scale, ep.sA, ep.sB = F, 1.0, 1.0, 1.0
    call = lambda a: lib.bolt_b200_gemm_u8s8_ex(n, m, k, C.c_void_p(a), C.c_void_p(8192), C.c_void_p(8192), C.c_void_p(16384), C.byref(ep))
    assert call(4096) == B.SUCCESS and kernel_of(lib) == [expect]
    assert lib.bolt_b200_last_gemm_used_tensor_cores() == 1
    lib.fake_forget_launches()
    assert call(4097) == B.SUCCESS and kernel_of(lib) == ["gathered"]      # rows of A off the 16-byte grid


def test_matmul_reports_what_ran():
    lib = fake_gpu.load()
    for m, n, tc in ((4, 8, 1), (1, 8, 0), (4, 8, 1), (4, 1, 0)):
        assert matmul_code(lib, (2, m, 16), (2, 16, n), (2, m, n))[0] == B.SUCCESS
        assert lib.bolt_b200_last_gemm_used_tensor_cores() == tc, (m, n)


def matmul_route(lib, b, m, n, k, ta, tb, a_dt, b_dt, a_at=1 << 20):
    """(status, whether the call took the batched kernels)"""
    a, w, c = B.tensor_nd(a_dt, (b, k, m) if ta else (b, m, k)), B.tensor_nd(b_dt, (b, n, k) if tb else (b, k, n)), B.tensor_nd(F, (b, m, n))
    nbytes = C.c_uint32()
    assert lib.matmul_infer_forward_tmp_bytes_cuda_b200(C.byref(a), ta, C.byref(w), tb, C.byref(c), -1.0, C.byref(nbytes)) == B.SUCCESS
    tmp, out, s = np.empty(nbytes.value, np.uint8), np.empty(b * m * n, np.float32), C.c_float(-1.0)
    lib.fake_forget_launches()
    code = lib.matmul_cuda_b200(C.byref(a), ta, C.c_void_p(a_at), 11.0, C.byref(w), tb, C.c_void_p(1 << 40), 7.0, None, None, nbytes.value,
                                C.c_void_p(tmp.ctypes.data), C.byref(c), C.c_void_p(out.ctypes.data), C.byref(s))
    return code, any("absmax_pair_kernel" in x or "mvm_batch_kernel" in x or "gemm_gather_kernel" in x and "Lb1EE" in x for x in fake_gpu.launches(lib))


@pytest.mark.parametrize("b,m,n,k,tb,f32,batched", [
    (1, 128, 128, 1024, 1, 1, 1), (1, 128, 128, 2048, 1, 1, 0), (1, 1024, 1024, 256, 1, 1, 1), (1, 1024, 1024, 1024, 1, 1, 0), (1, 4096, 4096, 64, 1, 1, 1),
    (4, 128, 128, 2048, 1, 1, 1), (4, 128, 128, 8192, 1, 1, 0), (12, 16, 64, 16384, 1, 1, 1), (64, 128, 128, 2048, 1, 1, 1), (24, 128, 64, 128, 0, 1, 1),
    (1, 128, 128, 1024, 1, 0, 1), (1, 128, 128, 2048, 1, 0, 0), (4, 256, 256, 16384, 1, 0, 1), (1, 16, 16384, 4096, 1, 0, 1), (1, 2048, 2048, 2048, 0, 0, 0),
    (1, 1, 768, 768, 1, 1, 1), (1, 1, 768, 3072, 1, 1, 0), (1, 1, 768, 3072, 0, 1, 1), (4, 1, 2048, 2048, 1, 1, 1),
    (1, 1, 1024, 1024, 1, 0, 0), (1, 1, 1024, 1024, 0, 0, 1), (2, 1, 1024, 1024, 1, 0, 1), (96, 1, 2048, 64, 1, 0, 1), (3, 8, 1, 64, 0, 1, 0)])
def test_matmul_dispatch(b, m, n, k, tb, f32, batched):
    """both sides of the measured figures beside the rule"""
    lib = fake_gpu.load()
    dts = (F, F) if f32 else ((I, U) if 1 in (m, n) else (U, I))
    assert matmul_route(lib, b, m, n, k, 0, tb, *dts) == (B.SUCCESS, bool(batched))
    # a captured stream: operands whose scale the host cannot wait for stay with the batched kernels where these exist
    lib.fake_capture(1)
    code, took = matmul_route(lib, b, m, n, k, 0, tb, *dts)
    lib.fake_capture(0)
    if f32 and n != 1:
        assert (code, took) == (B.SUCCESS, True)
    elif not f32:
        assert (code, took) == (B.SUCCESS, bool(batched))
    else:
        assert code == B.UNKNOWN


def test_matmul_dispatch_of_operands_that_tma_cannot_fetch():
    lib = fake_gpu.load()
    route = lambda *a, **kw: matmul_route(lib, *a, **kw)[1]
    assert not route(1, 136, 36, 25084, 0, 0, F, F) and route(3, 12, 7, 5708, 0, 1, F, F)        # K off the 16-byte grid
    assert route(1, 87, 9, 20897, 1, 0, F, F) and not route(2, 1860, 4, 7664, 1, 1, F, I)        # A stored [K][M]
    assert not route(1, 64, 64, 4096, 0, 1, U, I) and route(1, 64, 64, 4096, 0, 1, U, I, a_at=(1 << 20) + 4)


def test_a_reported_error_does_not_stay_in_the_thread():
    """a launch that is refused fails its own call, and not the next one as well"""
    lib = fake_gpu.load()
    for call in (lambda: gemm_codes(lib, 8, 64, 64, False), lambda: gemm_codes(lib, 256, 64, 64, False),
                 lambda: [matmul_code(lib, (2, 4, 16), (2, 16, 8), (2, 4, 8))[0]]):
        lib.fake_refuse_programmatic(1)
        lib.fake_capture(1)                  # (no second try while a stream is captured)
        assert B.SUCCESS not in call() and lib.fake_last_error() == 0
        lib.fake_refuse_programmatic(0)
        lib.fake_capture(0)
        assert set(call()) == {B.SUCCESS}
    x, q, s = np.zeros(64, np.uint8), np.zeros(64, np.uint8), (C.c_float * 1)(-1.0)
    d, o = B.tensor1d(U, 64), B.tensor1d(I, 64)
    assert lib.quantize_cuda_b200(C.byref(d), C.c_void_p(x.ctypes.data), C.byref(o), C.c_void_p(q.ctypes.data), s, 0) == B.SUCCESS
