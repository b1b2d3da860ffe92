"""Several host threads, each with a stream of its own, through the calls whose scale is found on the device: the reported
maxima and the shared pool behind them must not mix.  Every thread's bytes and scales against its own serial run."""
import ctypes as C
import os
import sys
import threading

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(__file__))
import bolt_b200 as B  # noqa: E402
from bolt_b200 import synth  # noqa: E402
from test_conv_gpu import conv_gpu  # noqa: E402
from test_stack_gpu import make_stack  # noqa: E402

pytestmark = pytest.mark.gpu
THREADS, ROUNDS = 70, 12     # more threads than the pool has entries


class Work:
    def __init__(self, t):
        import torch

        self.n = 1000 + 517 * t
        self.x = torch.from_numpy((synth.normal(t, (self.n,)) * np.float32(0.1 + t)).astype(np.float32)).cuda()
        self.acc = torch.from_numpy(synth.integers(t + 500, (self.n,), -1000 * (t + 1), 1000 * (t + 1)).astype(np.int32)).cuda()
        self.q, self.r = (torch.empty(self.n, dtype=torch.uint8, device="cuda") for _ in range(2))
        self.a = torch.from_numpy(synth.normal(t + 900, (2, 24, 32)) * np.float32(1 + t)).cuda()
        self.b = torch.from_numpy(synth.normal(t + 901, (2, 32, 40))).cuda()
        self.c = torch.empty((2, 24, 40), dtype=torch.uint8, device="cuda")
        ad, bd = B.tensor_nd(B.DT_F32, (2, 24, 32)), B.tensor_nd(B.DT_F32, (2, 32, 40))
        cd = B.matmul_infer_output_size(ad, 0, bd, 0)
        cd.dt = B.DT_U8_Q
        self.nb = B.matmul_infer_forward_tmp_bytes(ad, 0, bd, 0, cd, -1.0)
        self.tmp = torch.empty(self.nb, dtype=torch.uint8, device="cuda")
        self.ad, self.bd, self.cd = ad, bd, cd
        self.conv = (1, 16, 6, 6, 16 + 8 * (t % 4), 3, 3, 1, 1)
        oc = self.conv[4]
        self.cx, self.cw = synth.u8(t + 1000, (1, 1, 6, 6, 16)), synth.s8(t + 1100, (oc, 16, 3, 3)) // np.int8(1 + t % 7)
        self.cb = synth.normal(t + 1200, (oc,))

    def run(self):
        p = lambda t: C.c_void_p(t.data_ptr())
        sq, sr = [-1.0], [-1.0, 40.0]
        B.quantize(B.tensor1d(B.DT_F32, self.n), p(self.x), B.tensor1d(B.DT_U8_Q, self.n), p(self.q), sq)
        B.quantize(B.tensor1d(B.DT_I32, self.n), p(self.acc), B.tensor1d(B.DT_U8_Q, self.n), p(self.r), sr)
        sm = B.matmul(self.ad, 0, p(self.a), -1.0, self.bd, 0, p(self.b), -1.0, None, None, self.nb, p(self.tmp), self.cd, p(self.c), -1.0)
        conv, sc, _ = conv_gpu(self.conv, self.cx, self.cw, self.cb, 16, True, True, [31.75, -1.0, 640.0])
        B.CHECK_STATUS(B.lib().bolt_b200_synchronize(), "synchronize")
        return (conv.tobytes(), sc[1], sq[0], sr[0], float(sm), self.q.cpu().numpy().tobytes(), self.r.cpu().numpy().tobytes(), self.c.cpu().numpy().tobytes())


def test_threads_and_streams_do_not_mix():
    import torch

    works = [Work(t) for t in range(THREADS)]
    expect = [w.run() for w in works]
    torch.cuda.synchronize()
    bad = []

    def body(t):
        st = torch.cuda.Stream()
        with torch.cuda.stream(st):
            B.CHECK_STATUS(B.lib().bolt_b200_set_stream(C.c_void_p(st.cuda_stream)))
            for i in range(ROUNDS):
                if works[t].run() != expect[t]:
                    bad.append((t, i))
            B.CHECK_STATUS(B.lib().bolt_b200_set_stream(None))

    ts = [threading.Thread(target=body, args=(t,)) for t in range(THREADS)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad, bad[:10]


def test_stacks_on_streams_do_not_mix():
    """The device-resident input scale: stacks whose inputs differ by orders of magnitude, each on a stream of its own."""
    import torch

    stacks, expect = [], []
    for t in range(4):
        st, _ = make_stack(48, [512, 256, 64], False, 300 + 10 * t)
        st.x_dev.copy_(torch.from_numpy((synth.normal(400 + t, (48 * 512,)) * np.float32(10.0 ** (2 * t - 3))).astype(np.float32)))
        st.calibrate()
        st.step()
        B.CHECK_STATUS(B.lib().bolt_b200_synchronize(), "synchronize")
        stacks.append(st)
        expect.append((st.d_scale[:1].clone(), st.out_dev.clone()))
    torch.cuda.synchronize()
    bad = []

    def body(t):
        st, (scale, out) = stacks[t], expect[t]
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            B.CHECK_STATUS(B.lib().bolt_b200_set_stream(C.c_void_p(stream.cuda_stream)))
            for i in range(200):
                st.step()
                if i % 10 == 9:
                    stream.synchronize()
                    if not (torch.equal(st.d_scale[:1], scale) and torch.equal(st.out_dev, out)):
                        bad.append((t, i))
            B.CHECK_STATUS(B.lib().bolt_b200_set_stream(None))

    ts = [threading.Thread(target=body, args=(t,)) for t in range(len(stacks))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad, bad[:10]
