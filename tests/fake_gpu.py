"""The library's own host code without a GPU: its built objects linked against native/fake_cudart.cpp, which records launches and
runs none.  What a call refuses, which kernels it launches and what it leaves behind can then be seen on the CPU."""
import ctypes as C
import os
import subprocess
import tempfile

import bolt_b200 as B
from bolt_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))
_lib = None


def fresh():
    """a copy of its own, which no call has used yet"""
    build.build()
    objs = [os.path.join(build.OBJ_DIR, os.path.basename(s)[:-3] + ".o") for s in build.sources()]
    with tempfile.TemporaryDirectory() as d:
        so = os.path.join(d, "libbolt_b200_fake.so")
        cmd = [build._nvcc(), "-shared", "-std=c++17", "-Xcompiler", "-fPIC", "-cudart", "none", "-Xlinker", "-Bsymbolic", "-o", so,
               os.path.join(HERE, "native", "fake_cudart.cpp")] + objs
        r = subprocess.run(cmd, capture_output=True, text=True)
        assert r.returncode == 0, r.stderr
        lib = C.CDLL(so)
    for name, (res, args) in B.SIGNATURES.items():
        fn = getattr(lib, name)
        fn.restype, fn.argtypes = res, args
    lib.fake_launch_name.restype = C.c_char_p
    lib.fake_max_words.restype = C.c_void_p
    lib.bolt_b200_set_pointer_mode(1)
    return lib


def load():
    global _lib
    if _lib is None:
        _lib = fresh()
    _lib.fake_refuse_programmatic(0)
    _lib.fake_capture(0)
    _lib.fake_set_last_error(0)
    _lib.fake_forget_launches()
    return _lib


def launches(lib):
    return [lib.fake_launch_name(i).decode() for i in range(lib.fake_launches())]
