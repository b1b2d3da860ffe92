"""The pool behind the calls that wait for a maximum, compiled for the host against a fake CUDA runtime: a mail whose kernel
has not reported must not reach another call, and a failed device must not make later calls wait for ever."""
import os
import subprocess

from bolt_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))


def test_mails_come_back_only_when_their_kernel_is_done(tmp_path):
    exe = str(tmp_path / "max_mail")
    srcs = [os.path.join(HERE, "native", "max_mail_harness.cu"), os.path.join(HERE, "native", "fake_cudart.cpp"), os.path.join(build.CSRC, "max_mail.cu")]
    cmd = [build._nvcc(), "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "-cudart", "none", "-I", os.path.join(build.ROOT, "include"),
           "-I", build.CSRC, "-o", exe] + srcs + ["-lpthread"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout
