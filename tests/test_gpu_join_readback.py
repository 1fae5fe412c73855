"""Values of a residual block read back through the op graph (join_readback.cc, run as a child process)."""
import os
import subprocess

import pytest

from tests.conftest import ROOT

pytestmark = pytest.mark.gpu
PKG = os.path.join(ROOT, "arraydiff_cuda_b200")


def test_a_convolution_that_writes_a_sum_reads_back_as_itself(tmp_path):
    cuda, exe = os.environ.get("CUDA_HOME", "/usr/local/cuda"), str(tmp_path / "join_readback")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-I", os.path.join(PKG, "host", "include"), "-I", os.path.join(ROOT, "include"),
                           "-I", os.path.join(cuda, "include"), os.path.join(ROOT, "tests", "join_readback.cc"), "-o", exe, "-L", PKG, "-larraydiff_host",
                           "-larraydiff_b200", "-L", os.path.join(cuda, "lib64"), "-lcudart", "-Wl,-rpath," + PKG])
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout == "ok\n", out.stdout + out.stderr
