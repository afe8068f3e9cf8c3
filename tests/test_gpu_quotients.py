"""The ghost fill's quotients are those of IEEE division, zeros and subnormal results included."""
import os
import subprocess

import pytest
from nlos_lbm import build

pytestmark = pytest.mark.gpu


@pytest.mark.skipif(not os.path.exists(build.NVCC), reason="no nvcc")
def test_quotients_equal_division(tmp_path, gpu):
    exe = str(tmp_path / "check_quotients")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cpp", "check_quotients.cu")
    r = subprocess.run([build.NVCC, *build.ARCH, "-O3", "-std=c++17", "-ccbin", build.CXX, "-I" + build.INCLUDE,
                        "-I" + build.CSRC, src, "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.stdout.split() == ["ok", "0", "0", "0", "0"], r.stdout + r.stderr
