"""No kernel of the adjoint keeps a copy of its arguments on the stack: an argument structure that is assigned to
and indexed at run time is copied to local memory by every thread before its first useful load.  What ptxas
reports when the source is compiled."""
import os
import re
import subprocess

import pytest
from nlos_lbm import build

FRAME = 64   # bytes; the argument structures start at some 150


@pytest.mark.skipif(not os.path.exists(build.NVCC), reason="no nvcc")
def test_adjoint_kernels_do_not_copy_their_arguments(tmp_path):
    r = subprocess.run([build.NVCC, *build.ARCH, "-O3", "-std=c++17", "-ccbin", build.CXX, "-Xptxas=-v",
                        "-I" + build.INCLUDE, "-I" + build.CSRC, "-c", os.path.join(build.CSRC, "adjoint.cu"), "-o",
                        str(tmp_path / "adjoint.o")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    frames = re.findall(r"Function properties for (\S+)\s+(\d+) bytes stack frame", r.stderr)
    assert len(frames) >= 5
    assert not {n: int(b) for n, b in frames if int(b) > FRAME}
