"""Kernels keep their registers: the compiler's resource report (-Xptxas -v) shows
no spill in any kernel of the library, built with the library's own flags."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "tensorkyber_b200", "csrc")


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="no nvcc")
@pytest.mark.parametrize("src", ["tk_tc5.cu", "tk_pack.cu", "tk_ntt_mma.cu", "tk_matvec.cu"])
def test_no_kernel_spills(src):
    p = subprocess.run(["nvcc", "-O3", "-std=c++17", "-lineinfo", "-gencode",
                        "arch=compute_100a,code=sm_100a", "-Xptxas", "-v", "-cubin",
                        "-o", os.devnull, os.path.join(CSRC, src)],
                       capture_output=True, text=True)
    assert p.returncode == 0, p.stderr[-3000:]
    found = re.findall(r"Function properties for (\S+)\s+\d+ bytes stack frame, "
                       r"(\d+) bytes spill stores, (\d+) bytes spill loads", p.stderr)
    assert found
    assert [f for f in found if int(f[1]) or int(f[2])] == []
