"""The 2-D temporally blocked kernels keep their chunks and exchange pairs in
registers: the compiler reports no spills for any of them."""
import os
import re
import subprocess

import pytest


def test_no_spills(tmp_path):
    from thesis_gb300 import build
    nvcc = build.nvcc()
    try:
        subprocess.run([nvcc, "--version"], check=True, capture_output=True)
    except OSError:
        pytest.skip("no nvcc")
    r = subprocess.run([nvcc] + build.ARCH + build.NVCC_FLAGS + ["-Xptxas", "-v", "-c", os.path.join(build.CSRC, "k_tb2d.cu"),
                                                                 "-o", str(tmp_path / "x.o")], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    kernels = re.findall(r"entry function '(\w*k_tb2d\w*)'.*?(\d+) bytes spill stores, (\d+) bytes spill loads", r.stderr, re.S)
    assert len(kernels) >= 24
    assert [k for k in kernels if k[1:] != ("0", "0")] == []
