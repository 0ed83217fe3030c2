"""Registers of kernels whose launch shape rests on them, from the compiler's report:
the general initial partition runs two blocks of 1,024 threads per SM, which leaves
32 registers a thread, and spilling there costs it 8 % (its sweeps are bound by
latency)."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "thegraphpartitioning_b200", "csrc")


def test_general_initial_partition_does_not_spill(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    r = subprocess.run([nvcc, "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-Xcompiler",
                        "-fPIC", "--expt-relaxed-constexpr", "-Xptxas", "-v", "-c", "gp_initpart.cu", "-o",
                        str(tmp_path / "x.o")], cwd=CSRC, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    m = re.search(r"k_initpartEN.*?(\d+) bytes spill stores, (\d+) bytes spill loads.*?Used (\d+) registers", r.stderr,
                  re.S)
    assert m, r.stderr[-2000:]
    stores, loads, regs = map(int, m.groups())
    assert stores == loads == 0 and regs <= 32
