"""The FP64 division where its proof has no slack: tests/arith/div_edges_check.cu
compares it with the division instruction for every pattern of a divisor's leading
bits under every reciprocal within the error bound the proof takes, and at the edges
of its exponent range (GPU); it compiles for sm_103a here (CPU)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
SRC = os.path.join(HERE, "arith", "div_edges_check.cu")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


def _compile(out, *extra):
    subprocess.run([NVCC, "-std=c++17", "-O2", "--fmad=false", "-gencode", "arch=compute_103a,code=sm_103a",
                    "-I", os.path.join(ROOT, "mom5_gb300", "csrc"), *extra, SRC, "-o", out], check=True)


@pytest.mark.skipif(not os.path.exists(NVCC), reason="nvcc not found")
def test_division_edges_check_compiles(tmp_path):
    _compile(str(tmp_path / "div_edges_check.o"), "-c")


@pytest.mark.gpu
def test_division_edges_are_exact(tmp_path):
    exe = str(tmp_path / "div_edges_check")
    _compile(exe)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
