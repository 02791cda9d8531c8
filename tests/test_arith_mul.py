"""The FP64 product on the integer pipe returns the multiplication instruction's
result: tests/arith/mul_check.cu compares it with that instruction and the host's
product over about 3.5 million operand pairs (GPU); it compiles for sm_103a here
(CPU)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
SRC = os.path.join(HERE, "arith", "mul_check.cu")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


def _compile(out, *extra):
    subprocess.run([NVCC, "-std=c++17", "-O2", "--fmad=false", "-gencode", "arch=compute_103a,code=sm_103a",
                    "-I", os.path.join(ROOT, "mom5_gb300", "csrc"), *extra, SRC, "-o", out], check=True)


@pytest.mark.skipif(not os.path.exists(NVCC), reason="nvcc not found")
def test_product_check_compiles(tmp_path):
    _compile(str(tmp_path / "mul_check.o"), "-c")


@pytest.mark.gpu
def test_products_on_the_integer_pipe_are_exact(tmp_path):
    exe = str(tmp_path / "mul_check")
    _compile(exe)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
