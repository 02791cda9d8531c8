"""Half, double, quarter and the product by a mask, formed on the integer pipe, return
the multiplication instruction's result: tests/arith/shortcut_check.cu compares them
over every exponent field, subnormals around ties and random bit patterns (GPU); it
compiles for sm_103a here (CPU)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
SRC = os.path.join(HERE, "arith", "shortcut_check.cu")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


def _compile(out, *extra):
    subprocess.run([NVCC, "-std=c++17", "-O2", "--fmad=false", "-gencode", "arch=compute_103a,code=sm_103a",
                    "-I", os.path.join(ROOT, "mom5_gb300", "csrc"), "-I", os.path.join(ROOT, "include"), *extra, SRC,
                    "-o", out], check=True)


@pytest.mark.skipif(not os.path.exists(NVCC), reason="nvcc not found")
def test_shortcut_check_compiles(tmp_path):
    _compile(str(tmp_path / "shortcut_check.o"), "-c")


@pytest.mark.gpu
def test_shortcuts_are_exact(tmp_path):
    exe = str(tmp_path / "shortcut_check")
    _compile(exe)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
