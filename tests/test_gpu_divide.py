"""csrc/rrtmg_divide.cuh against IEEE division, bit for bit: the reciprocal of
every binary32 significand at all exponents of its range, and 2.5e9 quotients
with operands chosen next to the hard cases."""

from __future__ import annotations

import ctypes
import shutil
import subprocess

import pytest

from conftest import REPO

pytestmark = pytest.mark.gpu


def test_reciprocals_and_quotients_equal_ieee_division(pkg, tmp_path):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    so = tmp_path / "divide_check.so"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-fmad=false",
                    "-prec-div=true", "-ftz=false", "-shared", "-Xcompiler", "-fPIC",
                    "-I", str(REPO / "wrf-jax_b200" / "csrc"), str(REPO / "tests" / "divide_check.cu"), "-o", str(so),
                    "-lcudart"], check=True)
    torch.cuda.synchronize()
    bad = (ctypes.c_ulonglong * 2)()
    assert ctypes.CDLL(str(so)).divide_check(-100, 101, 4096, bad) == 0
    assert list(bad) == [0, 0]
