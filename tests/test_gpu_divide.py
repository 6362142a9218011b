"""csrc/rrtmg_divide.cuh against IEEE division, bit for bit: the reciprocal of
every binary32 significand at all exponents of its range, and some 1.5e9
quotients with operands chosen next to the hard cases and at the ends of their
ranges; and the shortwave layer optics that use it against their general form."""

from __future__ import annotations

import ctypes
import shutil
import subprocess

import pytest

from conftest import REPO

pytestmark = pytest.mark.gpu


def _compile(tmp_path, source, *flags):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not shutil.which(nvcc):
        pytest.skip("no nvcc")
    so = tmp_path / (source + ".so")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-fmad=false",
                    "-prec-div=true", "-prec-sqrt=true", "-ftz=false", *flags, "-shared", "-Xcompiler",
                    "-fPIC,-ffp-contract=off", "-I", str(REPO / "wrf-jax_b200" / "csrc"), str(REPO / "tests" / source),
                    "-o", str(so), "-lcudart"], check=True)
    return ctypes.CDLL(str(so))


def test_reciprocals_and_quotients_equal_ieee_division(pkg, tmp_path):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    divide_check = _compile(tmp_path, "divide_check.cu").divide_check
    torch.cuda.synchronize()
    bad = (ctypes.c_ulonglong * 2)()
    assert divide_check(-100, 101, 4096, bad) == 0
    assert list(bad) == [0, 0]


@pytest.mark.parametrize("ends", [0, 1], ids=["ordinary", "ends"])
def test_sw_layers_equal_their_general_form(pkg, tmp_path, ends):
    """The shortwave layer optics that check their operands once against the
    general form, bit for bit (any NaN for a NaN, any zero for a zero): optical
    depths, cosines and cloud optics as they occur, and up to and beyond the
    ends of what the checked form accepts, zeros and infinities among them."""
    import numpy as np
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    check = _compile(tmp_path, "sw_layer_check.cu", "--expt-relaxed-constexpr").sw_layer_check
    ntbl, bpade = 10000, 1.0 / 0.278
    x = np.arange(ntbl + 1) / ntbl
    with np.errstate(divide="ignore"):
        table = np.maximum(np.exp(-np.where(x < 1.0, bpade * x / (1.0 - x), np.inf)), 1.0e-20).astype(np.float32)
    torch.cuda.synchronize()
    bad = (ctypes.c_ulonglong * 2)()
    assert check(ntbl, table.ctypes.data_as(ctypes.c_void_p), ctypes.c_float(bpade), 256, ends, bad) == 0
    assert list(bad) == [0, 0]
