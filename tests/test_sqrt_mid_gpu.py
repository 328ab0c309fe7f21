"""The warp pass's branchless square root on the device (GPU): every float of
its range against the rounded square root, bit for bit."""
import ctypes
import os
import subprocess

import pytest

from massccs_b200 import build as B

pytestmark = pytest.mark.gpu


def test_every_float_of_the_range_has_the_rounded_root(tmp_path):
    so = str(tmp_path / "sqrt_mid_probe.so")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "sqrt_mid_probe.cu")
    subprocess.run([B._nvcc()] + B.ARCH + B.NVCC_FLAGS + ["-I", B.CSRC, "-shared", "-o", so, src], check=True)
    lib = ctypes.CDLL(so)
    lib.sqrt_mid_mismatches.argtypes = [ctypes.c_float, ctypes.c_float, ctypes.c_void_p, ctypes.c_void_p]
    count, first = ctypes.c_ulonglong(1), ctypes.c_float()
    assert lib.sqrt_mid_mismatches(1e-18, 1e18, ctypes.byref(count), ctypes.byref(first)) == 0
    assert count.value == 0, (count.value, first.value)
