"""The multiply-add of the integer sums on the device, with factors that are words of its own
accumulator: exact in 64 bits."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "chorus-mhd_gb300", "csrc")


@pytest.mark.gpu
def test_factors_that_are_words_of_the_accumulator(tmp_path):
    nvcc = next((p for p in ("/usr/local/cuda/bin/nvcc", shutil.which("nvcc")) if p and os.path.exists(p)), None)
    if nvcc is None:
        pytest.skip("no nvcc")
    lib = str(tmp_path / "mad.so")
    r = subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                        "-I" + CSRC, os.path.join(HERE, "fixdot", "mad_device.cu"), "-o", lib], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    rng = np.random.default_rng(0)
    n = 1000
    a, b = rng.integers(-2 ** 30, 2 ** 30, (2, n)).astype(np.int32)
    a[:4], b[:4] = [0, -1, 2 ** 30, -2 ** 30], [0, 1, -2 ** 30, -2 ** 30]
    out = np.empty((n, 4), np.int64)
    p = lambda x, t: x.ctypes.data_as(ctypes.POINTER(t))  # noqa: E731
    rc = ctypes.CDLL(lib).mad_run(n, p(a, ctypes.c_int), p(b, ctypes.c_int), p(out, ctypes.c_longlong))
    assert rc == 0
    x, y = a.astype(np.int64), b.astype(np.int64)
    xy = (y << 32) + (x & 0xffffffff)
    want = np.stack([xy + x * y, xy + x * y, (x & 0xffffffff) + x * x, x + x * y], 1)
    assert np.array_equal(out, want)
