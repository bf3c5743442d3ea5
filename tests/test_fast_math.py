"""The routines that stand for a general one in the fast paths, over their
whole argument ranges on the device: exponential and logarithm without special
cases, and quotients by a reciprocal with exact corrections."""
import ctypes as C
import os
import subprocess

import pytest

from hw_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.gpu
def test_fast_routines_equal_the_general_ones(tmp_path):
    lib = str(tmp_path / "libfast_math_sweep.so")
    subprocess.run([build.NVCC] + build.NVCC_FLAGS + ["-shared", "-o", lib, os.path.join(HERE, "fast_math_sweep.cu")],
                   check=True)
    counts = (C.c_ulonglong * 4)(*[1] * 4)
    assert C.CDLL(lib).fast_math_sweep(counts) == 0
    assert dict(zip(("exp", "log", "tenth", "bin"), counts)) == {"exp": 0, "log": 0, "tenth": 0, "bin": 0}
