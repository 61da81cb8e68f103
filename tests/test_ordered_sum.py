"""The filter maker's threaded sum (ordered_sum.hpp) on the host: the value of a loop, bit for
bit, whatever number of threads starts."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("sum") / "libsum.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-pthread",
                    "-I" + os.path.join(ROOT, "biobloom_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "ordered_sum_model.cpp"), "-o", out],
                   check=True)
    fn = ctypes.CDLL(out).model_ordered_sum
    fn.restype = ctypes.c_double
    fn.argtypes = [ctypes.c_uint64, ctypes.c_uint64, ctypes.c_double, ctypes.c_uint, ctypes.c_int]
    return fn


@pytest.mark.parametrize("n", [0, 1, 1023, 2047, 2048, 8191, 8192, 100003])
@pytest.mark.parametrize("start", [0, 1, 3, 7])
def test_threads_that_do_not_start(model, n, start):
    one = model(1, 1 + n, 0.25, 1, 0)
    assert model(1, 1 + n, 0.25, 8, start) == one
