"""Pass 0 of the masking kernel (dust_may_mask): a read that it leaves out has no
masked interval in the oracle, and ordinary random reads are mostly left out."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from tests import oracle_lib as ol
from tests.test_dust_model import _sequences

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def may(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("dust") / "dust_may.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "biobloom_b200", "csrc"), "-o", out,
                    os.path.join(ROOT, "tests", "native", "dust_may_model.cpp")], check=True)
    f = ctypes.CDLL(out).model_may_mask
    f.argtypes = [ctypes.c_char_p, ctypes.c_uint64, ctypes.c_int, ctypes.c_int]
    return f


@pytest.mark.parametrize("T,W", [(20, 64), (10, 16), (30, 32), (0, 8), (20, 3), (5, 128),
                                 (100, 64), (20, 1024)])
def test_reads_left_out_have_no_masked_interval(may, T, W):
    rng = np.random.default_rng(T * 2000 + W)
    acgt = np.frombuffer(b"ACGT", dtype=np.uint8)
    reads = _sequences(W, 150, 900) + [rng.choice(acgt, int(n)).tobytes()
                                       for n in rng.integers(0, 400, 300)] + [b"", b"AC", b"ACG"]
    for s in reads:
        if not may(s, len(s), T, W):
            assert ol.sdust(s, T, W)[0] == []


def test_most_random_reads_are_left_out(may):
    rng = np.random.default_rng(8)
    acgt = np.frombuffer(b"ACGT", dtype=np.uint8)
    n = sum(bool(may(s, len(s), 20, 64))
            for s in (rng.choice(acgt, 150).tobytes() for _ in range(2000)))
    assert n < 300
