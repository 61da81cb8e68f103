"""The lane kernel's walks and its bit reduction (lane_walk.cuh), compiled for
the host, against the oracle: decisions, counts of algorithmic probes and
scores of random reads under the four scoring methods, in steps of 2, 4 and 8
frames; word indexes against the 64-bit remainder."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from tests import oracle_lib as ol

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("model") / "lane_model.so")
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", "-I", os.path.join(ROOT, "biobloom_b200",
                    "csrc"), "-I", os.path.join(ROOT, "oracle"), "-o", out,
                    os.path.join(ROOT, "tests", "native", "lane_model.cpp"),
                    os.path.join(ROOT, "oracle", "bbt_oracle.c")], check=True)
    m = ctypes.CDLL(out)
    m.lane_eval.argtypes = [ctypes.c_char_p, ctypes.c_uint64, ctypes.POINTER(ol._BF),
                            ctypes.c_double, ctypes.c_uint, ctypes.c_int, ctypes.c_int,
                            ctypes.POINTER(ctypes.c_uint64)]
    m.lane_score.restype = ctypes.c_double
    m.lane_score.argtypes = [ctypes.c_char_p, ctypes.c_uint64, ctypes.POINTER(ol._BF),
                             ctypes.c_int, ctypes.c_uint, ctypes.c_double]
    m.lane_word_errors.restype = ctypes.c_uint64
    m.lane_word_errors.argtypes = [ctypes.c_void_p, ctypes.c_uint64, ctypes.c_uint32]
    return m


def _cases(seed, trials, reads):
    """Filters of random fill and reads of their sequence or of random bases,
    with substitutions, runs that are not ACGT and lower case; k up to 32."""
    rng = np.random.default_rng(seed)
    L = ol.lib()
    acgt = np.frombuffer(b"ACGT", dtype=np.uint8)
    for _ in range(trials):
        h = int(rng.integers(1, 6))
        k = max(h, int(rng.integers(3, 33)))
        f = ol.Filter.create(64 * int(rng.integers(1, 60)), h, k)
        g = rng.choice(acgt, 3000)
        fill = rng.random()
        for _, hv in ol.kmers(g.tobytes(), h, k):
            if rng.random() < fill:
                L.oracle_bf_insert(ctypes.byref(f.bf), (ctypes.c_uint64 * 64)(*hv))
        for _ in range(reads):
            n, st = int(rng.integers(0, 400)), int(rng.integers(0, 2600))
            s = (g[st:st + n] if rng.random() < 0.6 else rng.choice(acgt, n)).copy()
            m = rng.random(n) < rng.random() * 0.05
            s[m] = rng.choice(acgt, m.sum())
            if rng.random() < 0.3:
                m = rng.random(n) < rng.random() * 0.2
                s[m] = np.frombuffer(b"NnRX", dtype=np.uint8)[rng.integers(0, 4, m.sum())]
            if rng.random() < 0.2:
                s = np.where(rng.random(n) < 0.3, s | 0x20, s).astype(np.uint8)
            streak = int(rng.integers(1, 6)) if rng.random() > 0.05 else int(rng.integers(30, 80))
            yield rng, L, f, s.tobytes(), streak


@pytest.mark.parametrize("seed", range(4))
def test_decisions_and_probe_counts_match_oracle(model, seed):
    for rng, L, f, b, streak in _cases(300 + seed, 30, 60):
        bf = ctypes.byref(f.bf)
        thr = float(rng.integers(0, 3)) * 0.5 if rng.random() < 0.2 else float(rng.random())
        length = int(rng.integers(2, 60))
        minus = 10.0 ** (-float(rng.uniform(1, 100)) / 10.0)
        fpr = L.oracle_bf_fpr(bf)
        for mode, t, run in (
                (ol.SIMPLE, thr, lambda c: L.oracle_eval_simple(b, len(b), bf, thr, streak, c)),
                (ol.HARMONIC, thr,
                 lambda c: L.oracle_eval_harmonic(b, len(b), bf, thr, streak, c)),
                (ol.LENGTH, float(length),
                 lambda c: L.oracle_eval_min_match_len(b, len(b), bf, length, c)),
                (ol.BINOMIAL, minus,
                 lambda c: L.oracle_eval_binomial(b, len(b), bf, minus, fpr, streak, c))):
            c = ctypes.c_uint64(0)
            want = run(ctypes.byref(c))
            for n in (2, 4, 8):
                a = ctypes.c_uint64(0)
                got = model.lane_eval(b, len(b), bf, t, streak, mode, n, ctypes.byref(a))
                assert (got, a.value) == (want, c.value), (mode, n, t, streak, f.k, f.h, b)


@pytest.mark.parametrize("seed", range(3))
def test_scores_match_oracle(model, seed):
    for rng, L, f, b, streak in _cases(400 + seed, 25, 40):
        bf = ctypes.byref(f.bf)
        fpr = L.oracle_bf_fpr(bf)
        for mode in (ol.SIMPLE, ol.LENGTH, ol.HARMONIC, ol.BINOMIAL):
            want = L.oracle_eval_score(b, len(b), bf, mode, streak, fpr)
            got = model.lane_score(b, len(b), bf, mode, streak, fpr)
            assert np.float64(want).view(np.uint64) == np.float64(got).view(np.uint64), (mode, b)


@pytest.mark.parametrize("m5", [2, 4, 6, 10, 62, 64, 66, 855_062, 2**23 - 2, 2**23, 8_563_202,
                                530_000_006, 2**29 + 2, 2**30 - 2])
def test_word_index_is_the_64_bit_remainder(model, m5):
    rng = np.random.default_rng(m5)
    m = 32 * m5
    v = rng.integers(0, 2**64, 200_000, dtype=np.uint64)
    # multiples of the modulus and their neighbours, up to the largest value
    q = rng.integers(0, (2**64 - 1) // m + 1, 50_000, dtype=np.uint64) * np.uint64(m)
    top = np.uint64((2**64 - 1) // m * m)
    v = np.concatenate([v, q, q + np.uint64(m - 1), q - np.uint64(1), q + np.uint64(1),
                        np.array([0, 1, 63, 64, m - 1, m, 2**64 - 1, top, top - np.uint64(1)],
                                 dtype=np.uint64)])
    v = np.ascontiguousarray(v)
    assert model.lane_word_errors(v.ctypes.data, len(v), m5) == 0
