"""The filter maker on sequences that do not stay on the device: more than 256 Mbp in all,
one of them longer than a chunk."""
import numpy as np
import pytest

from tests import oracle_lib as ol
from tests.test_lane_gpu import ACGT

pytestmark = pytest.mark.gpu


def test_sequences_in_chunks(tmp_path):
    from biobloom_b200 import synth
    rng = np.random.default_rng(9)
    chunk = 256 << 20
    long = ACGT[rng.integers(0, 4, chunk + 5000, dtype=np.uint8)]
    long[chunk - 3:chunk + 2] = ord("N")  # around the chunk's end
    seqs = [ACGT[rng.integers(0, 4, 3000, dtype=np.uint8)], long, long[chunk - 1000:chunk + 1500].copy()]
    k, fpr, h = 25, 0.4, 1
    synth.make_filter(seqs, str(tmp_path / "g"), "g", k=k, fpr=fpr, hash_num=h)
    want = ol.make_filter_par(seqs, k=k, fpr=fpr, h=h)
    want.store(str(tmp_path / "o.bf"))
    got_bits, want_bits = ((tmp_path / f).read_bytes().split(b"[HeaderEnd]\n", 1)[1]
                           for f in ("g.bf", "o.bf"))
    assert got_bits == want_bits
    info = dict(line.split("=", 1) for line in (tmp_path / "g.txt").read_text().splitlines()
                if "=" in line)
    frames = 0
    for s in seqs:
        bad = np.concatenate([[-1], np.flatnonzero(s == ord("N")), [len(s)]])
        frames += int(np.maximum(np.diff(bad) - 1 - k + 1, 0).sum())
    new, again = int(info["num_entries"]), int(info["redundant_sequences"])
    assert new + again == frames
    # one hash: a k-mer is new when it is the first of its bit
    assert new == int(np.bitwise_count(np.frombuffer(got_bits, dtype=np.uint8)).sum())
