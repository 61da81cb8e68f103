"""Calls on torch's default stream come after what that stream was given before, and before
what it is given afterwards."""
import numpy as np
import pytest

from tests import oracle_lib as ol
from tests.test_lane_gpu import ACGT, _device, _filters, _open

pytestmark = pytest.mark.gpu


def _same_lengths(rng, genome):
    a = [genome[i:i + 100].tobytes() for i in range(500)]
    b = [rng.choice(ACGT, 100).tobytes() for _ in range(500)]
    return a, b


def test_bloom_filters(tmp_path):
    import torch
    rng = np.random.default_rng(1)
    genomes, filters, paths = _filters(tmp_path, rng, [25], 3)
    a, b = _same_lengths(rng, genomes[0])
    want, _ = ol.classify(*ol.pack_reads(a), filters, 0.15, 3)
    (seq_a, off), (seq, _) = _device(a), _device(b)
    with _open(paths, ol.SIMPLE, 0.15, 3) as bbc:
        bbc.classify_device(seq, off)  # loads the kernels
        torch.cuda.synchronize()
        torch.cuda._sleep(20_000_000)
        seq.copy_(seq_a)
        hits = bbc.classify_device(seq, off)[0].clone()
        torch.cuda.synchronize()
        assert np.array_equal(hits.cpu().numpy().view(np.uint64), want)


def test_multi_index_filter(tmp_path):
    import torch
    from biobloom_b200.mibf import MIBFClassifier
    rng = np.random.default_rng(2)
    genome = rng.choice(ACGT, 5000)
    f = ol.MIBF.build([genome.tobytes(), rng.choice(ACGT, 5000).tobytes()], [1, 2], k=25, h=3,
                      occupancy=0.5)
    f.store(str(tmp_path / "x"))
    (tmp_path / "x_ids.txt").write_text("1\ta\n2\tb\n")
    a, b = _same_lengths(rng, genome)
    (seq_a, off), (seq, _) = _device(a), _device(b)
    c = MIBFClassifier(str(tmp_path / "x.bf"))
    c.classify_device(seq, off)
    torch.cuda.synchronize()
    torch.cuda._sleep(20_000_000)
    seq.copy_(seq_a)
    hits, n, _ = (t.clone() for t in c.classify_device(seq, off))
    torch.cuda.synchronize()
    assert (n == 1).all() and (hits[:, 0, 0] == 1).all()
    c.close()
