"""The warp kernel at the length from which it takes a read in windows of 256 frames: hits
and probe counts against the oracle on both sides of it."""
import numpy as np
import pytest

from tests import oracle_lib as ol
from tests.test_lane_gpu import ACGT, _device, _filters, _open

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ks,scoring,score", [([25], ol.SIMPLE, 0.15), ([25, 31], ol.SIMPLE, 0.7),
                                              ([25], ol.HARMONIC, 0.15), ([21], ol.LENGTH, 60),
                                              ([25], ol.BINOMIAL, 100)])
def test_either_side_of_the_limit(tmp_path, ks, scoring, score):
    import torch
    rng = np.random.default_rng(ks[0] + scoring)
    genomes, filters, paths = _filters(tmp_path, rng, ks, 3)
    reads = []
    for n in (1535, 1536, 1537, 1536 + ks[0], 1792 + ks[0] - 1, 1792 + ks[0], 3000):
        for share in (0.0, 0.1, 0.2, 1.0):  # of the read's bases, from its start
            own = int(n * share)
            st = int(rng.integers(0, 20000 - n))
            r = np.concatenate([genomes[0][st:st + own], rng.choice(ACGT, n - own)])
            r[rng.random(n) < 0.002] = ord("N")
            reads += [r.tobytes(), r[::-1].tobytes()]
    thr = 10.0 ** (-score / 10.0) if scoring == ol.BINOMIAL else score
    want, alg = ol.classify(*ol.pack_reads(reads), filters, thr, 3, scoring=scoring,
                            count_probes=True)
    dev = _device(reads, 3)
    with _open(paths, scoring, score, 3, path=2) as bbc:
        for count in (False, True):
            bbc.set_counting(count)
            got = bbc.classify_device(*dev)
            torch.cuda.synchronize()
            assert np.array_equal(got[0].cpu().numpy().view(np.uint64), want)
        assert bbc.last_stats()["probes_algorithmic"] == alg
