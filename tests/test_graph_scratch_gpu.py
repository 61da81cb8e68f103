"""Captured graphs beside other calls on their context: calls that need more scratch than
the graph's own launches come between the capture and its replays."""
import numpy as np
import pytest

from tests import oracle_lib as ol
from tests.test_lane_gpu import _device, _filters, _open, _reads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,paired,n,schedule,first", [
    ("std", False, 20900, 0, False),     # a read per lane, long ones listed
    ("std", True, 14100, 0, False),
    ("best", False, 20900, 0, False),    # scores stored
    ("best", True, 14100, 0, True),      # after a call that has sized the context's scores
    ("std", False, 3000, 300, False),    # long reads first
])
def test_replays_after_larger_calls(tmp_path, mode, paired, n, schedule, first):
    import torch
    from biobloom_b200 import MODE_BESTHIT
    rng = np.random.default_rng(n + paired)
    genomes, filters, paths = _filters(tmp_path, rng, [25, 25], 3)
    mates = [_reads(rng, genomes, n, 25) for _ in range(2 if paired else 1)]
    more = [_reads(rng, genomes, 2 * n + 40, 25) for _ in mates]
    dev = [t for m in mates for t in _device(m)]
    dev_more = [t for m in more for t in _device(m)]
    hits = [torch.empty((n, 1), dtype=torch.int64, device="cuda") for _ in mates]
    torch.cuda.synchronize()

    def want(reads):
        seq, off = ol.pack_reads(reads)
        if mode == "best":
            return ol.best_hit(ol.classify_scores(seq, off, filters, ol.SIMPLE, 3))[0]
        return ol.classify(seq, off, filters, 0.15, 3)[0]

    with _open(paths, ol.SIMPLE, 0.15, 3, path=2) as bbc:
        if mode == "best":
            bbc.set_mode(MODE_BESTHIT)
        bbc.set_schedule(schedule)
        if first:
            bbc.classify_device(*dev)
        g = bbc.graph(dev[0], dev[1], hits[0], *dev[2:], **({"hits2": hits[1]} if paired else {}))
        stream = torch.cuda.Stream()
        for _ in range(2):
            got = bbc.classify_device(*dev_more)
            for h in hits:
                h.fill_(-1)
            torch.cuda.synchronize()
            g.launch(stream)
            torch.cuda.synchronize()
            for h, m in zip(hits, mates):
                assert np.array_equal(h.cpu().numpy().view(np.uint64), want(m))
            for h, m in zip(got, more):
                assert np.array_equal(h.cpu().numpy().view(np.uint64), want(m))
        g.close()


def test_binomial_thresholds_outlive_a_larger_table(tmp_path):
    """A call with longer reads replaces the context's threshold table; the graph reads on in
    the one it was captured with."""
    import torch
    rng = np.random.default_rng(17)
    genomes, filters, paths = _filters(tmp_path, rng, [25, 21], 3)
    reads = [genomes[0][i:i + 150].tobytes() for i in range(400)] + \
        [rng.choice(genomes[0], 150).tobytes() for _ in range(400)]
    longer = [genomes[1][:9000].tobytes(), rng.choice(genomes[1], 5000).tobytes()]
    want = [ol.classify(*ol.pack_reads(r), filters, 10.0 ** -10.0, 3, scoring=ol.BINOMIAL)[0]
            for r in (reads, longer)]
    dev, dev_longer = _device(reads), _device(longer)
    hits = torch.empty((len(reads), 1), dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    with _open(paths, ol.BINOMIAL, 100, 3, path=2) as bbc:
        g = bbc.graph(*dev, hits)
        for _ in range(2):
            got = bbc.classify_device(*dev_longer)[0]
            torch.cuda.synchronize()
            assert np.array_equal(got.cpu().numpy().view(np.uint64), want[1])
            taken = torch.full((1 << 22,), -1, dtype=torch.int32, device="cuda")  # over freed memory
            hits.fill_(-1)
            torch.cuda.synchronize()
            g.launch()
            torch.cuda.synchronize()
            assert np.array_equal(hits.cpu().numpy().view(np.uint64), want[0])
            del taken
        g.close()
