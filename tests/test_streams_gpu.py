"""Calls of one context on several streams, none of them waited for: each has the results it
has alone, although they share the context's scratch (work counters, list of long reads,
stored scores)."""
import numpy as np
import pytest

from tests import oracle_lib as ol
from tests.test_lane_gpu import _device, _filters, _open, _reads

pytestmark = pytest.mark.gpu

# reads of each stream's batch; the second of every pair ends long before the first
SIZES = {"lane": (46000, 41000), "small": (9000, 300), "both": (46000, 300)}


@pytest.mark.parametrize("mode,size,path,nf", [
    ("std", "lane", 2, 1), ("std", "small", 2, 1), ("std", "both", 2, 2), ("best", "lane", 2, 2),
    ("best", "both", 2, 2), ("std", "small", 3, 3), ("best", "small", 3, 3)])
def test_calls_in_flight_together(tmp_path, mode, size, path, nf):
    import torch
    from biobloom_b200 import MODE_BESTHIT
    rng = np.random.default_rng(nf * 10 + len(size))
    genomes, filters, paths = _filters(tmp_path, rng, [25] * nf, 3)
    batches = [_reads(rng, genomes, n, 25) for n in SIZES[size]]
    dev = [_device(b) for b in batches]
    want = []
    for b in batches:
        seq, off = ol.pack_reads(b)
        want.append(ol.best_hit(ol.classify_scores(seq, off, filters, ol.SIMPLE, 3))[0]
                    if mode == "best" else ol.classify(seq, off, filters, 0.15, 3)[0])
    streams = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    with _open(paths, ol.SIMPLE, 0.15, 3, path=path) as bbc:
        if mode == "best":
            bbc.set_mode(MODE_BESTHIT)
        got = []
        for i in range(12):
            with torch.cuda.stream(streams[i % 3]):
                got.append((i % 2, bbc.classify_device(*dev[i % 2])[0]))
        host = bbc.classify(batches[1])[0]  # beside what is in flight
        torch.cuda.synchronize()
        for which, hits in got:
            assert np.array_equal(hits.cpu().numpy().view(np.uint64), want[which])
        assert np.array_equal(host, want[1])


def test_a_stream_that_the_caller_captures(tmp_path):
    """Captured with the caller's own graph: the call takes kernels without growable scratch,
    and calls of any size may come between the replays."""
    import torch
    rng = np.random.default_rng(5)
    genomes, filters, paths = _filters(tmp_path, rng, [25], 3)
    reads, more = _reads(rng, genomes, 42000, 25), _reads(rng, genomes, 90000, 25)
    dev, dev_more = _device(reads), _device(more)
    hits = torch.empty((len(reads), 1), dtype=torch.int64, device="cuda")
    cat = torch.empty(len(reads), dtype=torch.int32, device="cuda")
    want = [ol.classify(*ol.pack_reads(r), filters, 0.15, 3)[0] for r in (reads, more)]
    with _open(paths, ol.SIMPLE, 0.15, 3) as bbc:
        bbc.classify_device(*dev, hits=hits, category=cat)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            bbc.classify_device(*dev, hits=hits, category=cat)
        for _ in range(2):
            got = bbc.classify_device(*dev_more)[0]
            hits.fill_(-1)
            torch.cuda.synchronize()
            graph.replay()
            torch.cuda.synchronize()
            assert np.array_equal(hits.cpu().numpy().view(np.uint64), want[0])
            assert np.array_equal(got.cpu().numpy().view(np.uint64), want[1])
        del graph


@pytest.mark.parametrize("layout", [1, 2])
def test_multi_index_queries_in_flight_together(tmp_path, layout):
    import torch
    from biobloom_b200.mibf import MIBFClassifier
    from tests.test_mibf_gpu import _reads as mibf_reads
    from tests.test_mibf_gpu import _targets
    rng = np.random.default_rng(6)
    targets = _targets(rng)
    f = ol.MIBF.build(targets, list(range(1, len(targets) + 1)), k=25, h=3, occupancy=0.5)
    f.store(str(tmp_path / "x"))
    with open(tmp_path / "x_ids.txt", "w") as fh:
        for i in range(len(targets)):
            fh.write(f"{i + 1}\tt{i}\n")
    c = MIBFClassifier(str(tmp_path / "x.bf"), layout=layout)
    batches = [mibf_reads(rng, targets, n)[0] for n in (30000, 700)]
    dev = [_device(b) for b in batches]
    streams = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    with torch.cuda.stream(streams[0]):
        want = [c.classify_device(*d, max_hits=4) for d in dev]
    torch.cuda.synchronize()
    got = []
    for i in range(12):
        with torch.cuda.stream(streams[i % 3]):
            got.append((i % 2, c.classify_device(*dev[i % 2], max_hits=4)))
    torch.cuda.synchronize()
    for which, result in got:
        for t, w in zip(result, want[which]):
            assert torch.equal(t, w)
    c.close()
