"""Contexts of different sizes in threads of one process: kernels whose shared memory depends
on the context are launched by all of them at once."""
import threading

import numpy as np
import pytest

from tests import oracle_lib as ol
from tests.test_lane_gpu import _device, _filters, _open, _reads
from tests.test_mibf_gpu import _genome

pytestmark = pytest.mark.gpu


def _at_once(calls, times):
    """Each call in a thread of its own, `times` times; returns what they raised."""
    raised = []
    go = threading.Barrier(len(calls))

    def loop(call):
        go.wait()
        try:
            for _ in range(times):
                call()
        except Exception as e:  # noqa: BLE001
            raised.append(e)

    threads = [threading.Thread(target=loop, args=(c,)) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return raised


def test_masking_windows(tmp_path):
    import torch
    rng = np.random.default_rng(3)
    genomes, filters, paths = _filters(tmp_path, rng, [25], 3)
    reads = [r[:100] for r in _reads(rng, genomes, 120, 25)]
    dev = _device(reads)
    torch.cuda.synchronize()
    opened, got = [], {}
    for W in (16, 64, 1024):
        c = _open(paths, ol.SIMPLE, 0.15, 3)
        c.set_dust(True, 20, W)
        opened.append(c)

    def call(i):
        with torch.cuda.stream(streams[i]):
            got[i] = opened[i].classify_device(*dev)[0]

    streams = [torch.cuda.Stream() for _ in opened]
    raised = _at_once([lambda i=i: call(i) for i in range(len(opened))], 300)
    assert not raised
    torch.cuda.synchronize()
    for i, W in enumerate((16, 64, 1024)):
        with ol.dust(20, W):
            want, _ = ol.classify(*ol.pack_reads(reads), filters, 0.15, 3)
        assert np.array_equal(got[i].cpu().numpy().view(np.uint64), want)
    for c in opened:
        c.close()


def test_window_sizes(tmp_path):
    """k and the frames a lane hashes size the windows of the read-major and filter-major kernels."""
    import torch
    rng = np.random.default_rng(5)
    opened, streams, got = [], [], {}
    for k, frames, path in ((8, 4, 2), (60, 8, 2), (25, 8, 2), (8, 4, 3), (60, 8, 3)):
        d = tmp_path / f"k{k}_{frames}_{path}"
        d.mkdir()
        genomes, filters, paths = _filters(d, rng, [k, k], 3)
        reads = [r[:200] for r in _reads(rng, genomes, 120, k)]
        c = _open(paths, ol.SIMPLE, 0.15, 3, path=path)
        c.set_launch(path, 8, frames)
        opened.append((c, _device(reads), ol.classify(*ol.pack_reads(reads), filters, 0.15, 3)[0]))
        streams.append(torch.cuda.Stream())
    torch.cuda.synchronize()

    def call(i):
        with torch.cuda.stream(streams[i]):
            got[i] = opened[i][0].classify_device(*opened[i][1])[0]

    raised = _at_once([lambda i=i: call(i) for i in range(len(opened))], 300)
    assert not raised
    torch.cuda.synchronize()
    for i, (c, _, want) in enumerate(opened):
        assert np.array_equal(got[i].cpu().numpy().view(np.uint64), want)
        c.close()


@pytest.mark.parametrize("long_read", [False, True])
def test_numbers_of_ids(tmp_path, long_read):
    """The scan kernel, and the general one, which a batch with a long read takes."""
    import torch
    from biobloom_b200.mibf import MIBFClassifier
    rng = np.random.default_rng(4)
    opened = []
    for n in (5, 400, 1000):
        targets = [_genome(rng, 200).tobytes() for _ in range(n)]
        f = ol.MIBF.build(targets, list(range(1, n + 1)), k=25, h=8, occupancy=0.5)
        f.store(str(tmp_path / f"x{n}"))
        with open(tmp_path / f"x{n}_ids.txt", "w") as fh:
            for i in range(n):
                fh.write(f"{i + 1}\tt{i}\n")
        opened.append((MIBFClassifier(str(tmp_path / f"x{n}.bf"), layout=2),
                       _device(targets[:5] * 20 + [_genome(rng, 9000 if long_read else 90).tobytes()]),
                       torch.cuda.Stream()))
    torch.cuda.synchronize()
    got = {}

    def call(i):
        c, dev, stream = opened[i]
        with torch.cuda.stream(stream):
            got[i] = c.classify_device(*dev, max_hits=2)

    raised = _at_once([lambda i=i: call(i) for i in range(len(opened))], 300)
    assert not raised
    torch.cuda.synchronize()
    for i, (c, _, _) in enumerate(opened):
        hits, n_hits, _ = (t.cpu().numpy() for t in got[i])
        assert (n_hits[:100] == 1).all() and n_hits[100] == 0
        assert np.array_equal(hits[:100, 0, 0], np.tile(np.arange(1, 6), 20))
        c.close()
