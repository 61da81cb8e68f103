"""Which kernels a batch goes to by the lengths of its reads: hits, categories, probe counts
and best hits against the oracle where the lane kernel always takes the batch, where the
lengths decide (on the device, or on the host for the filter-major path), and on both sides
of the lengths that are listed for whole warps."""
import numpy as np
import pytest

from tests import oracle_lib as ol
from tests.test_lane_gpu import ACGT, _device, _filters, _open

pytestmark = pytest.mark.gpu


def _reads(rng, genomes, lens):
    out = []
    for n in lens:
        g = genomes[int(rng.integers(0, len(genomes)))]
        st = int(rng.integers(0, len(g) - n))
        r = (g[st:st + n] if rng.random() < 0.7 else rng.choice(ACGT, n)).copy()
        if rng.random() < 0.2:
            r[rng.random(n) < 0.02] = ord("N")
        out.append(r.tobytes())
    return out


def _lengths(rng, kind, n):
    """n lengths; all but "even" have reads at the edges of the listed ones."""
    if kind == "even":  # the lane kernel's
        return rng.integers(100, 119, n)
    lens = rng.integers(20, 120, n)  # "ragged": the other kernels' in batches that do not fill it
    if kind == "long":  # the lane kernel's, but for many small filters
        lens[rng.random(n) < 0.02] = 1025 + int(rng.integers(0, 100))
    elif kind == "mids":
        lens = np.where(rng.random(n) < 0.65, rng.integers(385, 450, n), 40)
    elif kind == "some mids":
        lens = np.where(rng.random(n) < 0.14, rng.integers(385, 420, n), 40)
    edges = [24, 25, 383, 384, 385, 391, 1023, 1024, 1025, 1032, 2000]
    lens[rng.choice(n, len(edges), replace=False)] = edges
    return lens


def _check(tmp_path, rng, ks, kind, n, paired, best, scoring=ol.SIMPLE, score=0.15, path=0, **filters):
    import torch
    from biobloom_b200 import MODE_BESTHIT
    genomes, fs, paths = _filters(tmp_path, rng, ks, filters.pop("h", 3), **filters)
    mates = [_reads(rng, genomes, _lengths(rng, kind, n)) for _ in range(2 if paired else 1)]
    dev = [t for m in mates for t in _device(m, 3)]
    torch.cuda.synchronize()
    alg, want = 0, []
    for m in mates:
        seq, off = ol.pack_reads(m)
        if best:
            want.append(ol.best_hit(ol.classify_scores(seq, off, fs, scoring, 3))[0])
            continue
        w, a = ol.classify(seq, off, fs, score, 3, scoring=scoring, count_probes=True)
        want.append(w)
        alg += a
    with _open(paths, scoring, score, 3, path=path) as bbc:
        if best:
            bbc.set_mode(MODE_BESTHIT)
        for count in (False, True):
            bbc.set_counting(count and not best)
            got = bbc.classify_device(*dev)
            torch.cuda.synchronize()
            for w, t in zip(want, got):
                assert np.array_equal(t.cpu().numpy().view(np.uint64), w)
        stats = bbc.last_stats()
        if not best:
            assert stats["probes_algorithmic"] == alg
        return stats


@pytest.mark.parametrize("kind,n,paired,best", [
    ("even", 20100, False, False), ("ragged", 20100, False, False), ("long", 20100, False, False),
    ("mids", 30000, False, False), ("even", 10100, True, False), ("long", 12000, True, False),
    ("ragged", 40100, False, False), ("mids", 40100, False, False),  # 26,000: by lanes
    ("ragged", 20100, False, True), ("mids", 40100, False, True)])
def test_one_small_filter(tmp_path, kind, n, paired, best):
    _check(tmp_path, np.random.default_rng(n + paired), [25], kind, n, paired, best)


@pytest.mark.parametrize("ks,scoring,score,kind,n", [
    ([25], ol.HARMONIC, 0.15, "ragged", 61000), ([25], ol.HARMONIC, 0.15, "mids", 61000),
    ([25, 25], ol.HARMONIC, 0.15, "even", 28100), ([25], ol.LENGTH, 40, "even", 20100),
    ([25], ol.LENGTH, 40, "even", 61000), ([25], ol.LENGTH, 40, "long", 20100),
    ([25, 21], ol.LENGTH, 40, "even", 151000), ([25], ol.SIMPLE, 0.8, "even", 20100),
    ([25, 25], ol.SIMPLE, 0.8, "even", 151000)])
def test_other_scoring(tmp_path, ks, scoring, score, kind, n):
    _check(tmp_path, np.random.default_rng(n), ks, kind, n, False, False, scoring, score)


@pytest.mark.parametrize("kind,n,best", [
    ("even", 28100, False), ("ragged", 28100, False), ("long", 28100, False), ("mids", 28100, False),
    ("even", 28100, True), ("ragged", 28100, True), ("long", 28100, True),
    ("some mids", 160100, False), ("some mids", 160100, True)])
def test_a_filter_larger_than_l2(tmp_path, kind, n, best):
    """147 MB: probes past L2, reads above 384 bases listed unless there are many."""
    _check(tmp_path, np.random.default_rng(n), [25], kind, n, False, best, fpr=1.7e-5, h=1)


def test_listed_reads_by_match_length(tmp_path):
    _check(tmp_path, np.random.default_rng(3), [25], "long", 28100, False, False, ol.LENGTH, 40,
           fpr=1.7e-5, h=1)


@pytest.mark.parametrize("nf,kind,n,best,asked,lane", [
    (3, "even", 28100, False, False, False), (3, "even", 40100, False, True, True),
    (3, "ragged", 40100, False, True, False), (3, "long", 40100, False, True, True),
    (3, "mids", 41000, False, True, False), (3, "ragged", 150100, False, False, True),
    (3, "ragged", 40100, True, False, True), (6, "even", 30100, False, True, True),
    (6, "ragged", 30100, False, True, False), (6, "long", 30100, False, True, False),
    (6, "even", 28100, True, True, True), (6, "mids", 30100, True, True, False)])
def test_the_filter_major_path_asks_on_the_host(tmp_path, nf, kind, n, best, asked, lane):
    stats = _check(tmp_path, np.random.default_rng(nf * 1000 + n), [25] * nf, kind, n, False, best,
                   glen=4000)
    # summary, best hits; the list; two scans, and hash and filter pass or a kernel a filter
    assert stats["kernels"] == 1 + best + (asked or lane) + (2 if asked or not lane else 0) + \
        (nf if lane else 2)


@pytest.mark.parametrize("kind", ["even", "ragged"])
def test_a_graph_decides_at_each_launch(tmp_path, kind):
    """Captured on reads of one kind, replayed on both."""
    import torch
    rng = np.random.default_rng(77)
    genomes, fs, paths = _filters(tmp_path, rng, [25], 3)
    n = 21000
    batches = [_reads(rng, genomes, _lengths(rng, k, n)) for k in (kind, "even", "ragged")]
    dev = [_device(b) for b in batches]
    seq = torch.zeros(max(len(s) for s, _ in dev), dtype=torch.uint8, device="cuda")
    off, hits = dev[0][1].clone(), torch.empty((n, 1), dtype=torch.int64, device="cuda")
    seq[:len(dev[0][0])] = dev[0][0]
    torch.cuda.synchronize()
    with _open(paths, ol.SIMPLE, 0.15, 3) as bbc:
        g = bbc.graph(seq, off, hits)
        for reads, (s, o) in zip(batches[1:], dev[1:]):
            seq[:len(s)] = s
            off.copy_(o)
            hits.fill_(-1)
            torch.cuda.synchronize()
            g.launch()
            torch.cuda.synchronize()
            want, _ = ol.classify(*ol.pack_reads(reads), fs, 0.15, 3)
            assert np.array_equal(hits.cpu().numpy().view(np.uint64), want)
        g.close()
