"""The lane kernel (batches of at least 20,000 reads, over filters that fit L2): hits, probe
counts, categories and scores against the oracle, for ASCII and packed bases at
any offset, reads and pairs, filters of one and of several k, every scoring
method, masking, reads around the length from which a warp takes a read, a
CUDA graph and host batches."""
import ctypes

import numpy as np
import pytest

from tests import oracle_lib as ol

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", dtype=np.uint8)


@pytest.fixture(scope="module", autouse=True)
def _need_gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")
    from biobloom_b200 import _lib
    _lib.lib()


def _filters(tmp_path, rng, ks, h, glen=20000, fpr=0.1):
    genomes = [rng.choice(ACGT, glen) for _ in ks]
    filters = [ol.Filter.make([g.tobytes()], k=k, fpr=fpr, h=h) for g, k in zip(genomes, ks)]
    paths = []
    for i, f in enumerate(filters):
        stem = str(tmp_path / f"q{i}")
        f.store(stem + ".bf")
        ol.write_info(stem + ".txt", f"q{i}", f.k, fpr, f.h, 1, "x", f.m, 1, 0.1, 0, 0.1)
        paths.append(stem + ".bf")
    return genomes, filters, paths


def _reads(rng, genomes, n, k):
    """Lengths 0-300, with the edges of a k-mer, of a step of eight bases and of
    the lane kernel's longest read, and a few long ones."""
    edges = [0, 1, k - 1, k, k + 1, k + 6, k + 7, k + 8, 1023, 1024, 1025, 1032, 2600]
    lens = rng.integers(0, 300, n)
    lens[:len(edges)] = edges
    lens[len(edges):len(edges) + 40] = rng.integers(900, 1400, 40)
    rng.shuffle(lens)
    out = []
    for L in lens:
        g = genomes[int(rng.integers(0, len(genomes)))]
        st = int(rng.integers(0, len(g) - L))
        r = (g[st:st + L] if rng.random() < 0.7 else rng.choice(ACGT, L)).copy()
        m = rng.random(L) < 0.01
        r[m] = rng.choice(ACGT, m.sum())
        u = rng.random()
        if u < 0.2:
            m = rng.random(L) < 0.02
            r[m] = np.frombuffer(b"NnX-", dtype=np.uint8)[rng.integers(0, 4, m.sum())]
        elif u < 0.3:
            r = np.where(rng.random(L) < 0.5, r | 0x20, r).astype(np.uint8)
        elif u < 0.35 and L > 40:
            r[5:35] = np.frombuffer(b"ACACACACACACACACACACACACACACAC", dtype=np.uint8)
        out.append(r.tobytes())
    return out


def _open(paths, scoring, score, streak, **kw):
    from biobloom_b200 import BioBloomClassifier
    return BioBloomClassifier(paths, score, streak_threshold=streak, score_type="simple"
                              if scoring == ol.LENGTH else
                              {ol.SIMPLE: "simple", ol.HARMONIC: "harmonic",
                               ol.BINOMIAL: "binomial"}[scoring], **kw)


def _device(reads, lead=0):
    """Bases and offsets on the GPU, the first read at base `lead`."""
    import torch
    seq, off = ol.pack_reads(reads)
    buf = np.frombuffer(b"G" * lead + seq, dtype=np.uint8)
    return (torch.tensor(buf, device="cuda"),
            torch.tensor((off + np.uint64(lead)).astype(np.int64), device="cuda"))


CASES = [
    # ks, h, scoring, score, streak, paired, first base
    ([25], 3, ol.SIMPLE, 0.15, 3, False, 0),
    ([25], 0, ol.SIMPLE, 0.5, 1, True, 1),
    ([32], 1, ol.SIMPLE, 0.05, 2, False, 2),
    ([8], 6, ol.SIMPLE, 0.9, 4, False, 3),
    ([5, 31], 2, ol.SIMPLE, 0.3, 3, True, 5),
    ([16, 24, 17], 4, ol.SIMPLE, 1.0, 3, False, 7),
    ([25], 3, ol.HARMONIC, 0.15, 3, False, 0),
    ([21, 25], 3, ol.HARMONIC, 0.4, 2, True, 1),
    ([25], 3, ol.BINOMIAL, 100, 3, False, 0),
    ([25, 20], 2, ol.BINOMIAL, 30, 2, True, 3),
    ([25], 3, ol.LENGTH, 40, 3, False, 2),
    ([12, 28], 3, ol.LENGTH, 31, 3, True, 6),
]


@pytest.mark.parametrize("ks,h,scoring,score,streak,paired,lead", CASES)
def test_hits_and_probe_counts(tmp_path, ks, h, scoring, score, streak, paired, lead):
    import torch
    rng = np.random.default_rng(len(ks) * 1000 + ks[0] * 10 + scoring)
    genomes, filters, paths = _filters(tmp_path, rng, ks, h)
    n = 28100 // (2 if paired else 1) + 37
    mates = [_reads(rng, genomes, n, ks[0]) for _ in range(2 if paired else 1)]
    thr = 10.0 ** (-score / 10.0) if scoring == ol.BINOMIAL else score
    want, alg = [], 0
    for m in mates:
        w, a = ol.classify(*ol.pack_reads(m), filters, thr, streak, scoring=scoring,
                           count_probes=True)
        want.append(w)
        alg += a
    _, cats = ol.summary_counts(want[0], len(ks), want[1] if paired else None)
    with _open(paths, scoring, score, streak) as bbc:
        dev = [t for m in mates for t in _device(m, lead)]
        for count in (False, True):
            bbc.set_counting(count)
            got = bbc.classify_device(*dev)
            torch.cuda.synchronize()
            for w, t in zip(want, (got[0], got[1])):
                assert np.array_equal(t.cpu().numpy().view(np.uint64), w)
            assert np.array_equal(got[2].cpu().numpy().view(np.uint32), cats)
        st = bbc.last_stats()
        assert st["probes_algorithmic"] == alg
        assert st["probes_issued"] >= alg
        host = bbc.classify(*mates)
        for w, t in zip(want, (host[0], host[1])):
            assert np.array_equal(t, w)


@pytest.mark.parametrize("ks,h,lead,with_valid", [([25], 3, 0, True), ([25], 2, 13, True),
                                                  ([32, 9], 3, 37, True), ([25], 3, 21, False)])
def test_packed_bases(tmp_path, ks, h, lead, with_valid):
    import torch
    from biobloom_b200 import _lib as L
    rng = np.random.default_rng(50 + lead)
    genomes, filters, paths = _filters(tmp_path, rng, ks, h)
    reads = _reads(rng, genomes, 20300, ks[0])
    if not with_valid:
        reads = [bytes(c if c in b"ACGTacgt" else 65 for c in r) for r in reads]
    seq, off = ol.pack_reads(reads)
    want, _ = ol.classify(seq, off, filters, 0.15, 3)
    data = b"C" * lead + seq
    words = np.zeros((len(data) + 15) // 16, dtype=np.uint32)
    valid = np.zeros((len(data) + 31) // 32, dtype=np.uint32)
    buf = np.frombuffer(data, dtype=np.uint8)
    L.check(L.lib().bbt_pack_bases(buf.ctypes.data, len(data), words.ctypes.data,
                                   valid.ctypes.data, None))
    with _open(paths, ol.SIMPLE, 0.15, 3) as bbc:
        dw = torch.tensor(words.view(np.int32), device="cuda")
        dv = torch.tensor(valid.view(np.int32), device="cuda")
        do = torch.tensor((off + np.uint64(lead)).astype(np.int64), device="cuda")
        hits = torch.full((len(reads), 1), -1, dtype=torch.int64, device="cuda")
        b, r = L.Batch(), L.Result()
        b.seq, b.offsets, b.n_reads = dw.data_ptr(), do.data_ptr(), len(reads)
        b.valid = dv.data_ptr() if with_valid else None
        b.location = r.location = L.DEVICE
        b.encoding, r.hits = L.BASES_2BIT, hits.data_ptr()
        L.check(L.lib().bbt_classify_batch(bbc._ctx, ctypes.byref(b), ctypes.byref(r), None),
                bbc._ctx)
        bbc.sync()
        assert np.array_equal(hits.cpu().numpy().view(np.uint64), want)


@pytest.mark.parametrize("ks,scoring,paired", [([25], ol.SIMPLE, False), ([25, 25], ol.SIMPLE, True),
                                               ([25, 21], ol.HARMONIC, False),
                                               ([25, 25], ol.HARMONIC, True),
                                               ([25, 18], ol.LENGTH, False),
                                               ([25], ol.BINOMIAL, False)])
def test_scores_and_best_hits(tmp_path, ks, scoring, paired):
    import torch
    from biobloom_b200 import MODE_BESTHIT, MODE_SCORES
    rng = np.random.default_rng(70 + scoring + len(ks))
    genomes, filters, paths = _filters(tmp_path, rng, ks, 3)
    n = 20100 // (2 if paired else 1) + 11
    mates = [_reads(rng, genomes, n, ks[0]) for _ in range(2 if paired else 1)]
    want = [ol.classify_scores(*ol.pack_reads(m), filters, scoring, 3) for m in mates]
    score = {ol.LENGTH: 40, ol.BINOMIAL: 100}.get(scoring, 0.15)
    dev = [t for m in mates for t in _device(m, 3)]
    with _open(paths, scoring, score, 3) as bbc:
        bbc.set_mode(MODE_SCORES)
        sc = [torch.full((n, len(ks)), -7.0, dtype=torch.float64, device="cuda") for _ in mates]
        bbc.classify_device(*dev, scores=sc[0], scores2=sc[1] if paired else None)
        torch.cuda.synchronize()
        got = [t.cpu().numpy() for t in sc]
        for g, w in zip(got, want):
            if scoring != ol.BINOMIAL:
                assert np.array_equal(g.view(np.uint64), w.view(np.uint64))
            else:
                # terms of a tail in log space, as tests/test_filter_modes_gpu.py derives
                same = g.view(np.uint64) == w.view(np.uint64)
                assert np.all(same | np.isclose(g, w, rtol=1e-12, atol=1e-9))
        bbc.set_mode(MODE_BESTHIT)
        hits = bbc.classify_device(*dev)
        torch.cuda.synchronize()
        for t, g in zip(hits[:2], got):
            assert np.array_equal(t.cpu().numpy().view(np.uint64), ol.best_hit(g)[0])


def test_dust_and_ordered(tmp_path):
    import torch
    from biobloom_b200 import MODE_ORDERED
    rng = np.random.default_rng(90)
    genomes, filters, paths = _filters(tmp_path, rng, [25, 25, 25], 3)
    reads = _reads(rng, genomes, 20400, 25)
    with ol.dust():
        want, _ = ol.classify(*ol.pack_reads(reads), filters, 0.15, 3)
    with _open(paths, ol.SIMPLE, 0.15, 3) as bbc:
        bbc.set_dust()
        dev = _device(reads, 5)
        hits, _, _ = bbc.classify_device(*dev)
        torch.cuda.synchronize()
        assert np.array_equal(hits.cpu().numpy().view(np.uint64), want)
        bbc.set_mode(MODE_ORDERED)
        hits, _, _ = bbc.classify_device(*dev)
        torch.cuda.synchronize()
        assert np.array_equal(hits.cpu().numpy().view(np.uint64), ol.ordered(want, 3)[0])


def test_graph_replays_on_new_reads(tmp_path):
    """A graph captured before any other call of this size, replayed on other
    reads in the same buffers."""
    import torch
    rng = np.random.default_rng(91)
    genomes, filters, paths = _filters(tmp_path, rng, [25], 3)
    a, b = _reads(rng, genomes, 20900, 25), _reads(rng, genomes, 20900, 25)
    (sa, oa), (sb, ob) = _device(a), _device(b)
    seq = torch.zeros(max(len(sa), len(sb)), dtype=torch.uint8, device="cuda")
    off, hits = oa.clone(), torch.empty((20900, 1), dtype=torch.int64, device="cuda")
    stream = torch.cuda.Stream()
    with _open(paths, ol.SIMPLE, 0.15, 3) as bbc:
        g = bbc.graph(seq, off, hits)
        for reads, s, o in ((a, sa, oa), (b, sb, ob)):
            seq[:len(s)] = s
            off.copy_(o)
            hits.fill_(-1)
            torch.cuda.synchronize()
            g.launch(stream)
            torch.cuda.synchronize()
            want, _ = ol.classify(*ol.pack_reads(reads), filters, 0.15, 3)
            assert np.array_equal(hits.cpu().numpy().view(np.uint64), want)
        g.close()


@pytest.mark.parametrize("ks,h,scoring,score,streak,paired,lead", CASES)
def test_long_reads_of_small_batches(tmp_path, ks, h, scoring, score, streak, paired, lead):
    """Below that size the warp kernel takes the batch, and evaluates reads above
    384 bases in windows of 256 frames."""
    import torch
    rng = np.random.default_rng(ks[0] * 10 + scoring)
    genomes, filters, paths = _filters(tmp_path, rng, ks, h)
    mates = [_reads(rng, genomes, 300, ks[0]) + _reads(rng, genomes, 60, ks[0])
             for _ in range(2 if paired else 1)]
    for m in mates:
        for n in (383, 384, 385, 256 + ks[0] - 1, 512 + ks[0] - 1, 512 + ks[0], 6000):
            st = int(rng.integers(0, 20000 - n))
            m[int(rng.integers(0, 300))] = genomes[0][st:st + n].tobytes()
            m[int(rng.integers(0, 300))] = rng.choice(ACGT, n).tobytes()
    thr = 10.0 ** (-score / 10.0) if scoring == ol.BINOMIAL else score
    with _open(paths, scoring, score, streak, path=2) as bbc:
        dev = [t for m in mates for t in _device(m, lead)]
        for count in (False, True):
            bbc.set_counting(count)
            got = bbc.classify_device(*dev)
            torch.cuda.synchronize()
            alg = 0
            for m, t in zip(mates, (got[0], got[1])):
                w, a = ol.classify(*ol.pack_reads(m), filters, thr, streak, scoring=scoring,
                                   count_probes=True)
                alg += a
                assert np.array_equal(t.cpu().numpy().view(np.uint64), w)
        assert bbc.last_stats()["probes_algorithmic"] == alg


@pytest.mark.parametrize("ks,scoring,score,paired", [([25], ol.SIMPLE, 0.15, False),
                                                     ([25, 25], ol.SIMPLE, 0.6, True),
                                                     ([25, 21], ol.HARMONIC, 0.15, False),
                                                     ([18, 25], ol.LENGTH, 40, True),
                                                     ([25], ol.BINOMIAL, 100, False)])
def test_hits_beside_scores(tmp_path, ks, scoring, score, paired):
    """SCORES mode takes hits and scores from one walk: the hits are those of a
    call without scores."""
    import torch
    from biobloom_b200 import MODE_SCORES
    rng = np.random.default_rng(120 + scoring + len(ks))
    genomes, filters, paths = _filters(tmp_path, rng, ks, 3)
    n = 20100 // (2 if paired else 1) + 3
    mates = [_reads(rng, genomes, n, ks[0]) for _ in range(2 if paired else 1)]
    thr = 10.0 ** (-score / 10.0) if scoring == ol.BINOMIAL else score
    dev = [t for m in mates for t in _device(m, 1)]
    with _open(paths, scoring, score, 3) as bbc:
        bbc.set_mode(MODE_SCORES)
        sc = [torch.full((n, len(ks)), -7.0, dtype=torch.float64, device="cuda") for _ in mates]
        got = bbc.classify_device(*dev, scores=sc[0], scores2=sc[1] if paired else None)
        torch.cuda.synchronize()
    for m, t in zip(mates, got[:2]):
        want, _ = ol.classify(*ol.pack_reads(m), filters, thr, 3, scoring=scoring)
        assert np.array_equal(t.cpu().numpy().view(np.uint64), want)


@pytest.mark.parametrize("nf,n,mode,lane", [
    (4, 19999, "std", False), (4, 20000, "std", True), (5, 24999, "std", False),
    (5, 25000, "std", True), (5, 20000, "best", True), (13, 59999, "std", False),
    (13, 60000, "std", True), (11, 27999, "best", False), (11, 28000, "best", True)])
def test_many_small_filters_choose_by_reads(tmp_path, nf, n, mode, lane):
    """Either side of the sizes from which several filters in L2 take the lane kernel
    (one launch a filter, against one for all)."""
    import torch
    from biobloom_b200 import MODE_BESTHIT, BioBloomClassifier
    from biobloom_b200 import _lib as L
    rng = np.random.default_rng(nf * 100000 + n)
    genomes, filters, paths = _filters(tmp_path, rng, [25] * nf, 3, glen=3000)
    reads = []
    for size in rng.integers(0, 60, n):
        g = genomes[int(rng.integers(0, nf))]
        st = int(rng.integers(0, len(g) - size))
        reads.append(g[st:st + size].tobytes())
    seq, off = ol.pack_reads(reads)
    if mode == "best":
        want, _ = ol.best_hit(ol.classify_scores(seq, off, filters, ol.SIMPLE, 3))
    else:
        want, _ = ol.classify(seq, off, filters, 0.15, 3)
    with BioBloomClassifier(paths, 0.15, streak_threshold=3, path=L.PATH_PERSISTENT) as bbc:
        if mode == "best":
            bbc.set_mode(MODE_BESTHIT)
        got = bbc.classify_device(*_device(reads, 0))
        torch.cuda.synchronize()
        assert np.array_equal(got[0].cpu().numpy().view(np.uint64), want)
        assert (bbc.last_stats()["kernels"] > nf) == lane
