"""The two direct miBF query kernels over the dense map against the oracle: the scan kernel
(16-bit counters, up to 1024 IDs and 8 values a frame, reads whose frames x values stay
below 65536) at the edges of what it takes, and the general kernel with its tally in
shared memory, which a batch with a longer read takes."""
import numpy as np
import pytest

from tests import oracle_lib
from tests.test_mibf_gpu import _genome, _opts, _oracle_query, _reads, _targets

pytestmark = pytest.mark.gpu

DENSE = 2


def _build(folder, targets, seeds=None, k=25, h=3):
    names = [f"t{i + 1}" for i in range(len(targets))]
    f = oracle_lib.MIBF.build(targets, list(range(1, len(targets) + 1)), seeds=seeds, k=k, h=h,
                              occupancy=0.5)
    f.store(str(folder / "x"))
    with open(folder / "x_ids.txt", "w") as fh:
        for i, n in enumerate(names):
            fh.write(f"{i + 1}\t{n}\n")
    return str(folder / "x.bf"), f, names


def _check(path, f, names, reads, reads2=None, **opts):
    """Results, saturation counts and summary of the batch equal the oracle's; returns them."""
    from biobloom_b200.mibf import MIBFClassifier
    o = _opts(opts)
    want = _oracle_query(f, names, reads, reads2, o)
    mc = MIBFClassifier(path, score=o["score"], frame_matches=o["frame_matches"],
                        multi=o["multi"], min_nonsat=o["min_nonsat"], best_hit_agree=o["best"],
                        layout=DENSE)
    assert mc.layout == DENSE
    got, sat = mc.classify(reads, reads2, max_hits=8)
    for i, (res, s) in enumerate(want):
        assert (got[i], int(sat[i])) == (res, s), i
    counts, n = mc.summary()
    nf = len(names) + 1
    assert n == len(reads)
    assert counts[2 * (nf + 2) + 1] == sum(1 for r, _ in want if not r)
    assert counts[2 * (nf + 2)] == sum(1 for r, _ in want if len(r) > 1)
    mc.close()
    return want


# values a frame, frames: frames x values = 65535 fills a 16-bit counter, one frame more is past it
LIMITS = [(1, 65535), (1, 65536), (2, 32767), (2, 32768), (3, 21845), (3, 21846),
          (5, 13107), (5, 13108), (8, 8191), (8, 8192)]


@pytest.mark.parametrize("h,frames", LIMITS)
def test_reads_that_fill_the_counters(tmp_path, h, frames):
    """A read all of whose frames are the target's, among short ones."""
    rng = np.random.default_rng(h * 100000 + frames)
    k = 25
    target = _genome(rng, frames + k - 1).tobytes()  # the only one: no other ID takes a value
    path, f, names = _build(tmp_path, [target], h=h)
    comp = bytes.maketrans(b"ACGT", b"TGCA")
    reads = [target, target[:200], _genome(rng, 200).tobytes(),
             target[:frames // 2] + b"N" + target[frames // 2 + 1:],
             target.translate(comp)[::-1]]
    want = _check(path, f, names, reads)
    ID, NONSAT_FRAMES, SOLID, COUNT, NONSAT, TOTAL_NONSAT, TOTAL = range(7)
    best = want[0][0][0]
    assert best[ID] == 1 and best[COUNT] == frames and best[TOTAL] == frames * h


@pytest.mark.parametrize("over", [0, 1])
def test_pairs_whose_sum_fills_the_counters(tmp_path, over):
    rng = np.random.default_rng(40 + over)
    k = 25
    targets = [_genome(rng, 3000).tobytes(), _genome(rng, 26000).tobytes()]
    path, f, names = _build(tmp_path, targets)
    a, b = 11000, 10845 + over
    reads = [targets[1][:a + k - 1], targets[0][:300]]
    reads2 = [targets[1][:b + k - 1], targets[0][500:800]]
    _check(path, f, names, reads, reads2)


SEEDS = {
    "32": ["11111011111011111111011111011111", "11011111111111000011111111111011"],
    "zeros at the ends": ["0011110111011101110101", "1011101110111011110000",
                          "0001111110111111111000"],
    "one position": ["1" + "0" * 20, "0" * 20 + "1", "0" * 10 + "1" + "0" * 10],
    "alternating": ["10" * 12 + "1"] * 2,
    "four": ["1101111011101110110111011", "1011101101110111011110111",
             "1110110111011011110110111", "1111111111111111111111111"],
    "six": ["1101111011101110110111011", "1011101101110111011110111", "1110110111011011110110111",
            "1111111111110111111111111", "1110001111111111111000111", "1010111111111111111110101"],
}


@pytest.mark.parametrize("tag", sorted(SEEDS))
@pytest.mark.parametrize("paired", [False, True])
def test_seed_shapes(tmp_path, tag, paired):
    rng = np.random.default_rng(len(tag) + paired)
    seeds = SEEDS[tag]
    targets = _targets(rng, 12, 9000)
    path, f, names = _build(tmp_path, targets, seeds=seeds, k=len(seeds[0]))
    reads, reads2 = _reads(rng, targets, 250, paired=paired)
    _check(path, f, names, reads, reads2, multi=3.0)


@pytest.mark.parametrize("k,h", [(32, 3), (31, 1), (25, 2), (20, 4), (25, 5), (25, 6), (25, 7),
                                 (32, 8), (8, 8)])
def test_kmer_values(tmp_path, k, h):
    rng = np.random.default_rng(k * 10 + h)
    targets = _targets(rng, 10, 8000)
    path, f, names = _build(tmp_path, targets, k=k, h=h)
    reads, _ = _reads(rng, targets, 250)
    edges = [targets[0][:n] for n in (k - 1, k, k + 1, 31, 32, 33, 63, 64, 65, k + 30, k + 31, k + 32)]
    _check(path, f, names, reads + edges)


@pytest.mark.parametrize("n", [126, 127, 128, 129, 255, 256, 1022, 1023])
def test_numbers_of_ids(tmp_path, n):
    """IDs on either side of the tally's groups of 128, up to the 1024 (ID 0 among them) that
    it holds; reads that several targets, the last ones too, answer for."""
    rng = np.random.default_rng(n)
    targets = [_genome(rng, 300) for _ in range(n)]
    for i in range(3, n, 4):
        targets[i][100:220] = targets[i - 3][50:170]
    targets = [t.tobytes() for t in targets]
    path, f, names = _build(tmp_path, targets,
                            seeds=["1101111011101110110111011", "1011101101110111011110111"])
    reads = []
    for _ in range(250):
        t = int(rng.integers(0, n))
        st = int(rng.integers(0, 150))
        r = np.frombuffer(targets[t][st:st + 150], dtype=np.uint8).copy()
        r[rng.random(150) < 0.01] = ord("N")
        reads.append(r.tobytes())
    for last in (0, 1, 127, 128, n - 2, n - 1):
        reads.append(targets[min(last, n - 1)])
    reads += [b"".join(targets[i] for i in rng.integers(0, n, 5)) for _ in range(4)]
    want = _check(path, f, names, reads, multi=200.0)
    assert any(len(r) > 2 for r, _ in want)


@pytest.mark.parametrize("seeds", [True, False])
@pytest.mark.parametrize("paired", [False, True])
@pytest.mark.parametrize("opts", [{}, {"multi": 3.0}, {"frame_matches": 2, "min_nonsat": 2},
                                  {"frame_matches": 3, "best": True}])
def test_batches_with_a_read_past_the_limit(tmp_path, seeds, paired, opts):
    """One read of 22,000 frames and more moves the whole batch to the general kernel."""
    rng = np.random.default_rng(7 + paired)
    targets = _targets(rng)
    path, f, names = _build(tmp_path, targets, seeds=["1111011101110010111011111",
                                                      "1101111101001011111011011",
                                                      "1111101011100111010111111"]
                            if seeds else None)
    reads, reads2 = _reads(rng, targets, 250, paired=paired)
    reads.append(targets[0] + targets[3] + b"N" * 40 + targets[0][:500])
    if paired:
        reads2.append(targets[6][:400])
    _check(path, f, names, reads, reads2, **opts)
