"""The work that programs have this library do, as cases that can be timed.

Three uses are covered: screening reads against Bloom filters
(`BioBloomClassifier`), assigning them to the targets of a multi-index filter
(`MIBFClassifier`), and building a filter (`synth.make_filter`).  The indexes
have the sizes of this repository's benchmark workloads (k = 25, FPR 0.075,
three hashes):

  small    one filter of a 5 Mbp reference (3.4 MB: it stays in L2);
  genome   one filter of the size of a 3.1 Gbp reference (2.1 GB: every probe
           is a DRAM access); its bits are those of a 64 Mbp part of that
           reference, the rest set at random to the density a full one has;
  panel    ten filters of 100 Mbp references (68 MB each);
  targets  a multi-index filter over 500 targets of 400 kbp, three spaced seeds
           of span 25 and weight 19;
  strains  a multi-index filter over 100 targets of 400 kbp, k-mers.

They are opened once in a process and kept, as a program that classifies many
batches keeps them; their files are built once and lie in the temporary
folder.  The reads of a case come from its seed.
"""
import math
import os
import shutil
import tempfile

import numpy as np
import torch

from biobloom_b200 import MODE_BESTHIT, MODE_ORDERED, MODE_SCORES, MODE_STD, BioBloomClassifier
from biobloom_b200 import MIBFClassifier, make_mibf, synth
from biobloom_b200 import _lib as L

K, FPR, HASHES, STREAK = 25, 0.075, 3, 3
MODES = {"std": MODE_STD, "ordered": MODE_ORDERED, "best": MODE_BESTHIT, "scores": MODE_SCORES}
# threshold of each scoring method: the defaults of the command line, and a
# minimum match of 40 bases
THRESHOLD = {"simple": 0.15, "harmonic": 0.15, "binomial": 100, "length": 40}
BLOOM = {"small": (1, 5_000_000), "genome": (1, 64_000_000), "panel": (10, 100_000_000)}
GENOME_BASES = 3_100_000_000
MIBF = {"targets": (500, 400_000, True), "strains": (100, 400_000, False)}
SEEDS = ["1101111011101110110111011", "1011101101110111011110111", "1110110111011011110110111"]


def _reads(name, index, reads, lo=150, hi=150, long_frac=0.0, paired=False, **more):
    c = {"kind": "mibf" if index in MIBF else "bloom", "index": index, "reads": reads,
         "len_min": lo, "len_max": hi, "long_frac": long_frac, "paired": paired}
    if c["kind"] == "bloom":
        c.update(mode="std", scoring="simple", dust=False, packed=False, host=False)
    c.update(more)
    return {"name": name, **c} if name else c


def listed():
    return [
        # the smallest request of a serving loop: launches and latency
        _reads("small-1k", "small", 1000),
        # an ordinary batch of short reads against a bacterial reference
        _reads("small-1m", "small", 1_000_000),
        # a request of ragged reads, 2-bit packed as the file pipeline sends them,
        # against a human-sized reference
        _reads("genome-mixed-50k", "genome", 50_000, 50, 300, 0.05, packed=True),
        # an offline batch of ragged reads: short ones with 5% of 300 bp to 10 kb
        _reads("genome-mixed-2m", "genome", 2_000_000, 50, 300, 0.05),
        # contamination screen of read pairs against several references
        _reads("panel-pairs-400k", "panel", 400_000, paired=True),
        # the same, each pair to its best reference (-b)
        _reads("panel-best-200k", "panel", 200_000, paired=True, mode="best"),
        # every filter's score of every read, written out (-w), harmonic scoring
        _reads("panel-scores-100k", "panel", 100_000, mode="scores", scoring="harmonic"),
        # low-complexity masking before the screen (-D), trimmed reads
        _reads("panel-dust-100k", "panel", 100_000, 101, 151, dust=True),
        # reads handed over in host memory, as a program that parses files has them
        _reads("host-400k", "small", 400_000, host=True),
        # metagenomic reads to 500 targets, spaced seeds
        _reads("targets-500k", "targets", 500_000),
        # ragged pairs to 100 strains, k-mers
        _reads("strains-pairs-50k", "strains", 50_000, 75, 300, paired=True),
        # the filter of one chromosome-sized reference
        {"name": "make-20m", "kind": "make", "bases": 20_000_000},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("single", "single", "panel", "panel", "mibf", "host", "make"))
    if kind == "make":
        return {"kind": "make", "bases": log(100_000, 20_000_000)}
    lo = rng.randint(50, 151)
    hi = lo if rng.random() < 0.3 else rng.randint(lo, 300)
    paired = rng.random() < 0.5
    if kind == "single":
        index, long_frac = rng.choice(("small", "genome")), rng.choice((0.0, 0.05, 0.1))
        bases = 0.5 * (lo + hi) + 2765 * long_frac
        most = min(1_500_000, 4e8 / bases / (2 if paired else 1))
        return _reads("", index, log(1000, most), lo, hi, long_frac, paired,
                      scoring=rng.choice(("simple", "simple", "length", "binomial")),
                      packed=rng.random() < 0.4)
    if kind == "panel":
        mode = rng.choice(("std", "std", "ordered", "best", "scores"))
        return _reads("", "panel", log(1000, 120_000), lo, hi, 0.0, paired, mode=mode,
                      scoring=rng.choice(("simple", "simple", "harmonic", "length")),
                      dust=rng.random() < 0.15)
    if kind == "host":
        return _reads("", "small", log(1000, 400_000), lo, hi, 0.0, paired, host=True)
    return _reads("", rng.choice(("targets", "strains")), log(1000, 250_000), lo, hi,
                  rng.choice((0.0, 0.0, 0.02)), paired)


# ---- indexes -------------------------------------------------------------------

_kept = {}


def _once(key, make):
    if key not in _kept:
        _kept[key] = make()
    return _kept[key]


def _stream():
    return _once("stream", torch.cuda.Stream)


def _bases(seed, n):
    """n uniform random bases (codes 0..3) on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(0, 4, (n,), generator=g, device="cuda", dtype=torch.uint8)


_ASCII = (65, 67, 71, 84)


def _ascii(codes):
    return torch.tensor(_ASCII, dtype=torch.uint8, device="cuda")[codes.to(torch.int64)]


def _references(index):
    """The references an index was built from, one after another, as codes."""
    n, bases = (BLOOM if index in BLOOM else MIBF)[index][:2]
    return _once(("ref", index), lambda: torch.cat(
        [_bases(1000 + 17 * len(index) + i, bases) for i in range(n)]).view(n, bases))


def _fill(path):
    """Sets the bits of a filter at random, beside those it has, to a density of
    27/64: that of a filter filled to an FPR of 0.075 with three hashes."""
    g = torch.Generator(device="cuda").manual_seed(77)
    with open(path, "rb") as f:
        at = f.read(4096).index(b"[HeaderEnd]\n") + 12
    words = np.memmap(path, dtype=np.uint8, mode="r+", offset=at)
    for i in range(0, len(words), 1 << 28):
        part = torch.from_numpy(words[i:i + (1 << 28)]).cuda()
        fill = torch.zeros_like(part)
        for bit in (1, 1, 0, 1, 1, 0):
            r = torch.randint(0, 256, part.shape, generator=g, device="cuda", dtype=torch.uint8)
            fill = fill | r if bit else fill & r
        words[i:i + (1 << 28)] = (part | fill).cpu().numpy()
    words.flush()


def _build(index, folder):
    refs = _references(index)
    if index in BLOOM:
        for i in range(len(refs)):
            stem = os.path.join(folder, f"{index}{i}")
            synth.make_filter([_ascii(refs[i]).cpu().numpy()], stem, f"{index}{i}", k=K, fpr=FPR,
                              hash_num=HASHES, entries=GENOME_BASES if index == "genome" else 0)
            if index == "genome":
                _fill(stem + ".bf")
        return
    n, _, spaced = MIBF[index]
    make_mibf(os.path.join(folder, index), [_ascii(r).cpu().numpy().tobytes() for r in refs],
              list(range(1, n + 1)), [f"{index}{i + 1}" for i in range(n)],
              seeds=SEEDS if spaced else None, k=K, hash_num=HASHES)


def _files(index):
    """The index's folder, built by the first process that needs it."""
    base = os.path.join(tempfile.gettempdir(), f"biobloom_b200_indexes_{os.getuid()}")
    folder = os.path.join(base, index)
    if not os.path.isdir(folder):
        os.makedirs(base, exist_ok=True)
        part = tempfile.mkdtemp(dir=base)
        _build(index, part)
        try:
            os.rename(part, folder)
        except OSError:  # another process was first
            shutil.rmtree(part)
    return folder


def _classifier(case):
    index = case["index"]
    if index in MIBF:
        return _once(index, lambda: MIBFClassifier(os.path.join(_files(index), index + ".bf")))

    def make():
        folder = _files(index)
        c = BioBloomClassifier(
            [os.path.join(folder, f"{index}{i}.bf") for i in range(BLOOM[index][0])],
            THRESHOLD[case["scoring"]], streak_threshold=STREAK,
            score_type="simple" if case["scoring"] == "length" else case["scoring"])
        c.set_mode(MODES[case["mode"]])
        if case["dust"]:
            c.set_dust()
        return c
    return _once((index, case["mode"], case["scoring"], case["dust"]), make)


# ---- reads ---------------------------------------------------------------------

def _lengths(g, case):
    """Log-uniform lengths; long_frac of the reads from 300 bp to 10 kb."""
    n, lo, hi = case["reads"], case["len_min"], case["len_max"]

    def spread(a, b):
        u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
        return torch.exp(u * math.log((b + 1) / a)).mul(a).long().clamp(a, b)

    lens = spread(lo, hi)
    if case["long_frac"]:
        far = torch.rand(n, generator=g, device="cuda") < case["long_frac"]
        lens = torch.where(far, spread(300, 10_000), lens)
    return lens


def _take(g, refs, which, start, lens, flip, rates):
    """Codes (4 = N) of the reads: lens[i] bases of reference which[i] (-1:
    random ones) from start[i], reversed and complemented where flip[i], with
    substitutions and Ns."""
    out = torch.empty(int(lens.sum()), dtype=torch.uint8, device="cuda")
    flat, width, at = refs.view(-1), refs.shape[1], 0
    for i in range(0, len(lens), 1 << 18):
        s = slice(i, i + (1 << 18))
        l, w, f = lens[s], which[s], flip[s]
        ends = l.cumsum(0)
        total = int(ends[-1])
        j = torch.arange(total, device="cuda") - torch.repeat_interleave(ends - l, l)
        j = torch.where(torch.repeat_interleave(f, l), torch.repeat_interleave(l - 1, l) - j, j)
        c = flat[j + torch.repeat_interleave(w.clamp(min=0) * width + start[s], l)]
        del j
        c = torch.where(torch.repeat_interleave(f, l), 3 - c, c)
        r = torch.randint(0, 4, (total,), generator=g, device="cuda", dtype=torch.uint8)
        u = torch.rand(total, generator=g, device="cuda")
        c = torch.where((u < rates[0]) | torch.repeat_interleave(w < 0, l), r, c)
        out[at:at + total] = torch.where(u > 1 - rates[1], torch.full_like(c, 4), c)
        at += total
    return out


# Share of the reads that come from the index's references, and substitutions
# and Ns per base, as in the benchmark's workloads.
SOURCE = {"small": (0.7, 0.01, 1e-4), "genome": (0.7, 0.01, 1e-4), "panel": (0.8, 0.005, 1e-4),
          "targets": (0.9, 0.01, 1e-4), "strains": (0.9, 0.01, 1e-4)}


def _mates(case, seed):
    """Codes and offsets of the reads (of both mates: the ends of fragments of
    at least 300 bp, facing each other)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    refs = _references(case["index"])
    share, *rates = SOURCE[case["index"]]
    n = case["reads"]
    which = torch.randint(0, len(refs), (n,), generator=g, device="cuda")
    which[torch.rand(n, generator=g, device="cuda") >= share] = -1
    l1 = _lengths(g, case)
    start = (torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
             * (refs.shape[1] - 30_000)).long()
    if case["paired"]:
        l2 = _lengths(g, case)
        flip = torch.zeros(n, dtype=torch.bool, device="cuda")
        span = torch.randint(300, 501, (n,), generator=g, device="cuda")
        span = torch.maximum(span, torch.maximum(l1, l2))
        mates = [(l1, start, flip), (l2, start + span - l2, ~flip)]
    else:
        mates = [(l1, start, torch.rand(n, generator=g, device="cuda") < 0.5)]
    got = []
    for lens, at, flip in mates:
        off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
        off[1:] = lens.cumsum(0)
        got.append((_take(g, refs, which, at, lens, flip, rates), off))
    return got


def _two_bit(codes):
    """2-bit code words and validity bits of the codes."""
    n = len(codes)
    pad = torch.zeros((n + 31) // 32 * 32, dtype=torch.uint8, device="cuda")
    pad[:n] = codes
    ok = (pad != 4).view(-1, 8)
    ok.view(-1)[n:] = False
    weights = torch.tensor([1, 2, 4, 8, 16, 32, 64, 128], dtype=torch.uint8, device="cuda")
    valid = (ok * weights).sum(1, dtype=torch.uint8).view(torch.int32)
    q = (pad & 3).view(-1, 4)
    return (q[:, 0] | q[:, 1] << 2 | q[:, 2] << 4 | q[:, 3] << 6).view(torch.int32), valid


def prepare(case, seed):
    if case["kind"] == "make":
        folder = _once("make", tempfile.mkdtemp)
        return {"case": case, "stem": os.path.join(folder, f"made{seed}"),
                "bases": _ascii(_bases(seed, case["bases"])).cpu().numpy()}
    state = {"case": case, "classifier": _classifier(case)}
    mates = _mates(case, seed)
    if case["kind"] == "bloom" and case["packed"]:
        state["mates"] = [(*_two_bit(codes), off) for codes, off in mates]
        return state
    table = torch.tensor(_ASCII + (78,), dtype=torch.uint8, device="cuda")
    mates = [(table[codes.to(torch.int32)], off) for codes, off in mates]
    if case["kind"] == "bloom" and case["host"]:
        mates = [(seq.cpu().numpy(), off.cpu().numpy().astype(np.uint64)) for seq, off in mates]
    state["mates"] = mates
    return state


# ---- passes --------------------------------------------------------------------

def _run_make(state):
    stem = state["stem"]
    synth.make_filter([state["bases"]], stem, "made", k=K, fpr=FPR, hash_num=HASHES)
    with open(stem + ".txt") as f:
        info = dict(line.split("=", 1) for line in f if "=" in line)
    with open(stem + ".bf", "rb") as f:
        bits = np.frombuffer(f.read(), dtype=np.uint8)
    os.remove(stem + ".bf")
    os.remove(stem + ".txt")
    return {"bf": bits, "entries": int(info["num_entries"]),
            "redundant": int(info["redundant_sequences"])}


def _run_packed(state):
    """A device batch of 2-bit packed reads, through the C interface."""
    c, mates = state["classifier"], state["mates"]
    n = len(mates[0][2]) - 1
    hits = [torch.empty((n, c.words), dtype=torch.int64, device="cuda") for _ in mates]
    category = torch.empty(n, dtype=torch.int32, device="cuda")
    b, r = L.Batch(), L.Result()
    b.n_reads, b.location, b.encoding = n, L.DEVICE, L.BASES_2BIT
    b.seq, b.valid, b.offsets = (t.data_ptr() for t in mates[0])
    r.hits, r.category, r.location = hits[0].data_ptr(), category.data_ptr(), L.DEVICE
    if len(mates) == 2:
        b.seq2, b.valid2, b.offsets2 = (t.data_ptr() for t in mates[1])
        r.hits2 = hits[1].data_ptr()
    L.check(L.lib().bbt_classify_batch(c._ctx, b, r, torch.cuda.current_stream().cuda_stream),
            c._ctx)
    return *hits, category


def run(state):
    case = state["case"]
    if case["kind"] == "make":
        return _run_make(state)
    c, mates = state["classifier"], state["mates"]
    with torch.cuda.stream(_stream()):
        if case["kind"] == "mibf":
            return c.classify_device(*(t for m in mates for t in m), max_hits=4)
        if case["host"]:
            return c.classify(*mates)
        if case["packed"]:
            return _run_packed(state)
        if case["mode"] != "scores":
            return c.classify_device(*(t for m in mates for t in m))
        scores = [torch.empty((case["reads"], c.n_filters), dtype=torch.float64, device="cuda")
                  for _ in mates]
        got = c.classify_device(*(t for m in mates for t in m), scores=scores[0],
                                scores2=scores[1] if case["paired"] else None)
        return *got, scores


def _filter_bits(bases, entries=0):
    n = entries or bases - K + 1
    return -n * HASHES / math.log(1 - FPR ** (1 / HASHES))


def work(case):
    """Bases and offsets read once, results written once, and the index: the
    sectors its probes touch, or all of it once where that is less.  A read that
    matches needs three tests for each of the frames that decide it, one that
    does not about 1.6 for each of the frames that rule it out; scores and
    multi-index queries visit every frame."""
    if case["kind"] == "make":
        return {"bytes": case["bases"] + _filter_bits(case["bases"]) / 8, "flops": 0}
    lo, hi, mates = case["len_min"], case["len_max"], 2 if case["paired"] else 1
    mean = lo if lo == hi else (hi - lo) / math.log(hi / lo)
    mean += case["long_frac"] * (9700 / math.log(10_000 / 300) - mean)
    reads, frames = case["reads"] * mates, mean - K + 1
    share = SOURCE[case["index"]][0]
    if case["kind"] == "mibf":
        n, bases, spaced = MIBF[case["index"]]
        index = 2 * n * bases * HASHES / math.log(2)
        probes, out = reads * frames * HASHES, case["reads"] * (28 + 8)
    else:
        n, bases = BLOOM[case["index"]]
        entries = GENOME_BASES if case["index"] == "genome" else 0
        index = n * _filter_bits(bases, entries) / 8
        out = reads * 8 + case["reads"] * 4
        if case["mode"] == "best" or case["mode"] == "scores":
            hit = miss = 1.6 * frames
            out += reads * n * 8 if case["mode"] == "scores" else 0
        else:
            hit, miss = 0.15 * frames * HASHES, 0.85 * frames * 1.6
        probes = reads * (share * (hit + (n - 1) * miss) + (1 - share) * n * miss)
    packed = case["kind"] == "bloom" and case["packed"]
    return {"bytes": reads * (mean * (0.375 if packed else 1) + 8) + out + min(index, 32 * probes),
            "flops": 0}


# ---- scores in 64 bits ---------------------------------------------------------

_SEED = (0x3c8bfbb395c60474, 0x3193c18562a02b4c, 0x20323ed082572324, 0x295549f54be24456)


def _signed(v):
    v &= (1 << 64) - 1
    return v - (1 << 64) if v >> 63 else v


def _rol(v, s):
    s %= 64
    return _signed((v << s) | ((v & ((1 << 64) - 1)) >> (64 - s)))


def _hashes(codes):
    """Canonical ntHash of every frame of reads of one length (n x len codes)
    and whether the frame holds only bases."""
    frames = codes.shape[1] - K + 1
    fw = torch.zeros((codes.shape[0], frames), dtype=torch.int64, device="cuda")
    rc = torch.zeros_like(fw)
    ok = torch.ones_like(fw, dtype=torch.bool)
    for j in range(K):
        c = codes[:, j:j + frames].long()
        f = torch.tensor([_rol(s, K - 1 - j) for s in _SEED] + [0], device="cuda")
        r = torch.tensor([_rol(s, j) for s in reversed(_SEED)] + [0], device="cuda")
        fw ^= f[c]
        rc ^= r[c]
        ok &= c < 4
    top = -1 << 63
    return torch.where((fw ^ top) < (rc ^ top), fw, rc), ok


def _mod(v, m):
    """The unsigned 64-bit v mod m, m below 2^31."""
    low = (1 << 32) - 1
    return (((v >> 32) & low) % m * ((1 << 32) % m) + (v & low)) % m


def _contains(path, canon):
    with open(path, "rb") as f:
        data = f.read()
    at = data.index(b"[HeaderEnd]\n") + 12
    bits = torch.frombuffer(bytearray(data[at:]), dtype=torch.uint8).cuda()
    m, hit = len(bits) * 8, torch.ones_like(canon, dtype=torch.bool)
    for i in range(HASHES):
        v = canon
        if i:
            v = canon * _signed(i ^ (K * 0x90b45d39fb6da1fa))
            v = v ^ ((v >> 27) & ((1 << 37) - 1))
        b = _mod(v, m)
        hit &= ((bits[b >> 3].long() >> (b & 7)) & 1).bool()
    return hit


def exact(case, seed):
    """The scores of the SCORES mode (everything else returned is whole
    numbers): simple or harmonic scoring of reads of one length, no masking."""
    if case["kind"] != "bloom" or case["mode"] != "scores" or case["dust"] or \
            case["scoring"] not in ("simple", "harmonic") or case["len_min"] != case["len_max"]:
        return None
    folder, (nf, _), out = _files(case["index"]), BLOOM[case["index"]], []
    for codes, _ in _mates(case, seed):
        canon, ok = _hashes(codes.view(case["reads"], -1))
        n, frames = canon.shape
        score = torch.zeros((n, nf), dtype=torch.float64, device="cuda")
        for f in range(nf):
            hits = _contains(os.path.join(folder, f"{case['index']}{f}.bf"), canon) & ok
            s = torch.zeros(n, dtype=torch.float64, device="cuda")
            streak, skip = (torch.zeros(n, dtype=torch.int64, device="cuda") for _ in range(2))
            for p in range(frames):
                at = ok[:, p] & (skip <= p)
                if p and not bool(ok[:, p - 1].all()):
                    streak = torch.where(ok[:, p - 1], streak, 0)
                hit, miss = at & hits[:, p], at & ~hits[:, p]
                later = (1.0 if case["scoring"] == "simple"
                         else 1.0 - 1.0 / (1.0 + streak.double()))
                s += hit * torch.where(streak > 0, later, 0.5)
                skip = torch.where(miss & (streak >= STREAK), p + K, skip)
                streak = torch.where(hit, streak + 1, torch.where(miss, 0, streak))
            score[:, f] = s / frames
        out.append(score)
    whole = (None, None, None)  # hits, hits2, category
    return *whole, out
