"""Device memory of best-hit calls: what is kept for their scores, and calls for which there
is no room."""
import numpy as np
import pytest

from tests import oracle_lib as ol
from tests.test_lane_gpu import _device, _filters, _open

pytestmark = pytest.mark.gpu

NF, READS = 40, 400_000
SCORES = 8 * NF * READS  # 128 MB a mate


def _open_best(tmp_path):
    from biobloom_b200 import MODE_BESTHIT
    rng = np.random.default_rng(2)
    genomes, filters, paths = _filters(tmp_path, rng, [25] * NF, 3, glen=3000)
    c = _open(paths, ol.SIMPLE, 0.15, 3, path=2)
    c.set_mode(MODE_BESTHIT)
    starts = rng.integers(0, 2970, READS)
    which = rng.integers(0, NF, READS)
    reads = [genomes[w][s:s + 30].tobytes() for w, s in zip(which, starts)]
    return c, filters, reads


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("mates", [1, 2])
def test_scores_of_the_mates_that_there_are(tmp_path, mates):
    import torch
    c, _, reads = _open_best(tmp_path)
    dev = _device(reads) * mates
    out = {"hits": torch.empty((READS, 1), dtype=torch.int64, device="cuda"),
           "category": torch.empty(READS, dtype=torch.int32, device="cuda")}
    if mates == 2:
        out["hits2"] = out["hits"].clone()
    small = _device(reads[:60_000]) * mates  # loads the kernels
    loaded = c.classify_device(*small)
    before = _free()
    del loaded
    c.classify_device(*dev, **out)
    used = before - _free()
    c.close()
    # the scores, 4 bytes a read for the list, and an allocation's granularity for each
    assert mates * SCORES * 0.8 < used < mates * SCORES + 4 * mates * READS + (8 << 20)


def test_calls_without_room_for_scores(tmp_path):
    """The call takes the kernels that need none, and the others again once there is room."""
    import torch
    c, filters, reads = _open_best(tmp_path)
    want, _ = ol.best_hit(ol.classify_scores(*ol.pack_reads(reads), filters, ol.SIMPLE, 3))
    dev, small, few = _device(reads), _device(reads[:60_000]), _device(reads[:1000])
    out = {"hits": torch.empty((READS, 1), dtype=torch.int64, device="cuda"),
           "category": torch.empty(READS, dtype=torch.int32, device="cuda")}
    loaded = [c.classify_device(*b) for b in (small, few)]  # the lane kernel, and the others
    torch.cuda.synchronize()
    del loaded
    out["hits"].fill_(0)  # and torch's
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    taken = torch.empty(_free() - SCORES * 3 // 4, dtype=torch.uint8, device="cuda")
    assert _free() < SCORES
    for room in (False, True):
        if room:
            del taken
            torch.cuda.empty_cache()
        out["hits"].fill_(-1)
        torch.cuda.synchronize()
        c.classify_device(*dev, **out)
        torch.cuda.synchronize()
        assert np.array_equal(out["hits"].cpu().numpy().view(np.uint64), want)
        assert (c.last_stats()["kernels"] > NF) == room
    c.close()
