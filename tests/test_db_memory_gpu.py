"""A DB that fits the device only without the room for windows of long pairs loads
all the same, and is searched without windows."""
import numpy as np
import pytest

import oracle
from swhybrid_b200 import capi, param, synth

pytestmark = pytest.mark.gpu
M = param.blosum62()


# bytes left to the DB beyond its own: less than the room for windows (20 MiB
# here), and less than twice that room
@pytest.mark.parametrize("spare_mib", [14, 34, 400])
def test_a_db_that_nearly_fills_the_device(spare_mib):
    import torch
    rng = np.random.default_rng(61)
    lens = np.concatenate([rng.integers(300, 501, size=39_990), rng.integers(8_000, 30_000, size=10)])
    db = synth.db_from_lengths(rng, lens[rng.permutation(len(lens))])
    q = synth.residues(rng, 130)
    srt = np.sort(lens)[::-1][::2]
    need = int(((srt + 7) // 8).sum()) * 144          # column streams and boundary rows
    with capi.Context(0) as c:
        c.load_db(db.residues, db.offsets)
        roomy = int(c.db_stats().device_bytes)
        hits, scores = c.search(q, want_scores=True)   # loads the kernels
        np.testing.assert_array_equal(scores, oracle.search(q, db.residues, db.offsets, M, 12, 2))
        c.load_db(np.zeros(1, dtype=np.uint8), np.array([0, 1], dtype=np.uint64))
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info(0)[0]
        assert roomy - need > 18 << 20
        # (the other buffers: scores, lists, keys and 296 re-score rows)
        other = 296 * 8 * (int(srt[0]) + 8) + 40_000 * 24 + 2 * 11 * 1024 * 8
        hog = torch.empty(free - need - other - (spare_mib << 20), dtype=torch.uint8, device="cuda:0")
        try:
            c.load_db(db.residues, db.offsets)
            tight = int(c.db_stats().device_bytes)
            hits2, scores2 = c.search(q, want_scores=True)
        finally:
            del hog
            torch.cuda.empty_cache()
    assert (tight < roomy) == (spare_mib < 100)
    np.testing.assert_array_equal(scores2, scores)
    assert hits2 == hits
