"""The long records' items of a batch run in one launch whatever row counts its
queries need: launches of their own queued behind the first one lost the SMs the
first paired launch leaves free to the next paired launch."""
import numpy as np
import pytest

import oracle
from swhybrid_b200 import capi, param, synth

pytestmark = pytest.mark.gpu
M = param.blosum62()


def test_one_launch_for_every_row_count():
    rng = np.random.default_rng(43)
    lens = np.concatenate([rng.integers(20, 400, size=1500), [9000, 8999, 7000, 5000, 3001]])
    db = synth.db_from_lengths(rng, lens[rng.permutation(len(lens))])
    # both batches: two lanes of 5,000 rows (three segment levels) and a tall
    # double stack or two beside them, so the same paired launches
    same = [synth.residues(rng, 5000) for _ in range(4)]            # 16 rows a lane
    mixed = same[:2] + [synth.residues(rng, n) for n in (2600, 700)]    # 16, 8 and 4
    with capi.Context(0) as c:
        c.load_db(db.residues, db.offsets)
        c.search_batch(same)
        one = c.run_stats().launches
        hits, scores = c.search_batch(mixed, want_scores=True)
        assert c.run_stats().launches == one
    for q, sc in zip(mixed, scores):
        np.testing.assert_array_equal(sc, oracle.search(q, db.residues, db.offsets, M, 12, 2, mode=0))
