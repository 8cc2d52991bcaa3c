"""A caller's table without a cut-over, on a DB whose longest records need no
layout of their own: its long shape takes the whole DB."""
import numpy as np
import pytest

import oracle
from swhybrid_b200 import capi, param, synth

pytestmark = pytest.mark.gpu
M = param.blosum62()


@pytest.mark.parametrize("long,short", [((8, 16), (16, 32)), ((16, 32), (8, 16)), ((32, 8), (4, 40))])
def test_long_shape_takes_the_whole_db(long, short):
    rng = np.random.default_rng(83)
    db = synth.db_from_lengths(rng, rng.integers(150, 201, size=60_000))
    q = synth.residues(rng, 250)
    with capi.Context(0) as c:
        c.load_db(db.residues, db.offsets)
        c.set_tuning([(100_000, (*long, *short, 0))])
        assert [st[:2] for st in c.plan(len(q))] == [long]
        _, scores = c.search(q, want_scores=True)
    np.testing.assert_array_equal(scores, oracle.search(q, db.residues, db.offsets, M, 12, 2))
